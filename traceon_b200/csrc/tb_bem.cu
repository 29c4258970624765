// tb_bem.cu -- BEM assembly and field-sum kernels of the radial path.
//
//   jacobian buffer      radial.c:224-246
//   matrix fill          radial.c:249-310 (off-diagonal Gauss sums, tb_fill.cuh)
//   self integrals       radial.c:182-222 + traceon/backend/__init__.py:688-708
//   potential / field    radial.c:105-173, batched over points
//   axial derivatives    radial.c:18-36
//   axial coefficients   traceon/field.py:914-937
//   axial evaluation     radial.c:312-384, batched over points
//
// Everything is FP64.  The sums over rings are FP64-pipe bound (one reciprocal
// square root and a table logarithm per ring pair); large maps go through the
// ring tree (tb_tree.cu), a few points take a cluster of CTAs each.
#include <cooperative_groups.h>

#include "tb_common.cuh"
#include "tb_internal.cuh"
#include "tb_fill.cuh"
#include "../../include/traceon_b200.h"

namespace tb {

// ---------------------------------------------------------------- graded meshes
// Cubic line elements along straight segments, graded toward both ends of
// every segment: segment s from (r0, z0) to (r1, z1) carries off[s + 1] -
// off[s] elements whose nodes are the Chebyshev-Lobatto points
// t_k = (1 - cos(pi k / n)) / 2 (t_0 = 0, t_n = 1) -- the host mesher's rule
// (geometry.graded_nodes), with its operations in the same order and without
// fused multiply-adds.  Rows in the reference's line4 layout [start, end,
// 1/3-point, 2/3-point] of (r, 0, z) (traceon/mesher.py:188-227), every
// coordinate with its low 16 mantissa bits cleared: the truncation the
// reference's Mesh merges points with (traceon/mesher.py:262-290).  One
// thread per element; its segment by binary search of the offsets.
__device__ __forceinline__ double snap16(double x) {
  return __longlong_as_double(__double_as_longlong(x) & (long long)0xFFFFFFFFFFFF0000ULL);
}

__device__ __forceinline__ double cheb_node(int64_t k, int64_t n) {
  if (k <= 0) return 0.0;
  if (k >= n) return 1.0;
  return __dmul_rn(0.5, __dsub_rn(1.0, cos(__ddiv_rn(__dmul_rn(PI, double(k)), double(n)))));
}

__global__ void k_mesh_segments(const double* __restrict__ seg, const int64_t* __restrict__ off, int64_t S,
                                double* __restrict__ out, int64_t N) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= N) return;
  int64_t lo = 0, hi = S - 1;  // the last segment with off[s] <= i
  while (lo < hi) {
    const int64_t mid = (lo + hi + 1) / 2;
    if (off[mid] <= i)
      lo = mid;
    else
      hi = mid - 1;
  }
  const int64_t n = off[lo + 1] - off[lo], k = i - off[lo];
  const double a = cheb_node(k, n), b = cheb_node(k + 1, n);
  const double d = __dsub_rn(b, a);
  const double t[4] = {a, b, __dadd_rn(a, __ddiv_rn(d, 3.0)), __dadd_rn(a, __ddiv_rn(__dmul_rn(2.0, d), 3.0))};
  const double r0 = seg[4 * lo], z0 = seg[4 * lo + 1], dr = __dsub_rn(seg[4 * lo + 2], r0),
               dz = __dsub_rn(seg[4 * lo + 3], z0);
  double* row = out + i * 12;
  for (int q = 0; q < 4; q++) {
    row[3 * q] = snap16(__dadd_rn(r0, __dmul_rn(dr, t[q])));
    row[3 * q + 1] = 0.0;
    row[3 * q + 2] = snap16(__dadd_rn(z0, __dmul_rn(dz, t[q])));
  }
}

// ---------------------------------------------------------------- jacobian
__global__ void k_jacobian_buffer(const double* __restrict__ vertices, double* __restrict__ jac,
                                  double* __restrict__ pos, int64_t N) {
  int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (g >= N * NQ) return;
  int64_t i = g / NQ;
  int k = int(g % NQ);
  Cubic c;
  c.load(vertices + i * 12);
  double r, z, j;
  c.point(gauss_x(k), false, r, z, j);
  jac[g] = gauss_w(k) * j;
  pos[2 * g] = r;
  pos[2 * g + 1] = z;
}

__global__ void k_element_targets(const double* __restrict__ vertices, double* __restrict__ target,
                                  double* __restrict__ normal, int64_t N) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= N) return;
  Cubic c;
  c.load(vertices + i * 12);
  double r, z, j, nr, nz;
  c.point(0.0, false, r, z, j);
  c.normal(0.0, nr, nz);
  if (target) {
    target[2 * i] = r;
    target[2 * i + 1] = z;
  }
  if (normal) {
    normal[2 * i] = nr;
    normal[2 * i + 1] = nz;
  }
}

// ---------------------------------------------------------------- fill
// One CTA per tile of 64 columns and up to 64 rows (fewer when the matrix is
// small, launch_fill): the columns' quadrature nodes and the rows' collocation
// data staged in shared memory (fill_columns, fill_rows), then thread (c, g)
// walks rows g, g + 4, ... of column c: the 32 lanes of a warp write 256
// contiguous bytes, and neighbouring columns mostly take the same rule.
__device__ __forceinline__ void fill_tile(FillTile& s, double* __restrict__ A, int64_t lda,
                                          const double* __restrict__ vertices, const uint8_t* __restrict__ types,
                                          const double* __restrict__ values, const double* __restrict__ jac,
                                          const double* __restrict__ pos, int64_t N, int64_t i0, int64_t i1, int64_t j0,
                                          int accumulate, int gauss_diagonal) {
  fill_columns(s, vertices, jac, pos, N, j0);
  fill_rows(s, vertices, types, values, i0, i1);
  __syncthreads();
  const int c = threadIdx.x % FILL_TILE;
  const int64_t j = j0 + c;
  if (j < N) {
#pragma unroll 1
    for (int q = threadIdx.x / FILL_TILE; q < FILL_TILE && i0 + q < i1; q += FILL_THREADS / FILL_TILE) {
      const int64_t i = i0 + q;
      if (i == j && !gauss_diagonal) continue;
      const double v = fill_pair(s, q, c, vertices, jac, pos, j);
      double* a = A + i * lda + j;
      *a = accumulate ? *a + v : v;
    }
  }
}

__global__ void __launch_bounds__(FILL_THREADS)
    k_fill_matrix(double* __restrict__ A, int64_t lda, const double* __restrict__ vertices,
                  const uint8_t* __restrict__ types, const double* __restrict__ values,
                  const double* __restrict__ jac, const double* __restrict__ pos, int64_t N, int64_t row0,
                  int64_t row1, int rows, int accumulate, int gauss_diagonal) {
  __shared__ FillTile s;
  const int64_t i0 = row0 + blockIdx.y * (int64_t)rows;
  fill_tile(s, A, lda, vertices, types, values, jac, pos, N, i0, row1 - i0 < rows ? row1 : i0 + rows,
            blockIdx.x * (int64_t)FILL_TILE, accumulate, gauss_diagonal);
}

// ---------------------------------------------------------------- batched fill
// Many geometries of uneven N in one persistent launch: the tiles of all
// matrices are numbered globally (geometry g owns tiles [tile0[g], tile0[g] +
// T^2), T = ceil(N / 64)); CTAs stride over them and find their geometry by
// binary search.  Diagonal entries are left to the self integrals, as in the
// single-geometry fill.
__global__ void __launch_bounds__(FILL_THREADS)
    k_fill_matrix_batched(const tb_geometry_t* __restrict__ geoms, int n_geoms, int64_t total_tiles) {
  __shared__ FillTile s;
  for (int64_t t = blockIdx.x; t < total_tiles; t += gridDim.x) {
    int lo = 0, hi = n_geoms - 1;  // last geometry with tile0 <= t
    while (lo < hi) {
      const int mid = (lo + hi + 1) / 2;
      if (geoms[mid].tile0 <= t)
        lo = mid;
      else
        hi = mid - 1;
    }
    const tb_geometry_t& g = geoms[lo];
    const int64_t T = (g.N + FILL_TILE - 1) / FILL_TILE, local = t - g.tile0;
    __syncthreads();  // the previous tile's data is no longer read
    fill_tile(s, g.A, g.lda, g.vertices, g.types, g.values, g.jac, g.pos, g.N, (local / T) * FILL_TILE, g.N,
              (local % T) * FILL_TILE, 0, 0);
  }
}

// The self terms (one warp per element).
__global__ void k_self_integrals(const double* __restrict__ vertices, const uint8_t* __restrict__ types,
                                 const double* __restrict__ values, double* __restrict__ diag,
                                 double* __restrict__ A, int64_t lda, int64_t N) {
  int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / 32;
  int lane = threadIdx.x & 31;
  if (i >= N) return;
  const double v = self_term_warp(vertices, types, values, i, lane);
  if (lane == 0) {
    if (diag) diag[i] = v;
    if (A) A[i * lda + i] = v;
  }
}

// The self terms of all elements of many geometries (one warp per element,
// grid-strided over the global element numbering), onto their matrices'
// diagonals.
__global__ void k_self_integrals_batched(const tb_geometry_t* __restrict__ geoms, int n_geoms, int64_t total) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * blockDim.x / 32;
  for (int64_t e = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / 32; e < total; e += warps) {
    int lo = 0, hi = n_geoms - 1;  // last geometry with elem0 <= e
    while (lo < hi) {
      const int mid = (lo + hi + 1) / 2;
      if (geoms[mid].elem0 <= e)
        lo = mid;
      else
        hi = mid - 1;
    }
    const tb_geometry_t& g = geoms[lo];
    const int64_t i = e - g.elem0;
    const double v = self_term_warp(g.vertices, g.types, g.values, i, lane);
    if (lane == 0) g.A[i * g.lda + i] = v;
  }
}

__global__ void k_rhs(const uint8_t* __restrict__ types, const double* __restrict__ values,
                      double* __restrict__ F, int64_t N) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= N) return;
  int t = types[i];
  F[i] = (t == VOLTAGE_FIXED || t == VOLTAGE_FUN || t == MAGNETOSTATIC_POT) ? values[i] : 0.0;
}

// The full right-hand side of solver.py:118-150: voltage rows take their
// value, dielectric rows 0, magnetizable rows -factor(mu) H . n with H the
// pre-existing field at the element's collocation point (field (N, 3) =
// H_x, H_y, H_z at (r, 0, z), or none: zero field) and n its normal.
__global__ void k_rhs_field(const uint8_t* __restrict__ types, const double* __restrict__ values,
                            const double* __restrict__ normal, const double* __restrict__ field,
                            double* __restrict__ F, int64_t N) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int t = types[i];
  double f = 0.0;
  if (t == VOLTAGE_FIXED || t == VOLTAGE_FUN || t == MAGNETOSTATIC_POT) {
    f = values[i];
  } else if (t == MAGNETIZABLE && field) {
    const double hn = field[3 * i] * normal[2 * i] + field[3 * i + 2] * normal[2 * i + 1];
    f = -flux_factor(values[i]) * hn;
  }
  F[i] = f;
}

// ---------------------------------------------------------------- sources
__global__ void k_pack_sources(const double* __restrict__ q, const double* __restrict__ jac,
                               const double* __restrict__ pos, double* __restrict__ src, int64_t N) {
  int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int64_t Nq = N * NQ;
  if (g >= Nq) return;
  src[g] = pos[2 * g];
  src[Nq + g] = pos[2 * g + 1];
  src[2 * Nq + g] = q[g / NQ] * jac[g];
}

// ---------------------------------------------------------------- field
// Potential and field at a point from a slice of sources; returns the raw
// sums (see ring_field_acc).
template <bool POT>
__device__ __forceinline__ void source_sums(double r0, double z0, const double* __restrict__ src, int64_t Nq,
                                            int64_t first, int64_t stride, double& Sr, double& Sz, double& Sp) {
  const double* sr = src;
  const double* sz = src + Nq;
  const double* sw = src + 2 * Nq;
  for (int64_t j = first; j < Nq; j += stride) ring_field_acc<POT>(r0, z0, sr[j], sz[j], sw[j], Sr, Sz, Sp);
}

// One thread per point; source tiles staged through shared memory.
constexpr int FP_THREADS = 256;
template <bool POT>
__global__ void __launch_bounds__(FP_THREADS)
    k_field_points_thread(const double* __restrict__ points, int64_t M, const double* __restrict__ src,
                          int64_t Nq, double* __restrict__ pot, double* __restrict__ field) {
  __shared__ double t_r[FP_THREADS], t_z[FP_THREADS], t_w[FP_THREADS];
  int64_t m = blockIdx.x * (int64_t)FP_THREADS + threadIdx.x;
  double p[3] = {0, 0, 0};
  if (m < M) {
    p[0] = points[3 * m];
    p[1] = points[3 * m + 1];
    p[2] = points[3 * m + 2];
  }
  double r0 = axis_distance(p), z0 = p[2];
  double Sr = 0, Sz = 0, Sp = 0;
  for (int64_t base = 0; base < Nq; base += FP_THREADS) {
    int64_t j = base + threadIdx.x;
    __syncthreads();
    if (j < Nq) {
      t_r[threadIdx.x] = src[j];
      t_z[threadIdx.x] = src[Nq + j];
      t_w[threadIdx.x] = src[2 * Nq + j];
    } else {
      t_r[threadIdx.x] = 1.0;  // harmless ring of zero weight
      t_z[threadIdx.x] = 0.0;
      t_w[threadIdx.x] = 0.0;
    }
    __syncthreads();
    int cnt = Nq - base < FP_THREADS ? int(Nq - base) : FP_THREADS;
#pragma unroll 2
    for (int k = 0; k < cnt; k++) ring_field_acc<POT>(r0, z0, t_r[k], t_z[k], t_w[k], Sr, Sz, Sp);
  }
  if (m < M) finish_field(p, Sr, Sz, Sp, pot, field, m);
}

// One warp per point.
template <bool POT>
__global__ void __launch_bounds__(256)
    k_field_points_warp(const double* __restrict__ points, int64_t M, const double* __restrict__ src, int64_t Nq,
                        double* __restrict__ pot, double* __restrict__ field) {
  const int lane = threadIdx.x & 31;
  const int64_t m = blockIdx.x * (int64_t)8 + threadIdx.x / 32;
  if (m >= M) return;
  const double p[3] = {points[3 * m], points[3 * m + 1], points[3 * m + 2]};
  const double r0 = axis_distance(p);
  double Sr = 0, Sz = 0, Sp = 0;
  source_sums<POT>(r0, p[2], src, Nq, lane, 32, Sr, Sz, Sp);
  Sr = warp_sum(Sr);
  Sz = warp_sum(Sz);
  if (POT) Sp = warp_sum(Sp);
  if (lane == 0) finish_field(p, Sr, Sz, Sp, pot, field, m);
}

// One cluster of CTAs (1, 2, 4 or 8) per point, for a few points: a CTA alone
// would leave the other SMs idle for as long as its 256 threads take (one
// point on 16,000 rings: 35 us with one CTA, 8.5 with eight).  Each CTA's sums
// go to the first one's shared memory and are added there in a fixed order.
constexpr int FP_CLUSTER = 8;
template <bool POT>
__global__ void __launch_bounds__(256)
    k_field_points_cluster(const double* __restrict__ points, const double* __restrict__ src, int64_t Nq,
                           double* __restrict__ pot, double* __restrict__ field) {
  namespace cg = cooperative_groups;
  __shared__ double red[8][3], all[FP_CLUSTER][3];
  cg::cluster_group cl = cg::this_cluster();
  const int ctas = int(cl.num_blocks()), rank = int(cl.block_rank());
  const int64_t m = blockIdx.x / ctas;
  const double p[3] = {points[3 * m], points[3 * m + 1], points[3 * m + 2]};
  const double r0 = axis_distance(p);
  double S[3] = {0, 0, 0};
  source_sums<POT>(r0, p[2], src, Nq, rank * 256 + threadIdx.x, 256 * ctas, S[0], S[1], S[2]);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double v = k < 2 || POT ? warp_sum(S[k]) : 0.0;
    if ((threadIdx.x & 31) == 0) red[threadIdx.x / 32][k] = v;
  }
  __syncthreads();
  cl.sync();  // every CTA of the cluster runs: its shared memory can be written
  if (threadIdx.x < 3) {
    double t = 0;
    for (int k = 0; k < 8; k++) t += red[k][threadIdx.x];
    *cl.map_shared_rank(&all[rank][threadIdx.x], 0) = t;
  }
  cl.sync();
  if (rank == 0 && threadIdx.x == 0) {
    double t[3] = {0, 0, 0};
    for (int c = 0; c < ctas; c++)
      for (int k = 0; k < 3; k++) t[k] += all[c][k];
    finish_field(p, t[0], t[1], t[2], pot, field, m);
  }
}

template <bool POT>
static void launch_points_cluster(const double* points, int64_t M, const double* src, int64_t Nq, double* pot,
                                  double* field, cudaStream_t s) {
  // as many CTAs a point as leave every point's cluster a place on the chip at
  // once and every thread four rings
  unsigned ctas = 1;
  while (ctas < FP_CLUSTER && M * ctas * 2 <= num_sms() && Nq >= int64_t(ctas) * 2 * 256 * 4) ctas *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(M) * ctas);
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = ctas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_field_points_cluster<POT>, points, src, Nq, pot, field);  // errors: launch_status()
}

// ---------------------------------------------------------------- axial
// One block of 256 threads per z point; each thread sums a strided slice of
// the sources, then a block reduction of the 9 partial sums.
__global__ void __launch_bounds__(256)
    k_axial_derivs(const double* __restrict__ z, int64_t Nz, const double* __restrict__ src, int64_t Nq,
                   double* __restrict__ derivs) {
  __shared__ double red[NDERIV][8];
  int64_t iz = blockIdx.x;
  if (iz >= Nz) return;
  double z0 = z[iz];
  double acc[NDERIV];
#pragma unroll
  for (int l = 0; l < NDERIV; l++) acc[l] = 0.0;
  const double* sr = src;
  const double* sz = src + Nq;
  const double* sw = src + 2 * Nq;
  for (int64_t j = threadIdx.x; j < Nq; j += 256) axial_ring(z0, sr[j], sz[j], sw[j], acc);
  int w = threadIdx.x / 32;
#pragma unroll
  for (int l = 0; l < NDERIV; l++) {
    double v = warp_sum(acc[l]);
    if ((threadIdx.x & 31) == 0) red[l][w] = v;
  }
  __syncthreads();
  if (threadIdx.x < NDERIV) {
    double s = 0;
    for (int k = 0; k < 8; k++) s += red[threadIdx.x][k];
    derivs[iz * NDERIV + threadIdx.x] = s;
  }
}

// Quintic Hermite on [0, h] through (y, y', y'') at both ends, in the power
// basis of (x - z_i), highest degree first: the form
// PPoly.from_bernstein_basis(BPoly.from_derivatives(...)).c produces
// (field.py:906-911).
__global__ void k_axial_quintic(const double* __restrict__ d, int64_t Nz, double h, double* __restrict__ c) {
  int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int64_t iv = g / 7;
  int i = int(g % 7);
  if (iv >= Nz - 1) return;
  const double* a = d + iv * NDERIV;
  const double* b = d + (iv + 1) * NDERIV;
  double c0 = a[i], c1 = a[i + 1], c2 = 0.5 * a[i + 2];
  double D0 = b[i] - (c0 + h * (c1 + h * c2));
  double D1 = (b[i + 1] - (c1 + 2 * h * c2)) * h;
  double D2 = (b[i + 2] - 2 * c2) * h * h;
  double A3 = 10 * D0 - 4 * D1 + 0.5 * D2;  // c3 h^3
  double A4 = -15 * D0 + 7 * D1 - D2;       // c4 h^4
  double A5 = 6 * D0 - 3 * D1 + 0.5 * D2;   // c5 h^5
  double ih = 1.0 / h, ih3 = ih * ih * ih;
  double* o = c + (iv * NDERIV + i) * 6;
  o[0] = A5 * ih3 * ih * ih;
  o[1] = A4 * ih3 * ih;
  o[2] = A3 * ih3;
  o[3] = c2;
  o[4] = c1;
  o[5] = c0;
}

// Not-a-knot cubic spline (scipy.interpolate.CubicSpline default) of the
// columns 7 and 8 of d.  Unknowns are the node slopes s_0 .. s_{n-1}; on an
// equal grid with m_i = (y_{i+1} - y_i)/h:
//   s_{i-1} + 4 s_i + s_{i+1} = r_i = 3 (m_{i-1} + m_i),      0 < i < n-1
//   not-a-knot at x_1:      s_0 - s_2 = 2 (m_0 - m_1)
//   not-a-knot at x_{n-2}:  s_{n-1} - s_{n-3} = 2 (m_{n-2} - m_{n-3})
// Eliminating s_0 and s_{n-1} leaves a tridiagonal system in s_1..s_{n-2}
// with first row 4 s_1 + 2 s_2 = m_0 + 5 m_1 and last row
// 2 s_{n-3} + 4 s_{n-2} = 5 m_{n-3} + m_{n-2}.  n = 3 uses the single parabola
// through the three points, n = 2 the straight line (CubicSpline's special
// cases).
//
// The system is all but a Toeplitz one, whose inverse decays like c^k with
// c = 2 - sqrt(3): c^SPLINE_REACH = 7e-19.  Away from the ends each slope is
// therefore the sum s_i = (r_i + sum_k (-c)^k (r_{i-k} + r_{i+k})) / (2 sqrt 3)
// over k <= SPLINE_REACH, all slopes at once; within SPLINE_REACH of an end
// one thread solves the end's rows by elimination, closed by the first slope
// that the sum gives.  Grids too short for that are solved by one thread
// altogether.  (4,601 points: 5.9 ms with one thread eliminating the whole
// column from global memory, 44 us now, most of it the ends' eliminations.)
constexpr int SPLINE_MAX_NZ = 12288;
constexpr int SPLINE_REACH = 32;
constexpr int SPLINE_THREADS = 128;                   // intervals of a CTA
constexpr int SPLINE_SHORT = 4 * SPLINE_REACH + 8;    // up to here: elimination only (in the first CTA)
constexpr int SPLINE_ROWS = SPLINE_THREADS + 1 + 4 * SPLINE_REACH + 16;  // nodes that a CTA looks at

__global__ void __launch_bounds__(SPLINE_THREADS) k_axial_cubic(const double* __restrict__ d, int64_t Nz, double h,
                                                                double* __restrict__ c) {
  __shared__ double sy[SPLINE_ROWS], ss[SPLINE_ROWS], cp[SPLINE_ROWS];
  const int col = 7 + blockIdx.y, n = int(Nz);
  const bool whole = n <= SPLINE_SHORT;
  // nodes first .. first + rows - 1 of the column: this CTA's intervals and two reaches on either side
  const int i0 = blockIdx.x * SPLINE_THREADS;
  const int first = max(0, i0 - 2 * SPLINE_REACH - 4);
  const int rows = min(n, i0 + SPLINE_THREADS + 1 + 2 * SPLINE_REACH + 4) - first;
  for (int q = threadIdx.x; q < rows; q += SPLINE_THREADS) sy[q] = d[int64_t(first + q) * NDERIV + col];
  __syncthreads();
  auto mm = [&](int i) { return (sy[i + 1 - first] - sy[i - first]) / h; };
  auto rhs = [&](int i) {
    if (i == 1) return mm(0) + 5 * mm(1);
    if (i == n - 2) return 5 * mm(n - 3) + mm(n - 2);
    return 3 * (mm(i - 1) + mm(i));
  };
  const int last = whole ? n - 1 : min(n - 1, i0 + SPLINE_THREADS);  // slopes of nodes i0 .. last
  const int top = n - 2 - SPLINE_REACH;                              // the last node that the sum gives
  if (!whole) {
    // the sums (from `top` on, it closes the upper end's rows)
    const double q = -0.26794919243112270647, inv = 0.28867513459481288225;  // -(2 - sqrt 3), 1 / (2 sqrt 3)
    for (int i = max(min(i0, top), SPLINE_REACH + 1) + threadIdx.x; i <= min(last, top); i += SPLINE_THREADS) {
      double a = 0.0;
#pragma unroll 4
      for (int k = SPLINE_REACH; k > 0; k--) a = q * (a + (rhs(i - k) + rhs(i + k)));
      ss[i - first] = inv * (rhs(i) + a);
    }
  }
  __syncthreads();
  auto eliminate = [&](int lo, int hi, bool up) {  // rows lo .. hi from the end at lo (up) or hi, closed at the other
    const int step = up ? 1 : -1, from = up ? lo : hi, to = up ? hi : lo;
    double pc = 0.0, pd = 0.0;
    for (int i = from;; i += step) {
      const bool end = i == 1 || i == n - 2;
      const double a = i == from ? 0.0 : (end ? 2.0 : 1.0);       // towards the row before
      const double b = i == to && end ? 0.0 : (end ? 2.0 : 1.0);  // towards the row after
      const double den = 1.0 / (4.0 - a * pc);
      pd = (rhs(i) - a * pd) * den;
      pc = b * den;
      cp[i - first] = pc;
      ss[i - first] = pd;
      if (i == to) break;
    }
    for (int i = to;; i -= step) {
      const bool open = i == to && (i == 1 || i == n - 2);  // nothing after the other end's row
      if (!open) ss[i - first] -= cp[i - first] * ss[i + step - first];
      if (i == from) break;
    }
  };
  if (n > 3) {
    if (whole) {
      if (threadIdx.x == 0) eliminate(1, n - 2, true);
    } else {
      if (threadIdx.x == 0 && i0 == 0) eliminate(1, SPLINE_REACH, true);
      if (threadIdx.x == 32 && last > top) eliminate(top + 1, n - 2, false);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (n == 2) {
      ss[0] = ss[1] = mm(0);
    } else if (n == 3) {
      const double m0 = mm(0), m1 = mm(1), a = (m1 - m0) / (2 * h);  // the parabola's quadratic coefficient
      ss[0] = m0 - a * h;
      ss[1] = m0 + a * h;
      ss[2] = m1 + a * h;
    } else {
      if (i0 == 0) ss[0] = ss[2] + 2 * (mm(0) - mm(1));
      if (last == n - 1) ss[n - 1 - first] = ss[n - 3 - first] + 2 * (mm(n - 2) - mm(n - 3));
    }
  }
  __syncthreads();
  for (int iv = i0 + threadIdx.x; iv < n - 1 && (whole || iv < i0 + SPLINE_THREADS); iv += SPLINE_THREADS) {
    const double s0 = ss[iv - first], s1 = ss[iv + 1 - first], m = mm(iv);
    double* o = c + (int64_t(iv) * NDERIV + col) * 6;
    o[0] = 0.0;
    o[1] = 0.0;
    o[2] = (s0 + s1 - 2 * m) / (h * h);
    o[3] = (3 * m - 2 * s0 - s1) / h;
    o[4] = s0;
    o[5] = sy[iv - first];
  }
}

// ---------------------------------------------------------------- currents
__global__ void k_pack_current_sources(const double* __restrict__ I, const double* __restrict__ jac,
                                       const double* __restrict__ pos, double* __restrict__ src, int64_t N) {
  int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int64_t Nc = N * NTRI;
  if (g >= Nc) return;
  src[g] = pos[3 * g];
  src[Nc + g] = pos[3 * g + 2];
  src[2 * Nc + g] = I[g / NTRI] * jac[g];
}

// One warp per point: H from current rings (radial.c:55-83).
__global__ void k_current_field_points(const double* __restrict__ points, int64_t M,
                                       const double* __restrict__ src, int64_t Nc, double* __restrict__ field) {
  int64_t m = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / 32;
  int lane = threadIdx.x & 31;
  if (m >= M) return;
  double p[3] = {points[3 * m], points[3 * m + 1], points[3 * m + 2]};
  double r = axis_distance(p);
  double Br = 0, Bz = 0;
  for (int64_t j = lane; j < Nc; j += 32) {
    double hr, hz;
    current_field_ring(r, p[2], src[j], src[Nc + j], hr, hz);
    Br = fma(src[2 * Nc + j], hr, Br);
    Bz = fma(src[2 * Nc + j], hz, Bz);
  }
  Br = warp_sum(Br);
  Bz = warp_sum(Bz);
  if (lane == 0) {
    if (r >= MIN_AXIS) {
      field[3 * m] = p[0] / r * Br;
      field[3 * m + 1] = p[1] / r * Br;
    } else {
      field[3 * m] = 0.0;
      field[3 * m + 1] = 0.0;
    }
    field[3 * m + 2] = Bz;
  }
}

__global__ void __launch_bounds__(256)
    k_current_axial(const double* __restrict__ z, int64_t Nz, const double* __restrict__ src, int64_t Nc,
                    double* __restrict__ derivs) {
  __shared__ double red[NDERIV][8];
  int64_t iz = blockIdx.x;
  if (iz >= Nz) return;
  double z0 = z[iz];
  double acc[NDERIV];
#pragma unroll
  for (int l = 0; l < NDERIV; l++) acc[l] = 0.0;
  for (int64_t j = threadIdx.x; j < Nc; j += 256) current_axial_ring(z0, src[j], src[Nc + j], src[2 * Nc + j], acc);
  int w = threadIdx.x / 32;
#pragma unroll
  for (int l = 0; l < NDERIV; l++) {
    double v = warp_sum(acc[l]);
    if ((threadIdx.x & 31) == 0) red[l][w] = v;
  }
  __syncthreads();
  if (threadIdx.x < NDERIV) {
    double s = 0;
    for (int k = 0; k < 8; k++) s += red[threadIdx.x][k];
    derivs[iz * NDERIV + threadIdx.x] = s;
  }
}

// Axial series evaluation at points (radial.c:312-384).
__global__ void k_axial_points(const double* __restrict__ points, int64_t M, const double* __restrict__ zi,
                               int64_t Nz, const double* __restrict__ coeff, double* __restrict__ pot,
                               double* __restrict__ field) {
  int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (m >= M) return;
  double p[3] = {points[3 * m], points[3 * m + 1], points[3 * m + 2]};
  double dd[NDERIV];
  bool in = axial_eval(p[2], zi, coeff, Nz, dd);
  double r2 = p[0] * p[0] + p[1] * p[1];
  if (pot) pot[m] = in ? axial_potential(dd, r2) : 0.0;
  if (field) {
    double f[3] = {0, 0, 0};
    if (in) axial_field(dd, p, r2, f);
    field[3 * m] = f[0];
    field[3 * m + 1] = f[1];
    field[3 * m + 2] = f[2];
  }
}

}  // namespace tb

// ====================================================================== C ABI
using namespace tb;

extern "C" int tb_mesh_segments(const double* segments, const int64_t* offsets, int64_t S, double* vertices,
                                int64_t N, tb_stream_t stream) {
  if (S < 1 || N < 0 || !segments || !offsets || (N > 0 && !vertices)) return BAD_ARG;
  if (N == 0) return OK;
  k_mesh_segments<<<unsigned((N + 255) / 256), 256, 0, (cudaStream_t)stream>>>(segments, offsets, S, vertices, N);
  return launch_status();
}

extern "C" int tb_jacobian_buffer_radial(const double* vertices, double* jac, double* pos, int64_t N,
                                         tb_stream_t stream) {
  if (N < 0 || (N > 0 && (!vertices || !jac || !pos))) return BAD_ARG;
  if (N == 0) return OK;
  int64_t n = N * NQ;
  k_jacobian_buffer<<<unsigned((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(vertices, jac, pos, N);
  return launch_status();
}

extern "C" int tb_element_targets(const double* vertices, double* target, double* normal, int64_t N,
                                  tb_stream_t stream) {
  if (N < 0 || (N > 0 && !vertices)) return BAD_ARG;
  if (N == 0) return OK;
  k_element_targets<<<unsigned((N + 255) / 256), 256, 0, (cudaStream_t)stream>>>(vertices, target, normal, N);
  return launch_status();
}

extern "C" int tb_fill_matrix_radial(double* A, int64_t lda, const double* vertices, const uint8_t* types,
                                     const double* values, const double* jac, const double* pos, int64_t N,
                                     int64_t row0, int64_t row1, int accumulate, int gauss_diagonal,
                                     tb_stream_t stream) {
  if (N < 0 || lda < N || row0 < 0 || row1 > N || row0 > row1) return BAD_ARG;
  if (N == 0 || row0 == row1) return OK;
  if (!A || !vertices || !types || !values || !jac || !pos) return BAD_ARG;
  // Tall tiles share their columns' staging; a small matrix is cut lower until
  // four CTAs per SM have work (101 elements: 15 us, 60 more with tiles of 64
  // rows; from 3,072 elements on they are 64 rows high).
  const int64_t gx = (N + FILL_TILE - 1) / FILL_TILE;
  int rows = FILL_TILE;
  while (rows > 4 && gx * ((row1 - row0 + rows - 1) / rows) < 4 * num_sms()) rows /= 2;
  dim3 grid(unsigned(gx), unsigned((row1 - row0 + rows - 1) / rows));
  if (grid.y > 65535u) return BAD_ARG;
  k_fill_matrix<<<grid, FILL_THREADS, 0, (cudaStream_t)stream>>>(
      A, lda, vertices, types, values, jac, pos, N, row0, row1, rows, accumulate, gauss_diagonal);
  return launch_status();
}

extern "C" int tb_self_integrals(const double* vertices, const uint8_t* types, const double* values, double* diag,
                                 double* A, int64_t lda, int64_t N, tb_stream_t stream) {
  if (N < 0 || (A && lda < N)) return BAD_ARG;
  if (N == 0) return OK;
  if (!vertices || !types || !values || (!diag && !A)) return BAD_ARG;
  int64_t threads = N * 32;
  k_self_integrals<<<unsigned((threads + 255) / 256), 256, 0, (cudaStream_t)stream>>>(vertices, types, values, diag,
                                                                                      A, lda, N);
  return launch_status();
}

extern "C" int64_t tb_batch_plan(tb_geometry_t* geoms, int n_geoms, int64_t* total_elements) {
  if (!geoms || n_geoms <= 0) return -1;
  int64_t tiles = 0, elems = 0;
  for (int g = 0; g < n_geoms; g++) {
    const int64_t N = geoms[g].N;
    if (N <= 0 || geoms[g].lda < N) return -1;
    geoms[g].tile0 = tiles;
    geoms[g].elem0 = elems;
    tiles += ((N + FILL_TILE - 1) / FILL_TILE) * ((N + FILL_TILE - 1) / FILL_TILE);
    elems += N;
  }
  if (total_elements) *total_elements = elems;
  return tiles;
}

extern "C" int tb_fill_matrix_radial_batched(const tb_geometry_t* geoms, int n_geoms, int64_t total_tiles,
                                             tb_stream_t stream) {
  if (!geoms || n_geoms <= 0 || total_tiles <= 0) return BAD_ARG;
  // persistent: a few CTAs per SM stride over all tiles of all geometries
  int64_t blocks = (int64_t)num_sms() * 8;
  if (blocks > total_tiles) blocks = total_tiles;
  k_fill_matrix_batched<<<unsigned(blocks), FILL_THREADS, 0, (cudaStream_t)stream>>>(geoms, n_geoms, total_tiles);
  return launch_status();
}

extern "C" int tb_self_integrals_batched(const tb_geometry_t* geoms, int n_geoms, int64_t total_elements,
                                         tb_stream_t stream) {
  if (!geoms || n_geoms <= 0 || total_elements <= 0) return BAD_ARG;
  int64_t blocks = (total_elements * 32 + 255) / 256;
  if (blocks > (int64_t)num_sms() * 16) blocks = (int64_t)num_sms() * 16;
  k_self_integrals_batched<<<unsigned(blocks), 256, 0, (cudaStream_t)stream>>>(geoms, n_geoms, total_elements);
  return launch_status();
}

extern "C" int tb_rhs_radial(const uint8_t* types, const double* values, double* F, int64_t N, tb_stream_t stream) {
  if (N < 0 || (N > 0 && (!types || !values || !F))) return BAD_ARG;
  if (N == 0) return OK;
  k_rhs<<<unsigned((N + 255) / 256), 256, 0, (cudaStream_t)stream>>>(types, values, F, N);
  return launch_status();
}

extern "C" int tb_rhs_radial_field(const uint8_t* types, const double* values, const double* normal,
                                   const double* field, double* F, int64_t N, tb_stream_t stream) {
  if (N < 0 || (N > 0 && (!types || !values || !normal || !F))) return BAD_ARG;
  if (N == 0) return OK;
  k_rhs_field<<<unsigned((N + 255) / 256), 256, 0, (cudaStream_t)stream>>>(types, values, normal, field, F, N);
  return launch_status();
}

extern "C" int tb_pack_sources(const double* charges, const double* jac, const double* pos, double* sources,
                               int64_t N, tb_stream_t stream) {
  if (N < 0 || (N > 0 && (!charges || !jac || !pos || !sources))) return BAD_ARG;
  if (N == 0) return OK;
  int64_t n = N * NQ;
  k_pack_sources<<<unsigned((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(charges, jac, pos, sources, N);
  return launch_status();
}

extern "C" int tb_pack_current_sources(const double* currents, const double* jac, const double* pos,
                                       double* sources, int64_t N, tb_stream_t stream) {
  if (N < 0 || (N > 0 && (!currents || !jac || !pos || !sources))) return BAD_ARG;
  if (N == 0) return OK;
  int64_t n = N * NTRI;
  k_pack_current_sources<<<unsigned((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(currents, jac, pos, sources, N);
  return launch_status();
}

extern "C" int tb_current_field_points(const double* points, int64_t M, const double* sources, int64_t Nc,
                                       double* field, tb_stream_t stream) {
  if (M < 0 || Nc < 0) return BAD_ARG;
  if (M == 0) return OK;
  if (!points || !field || (Nc > 0 && !sources)) return BAD_ARG;
  int64_t threads = M * 32;
  k_current_field_points<<<unsigned((threads + 255) / 256), 256, 0, (cudaStream_t)stream>>>(points, M, sources, Nc,
                                                                                            field);
  return launch_status();
}

extern "C" int tb_current_axial_derivatives(const double* z, int64_t Nz, const double* sources, int64_t Nc,
                                            double* derivs, tb_stream_t stream) {
  if (Nz < 0 || Nc < 0 || Nz > 0x7fffffff) return BAD_ARG;
  if (Nz == 0) return OK;
  if (!z || !derivs || (Nc > 0 && !sources)) return BAD_ARG;
  k_current_axial<<<unsigned(Nz), 256, 0, (cudaStream_t)stream>>>(z, Nz, sources, Nc, derivs);
  return launch_status();
}

extern "C" int tb_field_radial_points(const double* points, int64_t M, const double* sources, int64_t Nq,
                                      double* pot, double* field, tb_stream_t stream) {
  if (M < 0 || Nq < 0) return BAD_ARG;
  if (M == 0) return OK;
  if (!points || (Nq > 0 && !sources) || (!pot && !field)) return BAD_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const int sms = num_sms();
  // Enough points to fill the GPU one thread per point: stage sources in
  // shared memory.  Otherwise split each point's sum over a warp or a cluster.
  if (M >= (int64_t)sms * 2048) {
    unsigned g = unsigned((M + FP_THREADS - 1) / FP_THREADS);
    if (pot)
      k_field_points_thread<true><<<g, FP_THREADS, 0, s>>>(points, M, sources, Nq, pot, field);
    else
      k_field_points_thread<false><<<g, FP_THREADS, 0, s>>>(points, M, sources, Nq, pot, field);
  } else if (M >= (int64_t)sms * 16) {
    unsigned g = unsigned((M + 7) / 8);
    if (pot)
      k_field_points_warp<true><<<g, 256, 0, s>>>(points, M, sources, Nq, pot, field);
    else
      k_field_points_warp<false><<<g, 256, 0, s>>>(points, M, sources, Nq, pot, field);
  } else if (pot) {
    launch_points_cluster<true>(points, M, sources, Nq, pot, field, s);
  } else {
    launch_points_cluster<false>(points, M, sources, Nq, pot, field, s);
  }
  return launch_status();
}

extern "C" int tb_axial_derivatives_radial(const double* z, int64_t Nz, const double* sources, int64_t Nq,
                                           double* derivs, tb_stream_t stream) {
  if (Nz < 0 || Nq < 0) return BAD_ARG;
  if (Nz == 0) return OK;
  if (!z || !derivs || (Nq > 0 && !sources)) return BAD_ARG;
  if (Nz > 0x7fffffff) return BAD_ARG;
  k_axial_derivs<<<unsigned(Nz), 256, 0, (cudaStream_t)stream>>>(z, Nz, sources, Nq, derivs);
  return launch_status();
}

extern "C" int tb_axial_coefficients(const double* derivs, int64_t Nz, double dz, double* coeffs,
                                     tb_stream_t stream) {
  if (Nz < 2 || Nz > SPLINE_MAX_NZ || !(dz > 0) || !derivs || !coeffs) return BAD_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  int64_t n = (Nz - 1) * 7;
  k_axial_quintic<<<unsigned((n + 255) / 256), 256, 0, s>>>(derivs, Nz, dz, coeffs);
  const unsigned g = Nz <= SPLINE_SHORT ? 1u : unsigned((Nz - 1 + SPLINE_THREADS - 1) / SPLINE_THREADS);
  k_axial_cubic<<<dim3(g, 2), SPLINE_THREADS, 0, s>>>(derivs, Nz, dz, coeffs);
  return launch_status();
}

extern "C" int tb_axial_field_points(const double* points, int64_t M, const double* z, int64_t Nz,
                                     const double* coeffs, double* pot, double* field, tb_stream_t stream) {
  if (M < 0 || Nz < 2) return BAD_ARG;
  if (M == 0) return OK;
  if (!points || !z || !coeffs || (!pot && !field)) return BAD_ARG;
  k_axial_points<<<unsigned((M + 255) / 256), 256, 0, (cudaStream_t)stream>>>(points, M, z, Nz, coeffs, pot, field);
  return launch_status();
}
