// tb_tree.cu -- builds the ring tree of tb_tree.cuh and evaluates fields
// through it.
//
//   k_tree_elements  one half-warp per element: its rings copied into chunks,
//                    its axis, whether a run starts at it
//   k_tree_runs      one CTA: runs numbered, node slots assigned (prefix sums)
//   k_tree_nodes     one warp per node: extent and proxies, first the nodes of
//                    at most TREE_MID elements from their rings, then, in a
//                    second launch, the larger ones from these nodes' proxies
//   k_field_points_tree  1 to 32 warps per point
//
// The build reads the rings once and interpolates them log2(TREE_MID /
// TREE_LEAF) + 1 times; it is latency-bound (four short launches: 24 us for
// 1,000 elements, 100 us for 16,384).  A point near straight stretches then
// sums some 400 rings however many there are: 2^18 points on 16,384 elements
// of a lens take 0.9 ms where the direct sums took 410, 9,797 points on 1,537
// elements 0.08 ms instead of 1.8.
#include <cooperative_groups.h>

#include "tb_tree.cuh"
#include "../../include/traceon_b200.h"

namespace tb {

__device__ __forceinline__ double half_min(double v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double half_max(double v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// The axis of 16 rings (one per lane of a half-warp) and the middle of their
// constant coordinate.
__device__ __forceinline__ int rings_axis(double r, double z, double w, double& mid) {
  const double r1 = half_min(r), r2 = half_max(r), z1 = half_min(z), z2 = half_max(z);
  const unsigned lanes = 0xffffu << (threadIdx.x & 16);
  const bool fine = isfinite(r) && isfinite(z) && isfinite(w);
  const bool ok = (__ballot_sync(0xffffffffu, fine) & lanes) == lanes && r1 >= 0.0;
  mid = 0.0;
  if (!ok) return TREE_DIRECT;
  if (r2 - r1 <= TREE_TOL * r2) {
    mid = 0.5 * (r1 + r2);
    return TREE_HORIZONTAL;
  }
  if (z2 - z1 <= TREE_TOL * fmax(fabs(z1), fabs(z2))) {
    mid = 0.5 * (z1 + z2);
    return TREE_VERTICAL;
  }
  return TREE_DIRECT;
}

// offsets (groups + 1): the first ring of each group; null: one group.
__global__ void __launch_bounds__(256)
    k_tree_elements(Tree T, const double* __restrict__ src, const int64_t* __restrict__ offsets) {
  const int64_t nq = int64_t(T.n) * TREE_P;
  const int e = int((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / TREE_P), k = threadIdx.x % TREE_P;
  const bool in = e < T.n;
  const int64_t j = int64_t(in ? e : 0) * TREE_P + k;
  const double r = src[j], z = src[nq + j], w = src[2 * nq + j];
  double mid, pmid;
  const int axis = rings_axis(r, z, w, mid);
  const int64_t q = j >= TREE_P ? j - TREE_P : j;  // the element before
  const int paxis = rings_axis(src[q], src[nq + q], src[2 * nq + q], pmid);
  if (!in) return;
  double* c = T.chunk + int64_t(e) * TREE_CHUNK;
  c[k] = r;
  c[TREE_P + k] = z;
  c[2 * TREE_P + k] = w;
  if (k) return;
  bool start = e == 0 || axis != paxis ||
               (axis != TREE_DIRECT && fabs(mid - pmid) > TREE_TOL * fmax(fabs(mid), fabs(pmid)));
  if (!start && offsets) {
    int lo = 0, hi = T.groups;  // the last group with offset <= j
    while (lo < hi) {
      const int m = (lo + hi + 1) / 2;
      if (offsets[m] <= j)
        lo = m;
      else
        hi = m - 1;
    }
    start = offsets[lo] == j;
  }
  T.kind[e] = uint8_t(axis + (start ? 4 : 0));
}

constexpr int TR_THREADS = 1024;

// Exclusive prefix sum of v over the CTA; total receives the sum.
__device__ __forceinline__ int cta_scan(int v, int* warp_sums, int& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x / 32;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) warp_sums[w] = x;
  __syncthreads();
  if (w == 0) {
    int s = warp_sums[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    warp_sums[lane] = s;
  }
  __syncthreads();
  total = warp_sums[31];
  return x - v + (w ? warp_sums[w - 1] : 0);
}

// Node slots of a run of m elements: a complete binary tree over
// 2^ceil(log2 m) elements down to TREE_LEAF of them (a direct run: its root).
__device__ __forceinline__ int run_levels(int m) { return m <= 1 ? 0 : 32 - __clz(m - 1); }
__device__ __forceinline__ int run_slots(int m, int axis) {
  const int l = run_levels(m);
  return axis == TREE_DIRECT || l < 2 ? 1 : (1 << (l - 1)) - 1;
}

// Whether the tree is of use is known here only: every point sums at least one
// chunk for each straight run and all chunks of the others, and each of a
// team's eight warps looks at every run (some eighth of a chunk's time).  Where
// that is more than all elements, each group becomes one run without proxies:
// its rings in the given order (elements in random order, 800 of them, one
// electron with eight warps: 2.0 times the direct sums' time through their runs
// of one element each, 1.1 so; the tracer sums ring by ring then).
__global__ void __launch_bounds__(TR_THREADS) k_tree_runs(Tree T, const int64_t* __restrict__ offsets) {
  __shared__ int sums[32];
  __shared__ int least;  // those chunks
  if (threadIdx.x == 0) least = 0;
  int runs, total;
  bool useless = false;
  for (;;) {
    runs = 0;
    int mine = 0;
    for (int base = 0; base < T.n; base += TR_THREADS) {
      const int e = base + threadIdx.x;
      const int k = e < T.n ? T.kind[e] : TREE_HORIZONTAL, s = k >> 2;
      mine += (k & 3) == TREE_DIRECT ? 1 : s;
      const int at = runs + cta_scan(s, sums, total);
      if (s) T.run_e0[at] = e;
      runs += total;
    }
    if (useless) break;
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (mine && (threadIdx.x & 31) == 0) atomicAdd(&least, mine);
    __syncthreads();
    useless = least + runs > T.n;
    if (!useless) break;
    for (int e = threadIdx.x; e < T.n; e += TR_THREADS) T.kind[e] = uint8_t(TREE_DIRECT + (e == 0 ? 4 : 0));
    __syncthreads();
    if (offsets)
      for (int g = threadIdx.x; g < T.groups; g += TR_THREADS) {
        const int64_t e = offsets[g] / TREE_P;
        if (e >= 0 && e < T.n) T.kind[e] = uint8_t(TREE_DIRECT + 4);
      }
    __syncthreads();
  }
  if (threadIdx.x == 0) T.run_e0[runs] = T.n;
  __syncthreads();
  int slots = 0;
  for (int base = 0; base < runs; base += TR_THREADS) {
    const int i = base + threadIdx.x;
    int s = 0;
    if (i < runs) {
      const int e0 = T.run_e0[i];
      s = run_slots(T.run_e0[i + 1] - e0, T.kind[e0] & 3);
    }
    const int at = slots + cta_scan(s, sums, total);
    if (i < runs) T.run_slot[i] = at;
    slots += total;
  }
  int split = 0;
  if (offsets)
    for (int g = threadIdx.x; g <= T.groups; g += TR_THREADS) split |= offsets[g] % TREE_P != 0;
  split = __syncthreads_or(split);
  if (threadIdx.x == 0) {
    T.run_slot[runs] = slots;
    T.count[0] = runs;
    T.count[1] = slots;
    T.count[2] = split != 0 || useless;
  }
  for (int g = threadIdx.x; g <= T.groups; g += TR_THREADS) {
    const int64_t e = g == T.groups && !offsets ? T.n : (offsets ? offsets[g] / TREE_P : 0);
    int lo = 0, hi = runs;  // the first run that starts at or after e
    while (lo < hi) {
      const int m = (lo + hi) / 2;
      if (T.run_e0[m] < e)
        lo = m + 1;
      else
        hi = m;
    }
    T.group_run[g] = lo;
  }
}

__device__ __forceinline__ double warp_min(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Chebyshev nodes of the first kind and their barycentric weights.
__device__ __forceinline__ double cheb_x(int m) { return cospi((2 * m + 1) / (2.0 * TREE_P)); }

// MID false: nodes of at most TREE_MID elements, from their rings; true: the
// larger ones, from the proxies of the nodes of TREE_MID elements below them.
template <bool MID>
__global__ void __launch_bounds__(128) k_tree_nodes(Tree T) {
  __shared__ double sx[TREE_P], sb[TREE_P];
  if (blockIdx.x * (int64_t)(blockDim.x / 32) >= T.count[1]) return;
  if (threadIdx.x < TREE_P) {
    sx[threadIdx.x] = cheb_x(threadIdx.x);
    sb[threadIdx.x] = sinpi((2 * threadIdx.x + 1) / (2.0 * TREE_P)) * (threadIdx.x & 1 ? -1.0 : 1.0);
  }
  __syncthreads();
  const int slot = int((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / 32), lane = threadIdx.x & 31;
  if (slot >= T.count[1]) return;
  int lo = 0, hi = T.count[0] - 1;  // the run that owns the slot
  while (lo < hi) {
    const int m = (lo + hi + 1) / 2;
    if (T.run_slot[m] <= slot)
      lo = m;
    else
      hi = m - 1;
  }
  const int base = T.run_slot[lo], run0 = T.run_e0[lo], m = T.run_e0[lo + 1] - run0;
  const int axis = T.kind[run0] & 3, levels = run_levels(m);
  TreeNode nd;
  nd.c = nd.v = 0.0;
  nd.h = 0.f;
  nd.reach = __int_as_float(0x7f800000);  // +inf: never by proxies
  if (axis == TREE_DIRECT) {
    nd.tag = 8 * m + 4 + axis;
    nd.link = run0;
    if (!MID && lane == 0) {
      T.node[slot] = nd;
      T.aux[slot] = TreeAux{0.0, 0.0, 0.0, 0.0};
    }
    return;
  }
  const int heap = slot - base + 1, depth = 31 - __clz(heap), span = 1 << (levels - depth);
  if ((span > TREE_MID) != MID) return;
  const int first = (heap - (1 << depth)) * span;
  int ne = m - first;
  ne = ne < 0 ? 0 : (ne > span ? span : ne);
  nd.tag = 8 * ne + (span > TREE_LEAF ? 0 : 4) + axis;
  nd.link = span > TREE_LEAF ? base + 2 * heap - 1 : run0 + first;
  if (ne == 0) {
    if (lane == 0) {
      T.node[slot] = nd;
      T.aux[slot] = TreeAux{0.0, 0.0, 0.0, 0.0};
    }
    return;
  }
  const int off_u = axis == TREE_HORIZONTAL ? TREE_P : 0, off_v = TREE_P - off_u;
  // the node's sources: chunks first_chunk .. + chunks - 1
  int first_chunk = run0 + first, chunks = ne;
  double umin = 1e300, umax = -1e300, vmin = 1e300, vmax = -1e300, wabs = 0.0, wv = 0.0;
  if (MID) {
    const int ratio = span / TREE_MID;
    const int s0 = base + (heap * ratio) - 1;  // the first node of TREE_MID elements below
    chunks = (ne + TREE_MID - 1) / TREE_MID;
    first_chunk = T.n + s0;
    for (int i = lane; i < chunks; i += 32) {
      const TreeNode c = T.node[s0 + i];
      const TreeAux x = T.aux[s0 + i];
      umin = fmin(umin, c.c - x.h);
      umax = fmax(umax, c.c + x.h);
      vmin = fmin(vmin, x.vmin);
      vmax = fmax(vmax, x.vmax);
      wabs += x.wabs;
      wv = fma(x.wabs, c.v, wv);
    }
  } else {
    for (int i = lane; i < chunks * TREE_P; i += 32) {
      const double* p = T.chunk + int64_t(first_chunk + i / TREE_P) * TREE_CHUNK + i % TREE_P;
      const double u = p[off_u], v = p[off_v], w = fabs(p[2 * TREE_P]);
      umin = fmin(umin, u);
      umax = fmax(umax, u);
      vmin = fmin(vmin, v);
      vmax = fmax(vmax, v);
      wabs += w;
      wv = fma(w, v, wv);
    }
  }
  umin = warp_min(umin);
  umax = warp_max(umax);
  vmin = warp_min(vmin);
  vmax = warp_max(vmax);
  wabs = warp_sum(wabs);
  wv = warp_sum(wv);
  const double c = 0.5 * (umin + umax), h = 0.5 * (umax - umin), ih = h > 0.0 ? 1.0 / h : 0.0;
  double v = wv / wabs;
  if (!(vmin <= v && v <= vmax)) v = 0.5 * (vmin + vmax);  // no charge, or out of range
  nd.c = c;
  nd.v = v;
  nd.h = float(h);
  if (ne > 1) nd.reach = fmaxf(TREE_KAPPA * float(h), TREE_JITTER * float(vmax - vmin));
  // W_m = sum_j w_j l_m(x_j), l_m(x) = (b_m / (x - x_m)) / sum_k b_k / (x - x_k)
  double W[TREE_P];
#pragma unroll
  for (int k = 0; k < TREE_P; k++) W[k] = 0.0;
  for (int i = lane; i < chunks * TREE_P; i += 32) {
    const double* p = T.chunk + int64_t(first_chunk + i / TREE_P) * TREE_CHUNK + i % TREE_P;
    const double x = (p[off_u] - c) * ih, w = p[2 * TREE_P];
    double q[TREE_P], s = 0.0;
    int hit = -1;
#pragma unroll
    for (int k = 0; k < TREE_P; k++) {
      const double d = x - sx[k];
      if (d == 0.0) hit = k;
      q[k] = sb[k] * rcp_nr(d == 0.0 ? 1.0 : d);
      s += q[k];
    }
    const double f = w / s;
#pragma unroll
    for (int k = 0; k < TREE_P; k++) W[k] += hit < 0 ? f * q[k] : (hit == k ? w : 0.0);
  }
  double mine = 0.0;
#pragma unroll
  for (int k = 0; k < TREE_P; k++) {
    const double t = warp_sum(W[k]);
    if (lane == k) mine = t;
  }
  if (lane < TREE_P) {
    double* o = T.chunk + int64_t(T.n + slot) * TREE_CHUNK + lane;
    o[off_u] = fma(h, sx[lane], c);
    o[off_v] = v;
    o[2 * TREE_P] = mine;
  }
  if (lane == 0) {
    T.node[slot] = nd;
    T.aux[slot] = TreeAux{h, wabs, vmin, vmax};
  }
}

int tree_build(const Tree& T, const double* src, const int64_t* offsets, cudaStream_t s) {
  const int64_t threads = int64_t(T.n) * TREE_P;
  k_tree_elements<<<unsigned((threads + 255) / 256), 256, 0, s>>>(T, src, offsets);
  k_tree_runs<<<1, TR_THREADS, 0, s>>>(T, offsets);
  const unsigned g = unsigned((int64_t(T.n) * 32 + 127) / 128);
  k_tree_nodes<false><<<g, 128, 0, s>>>(T);
  if (T.n > TREE_MID) k_tree_nodes<true><<<g, 128, 0, s>>>(T);
  return launch_status();
}

// PARTS warps per point, 1 to 32: what fills the chip's resident warps, so that
// few points on a mesh without straight stretches are not left to one warp
// each (4,096 elements of arcs: 64 points 960 us with one warp a point, 67 with
// 32, the direct sums 150; 512 points 960, 296 with four, 340).  16 and 32 are
// a cluster of CTAs.
constexpr int FT_WARPS = 8;  // of a CTA, two CTAs a SM

template <bool POT, int PARTS>
__global__ void __launch_bounds__(32 * FT_WARPS, 2)
    k_field_points_tree(Tree T, const double* __restrict__ points, int64_t M, double* __restrict__ pot,
                        double* __restrict__ field) {
  namespace cg = cooperative_groups;
  constexpr int CTAS = PARTS > FT_WARPS ? PARTS / FT_WARPS : 1, PER_CTA = PARTS > FT_WARPS ? 1 : FT_WARPS / PARTS;
  __shared__ TreeScratch sc[FT_WARPS];
  __shared__ double red[PARTS > 1 ? FT_WARPS * CTAS : 1][3];
  const int w = threadIdx.x / 32, lane = threadIdx.x & 31;
  const int part = (CTAS > 1 ? FT_WARPS * int(blockIdx.x % CTAS) : 0) + w % (PARTS / CTAS);
  const int runs = T.count[0];
  const int point = w * CTAS / PARTS;  // of the CTA's; where warps share one they all stay in the loop together
  for (int64_t m = blockIdx.x / CTAS * (int64_t)PER_CTA + point; (PARTS > 1 ? m - point : m) < M;
       m += int64_t(gridDim.x / CTAS) * PER_CTA) {
    const bool in = PARTS == 1 || m < M;
    double p[3], Sr = 0, Sz = 0, Sp = 0;
    if (in) {
      for (int k = 0; k < 3; k++) p[k] = points[3 * m + k];
      const double r0 = axis_distance(p);
      tree_sums<POT>(T, 0, runs, r0, p[2], sc[w], part, PARTS, Sr, Sz, Sp);
      Sr = warp_sum(Sr);
      Sz = warp_sum(Sz);
      if (POT) Sp = warp_sum(Sp);
    }
    if (PARTS > 1) {  // the first of the point's warps adds them up
      if (CTAS > 1) cg::this_cluster().sync();  // the other CTAs run, and the last sums are taken
      if (lane == 0) {
        double* to = &red[CTAS > 1 ? part : w][0];
        if (CTAS > 1) to = cg::this_cluster().map_shared_rank(to, 0);
        to[0] = Sr;
        to[1] = Sz;
        to[2] = Sp;
      }
      if (CTAS > 1)
        cg::this_cluster().sync();
      else
        __syncthreads();
      if (part == 0) {
        for (int k = 1; k < PARTS; k++) {
          Sr += red[w + k][0];
          Sz += red[w + k][1];
          Sp += red[w + k][2];
        }
      }
      if (CTAS == 1) __syncthreads();
    }
    if (in && part == 0 && lane == 0) finish_field(p, Sr, Sz, Sp, pot, field, m);
  }
}

template <int PARTS>
static void launch_points_tree(const Tree& T, const double* points, int64_t M, double* pot, double* field,
                               cudaStream_t s) {
  constexpr int CTAS = PARTS > FT_WARPS ? PARTS / FT_WARPS : 1;
  int64_t blocks = (M * PARTS + FT_WARPS - 1) / FT_WARPS;
  const int64_t resident = (int64_t)num_sms() * 2 / CTAS * CTAS;
  if (blocks > resident) blocks = resident;
  const unsigned threads = 32 * FT_WARPS;
  if (CTAS == 1) {
    if (pot)
      k_field_points_tree<true, PARTS><<<unsigned(blocks), threads, 0, s>>>(T, points, M, pot, field);
    else
      k_field_points_tree<false, PARTS><<<unsigned(blocks), threads, 0, s>>>(T, points, M, pot, field);
    return;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(blocks));
  cfg.blockDim = dim3(threads);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CTAS;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (pot)  // errors: launch_status()
    cudaLaunchKernelEx(&cfg, k_field_points_tree<true, PARTS>, T, points, M, pot, field);
  else
    cudaLaunchKernelEx(&cfg, k_field_points_tree<false, PARTS>, T, points, M, pot, field);
}

}  // namespace tb

using namespace tb;

extern "C" int64_t tb_field_points_workspace(int64_t M, int64_t Nq) {
  // The line between the two: the build's some 40 us (14 where the tree turns
  // out to be of no use) against the pairs that it saves.  64 points on 4,096
  // elements, 4.2e6 pairs: 60 us on a lens, 67 on arcs, cones or elements in
  // random order, 150 by the direct sums; 2,000 points 77, 1,140 and 1,165.
  if (M <= 0 || Nq <= 0 || Nq % TREE_P != 0 || Nq / TREE_P > TREE_MAX_ELEMENTS) return 0;
  if (M < 64 || double(M) * double(Nq) < 4e6) return 0;
  return tree_layout(Nq / TREE_P, 1, nullptr, nullptr);
}

extern "C" int tb_field_radial_points_ws(const double* points, int64_t M, const double* sources, int64_t Nq,
                                         double* pot, double* field, void* work, int64_t work_bytes,
                                         tb_stream_t stream) {
  const int64_t need = tb_field_points_workspace(M, Nq);
  if (!work || need == 0) return tb_field_radial_points(points, M, sources, Nq, pot, field, stream);
  if (!points || !sources || (!pot && !field) || work_bytes < need || reinterpret_cast<uintptr_t>(work) % 16 != 0)
    return BAD_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  Tree T;
  tree_layout(Nq / TREE_P, 1, static_cast<char*>(work), &T);
  const int st = tree_build(T, sources, nullptr, s);
  if (st != OK) return st;
  const int64_t warps = (int64_t)num_sms() * 2 * FT_WARPS;  // resident on the chip
  if (M * 32 <= warps)
    launch_points_tree<32>(T, points, M, pot, field, s);
  else if (M * 16 <= warps)
    launch_points_tree<16>(T, points, M, pot, field, s);
  else if (M * 8 <= warps)
    launch_points_tree<8>(T, points, M, pot, field, s);
  else if (M * 4 <= warps)
    launch_points_tree<4>(T, points, M, pot, field, s);
  else if (M * 2 <= warps)
    launch_points_tree<2>(T, points, M, pot, field, s);
  else
    launch_points_tree<1>(T, points, M, pot, field, s);
  return launch_status();
}
