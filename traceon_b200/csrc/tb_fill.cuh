// tb_fill.cuh -- matrix entries of the radial BEM fill: the off-diagonal
// Gauss sums and the singular self terms, shared by the single-
// geometry kernels and the batched persistent solve.
#pragma once

#include "tb_common.cuh"
#include "tb_internal.cuh"

namespace tb {

// An entry (i, j) of the matrix (radial.c:249-310) is the 16-point Gauss sum of
// element j's rings at the collocation point of element i.  How many nodes it
// needs depends on the distance d of that point from the element: the n-point
// rule integrates the kernel's expansion about the element's middle exactly up
// to degree 2 n - 1, and the rest falls like (h / d)^2n with h the element's
// half-length.  FILL_X lists the shorter rules and the d / h from which
// their value equals the 16-point rule's to about 1e-16 (checked in extended
// precision for the potential and the field kernels); on the lens meshes
// 95 % of the pairs of 16,384 elements need three nodes.  Elements whose cubic
// map is not linear in alpha to within eps need more distance (the degree 2 n
// terms then carry powers of eps, fill_column), and those that are not
// straight, or whose given rings are not the map's, always take all 16.
//
// The sums are bound by the FP64 pipe: the fill of 16,384 elements takes 5.5
// ms, 19.7 ms with 16 nodes for every pair (and a series logarithm); 2,501
// magnetizable elements 0.31 and 1.0 ms.
constexpr int FILL_TILE = 64;     // rows and columns of a tile, one CTA of FILL_THREADS
constexpr int FILL_THREADS = 256;
constexpr int FILL_NODES = 3 + 4 + 8;
// rules of 3, 4 and 8 points at d / h >= 240, 50 and 5
__device__ const double FILL_X[FILL_NODES] = {
    -0.77459666924148337704, 0.0, 0.77459666924148337704,
    -0.86113631159405257522, -0.3399810435848562648, 0.3399810435848562648, 0.86113631159405257522,
    -0.96028985649753623168, -0.79666647741362673959, -0.52553240991632898582, -0.18343464249564980494,
    0.18343464249564980494, 0.52553240991632898582, 0.79666647741362673959, 0.96028985649753623168};
__device__ const double FILL_W[FILL_NODES] = {
    0.55555555555555555556, 0.88888888888888888889, 0.55555555555555555556,
    0.34785484513745385737, 0.65214515486254614263, 0.65214515486254614263, 0.34785484513745385737,
    0.10122853629037625915, 0.22238103445337447054, 0.31370664587788728734, 0.36268378337836198297,
    0.36268378337836198297, 0.31370664587788728734, 0.22238103445337447054, 0.10122853629037625915};

// The data of a tile's columns and rows in shared memory.
struct FillTile {
  double r[FILL_NODES][FILL_TILE], z[FILL_NODES][FILL_TILE], w[FILL_NODES][FILL_TILE];  // w: weight x jacobian
  double cr[FILL_TILE], cz[FILL_TILE];           // the elements' middles
  float d3[FILL_TILE], d4[FILL_TILE], d8[FILL_TILE];  // squared distances from which each rule holds
  double tr[FILL_TILE], tz[FILL_TILE], nr[FILL_TILE], nz[FILL_TILE];  // rows: collocation points; normals x factor / pi
  int type[FILL_TILE];
};

enum FillRowType : int { FILL_POT = 0, FILL_FLUX = 1, FILL_UNKNOWN = 2 };

// Squared distance (times h^2 h = |x'| at the middle) limits of the shorter
// rules for an element whose map x(alpha) = c + (k1 alpha + k2 alpha^2 + k3
// alpha^3) / 16: eps = (|k2| + |k3|) / |k1| is its departure from linear,
// bend the part of it across the element.
__device__ __forceinline__ void fill_limits(const Cubic& cu, float& d3, float& d4, float& d8) {
  const double inf = __longlong_as_double(0x7ff0000000000000LL);
  const double l2 = cu.k1[0] * cu.k1[0] + cu.k1[1] * cu.k1[1];
  const double h2 = l2 / 256.0;
  const double eps = (sqrt(cu.k2[0] * cu.k2[0] + cu.k2[1] * cu.k2[1]) + sqrt(cu.k3[0] * cu.k3[0] + cu.k3[1] * cu.k3[1])) /
                     sqrt(l2);
  const double bend = (fabs(cu.k1[0] * cu.k2[1] - cu.k1[1] * cu.k2[0]) + fabs(cu.k1[0] * cu.k3[1] - cu.k1[1] * cu.k3[0])) / l2;
  const float e = float(eps), h2f = float(h2);
  const bool straight = eps <= 1e-4 && bend <= 1e-6 && l2 > 0.0;
  // the largest of eps (h/d)^4, eps^2 (h/d)^2 (three points), and so on, below 1e-16
  const float a3 = fmaxf(240.f, fmaxf(sqrtf(sqrtf(e) * 1e8f), e * 1e8f));
  const float a4 = fmaxf(50.f, fmaxf(powf(e * 1e16f, 1.f / 6.f), fmaxf(sqrtf(e * 1e8f), sqrtf(e * e * e) * 1e8f)));
  const float a8 = fmaxf(5.f, fmaxf(powf(e * 1e16f, 1.f / 14.f), powf(e * e * 1e16f, 1.f / 12.f)));
  d3 = straight ? a3 * a3 * h2f : float(inf);
  d4 = straight ? a4 * a4 * h2f : float(inf);
  d8 = straight ? a8 * a8 * h2f : float(inf);
}

// Stages columns j0 .. of the tile (all threads of the CTA; N columns in all).
// jac, pos: the rings given for the elements, or null: the map's own.
__device__ __forceinline__ void fill_columns(FillTile& s, const double* __restrict__ vertices,
                                             const double* __restrict__ jac, const double* __restrict__ pos, int64_t N,
                                             int64_t j0) {
  for (int e = threadIdx.x; e < FILL_TILE * 4; e += FILL_THREADS) {
    const int c = e >> 2, q = e & 3;  // four lanes per column
    const int64_t j = j0 + c;
    bool same = true;
    if (j < N) {
      Cubic cu;
      cu.load(vertices + j * 12);
      double r, z, jj;
      for (int k = q; k < FILL_NODES; k += 4) {
        cu.point(FILL_X[k], false, r, z, jj);
        s.r[k][c] = r;
        s.z[k][c] = z;
        s.w[k][c] = FILL_W[k] * jj;
      }
      if (jac) {
        for (int k = q; k < NQ; k += 4) {
          cu.point(gauss_x(k), false, r, z, jj);
          const int64_t g = j * NQ + k;
          const double size = 1e-14 * (fabs(r) + fabs(z));
          same = same && fabs(pos[2 * g] - r) <= size && fabs(pos[2 * g + 1] - z) <= size &&
                 fabs(jac[g] - gauss_w(k) * jj) <= 1e-13 * jj;
        }
      }
      if (q == 0) {
        cu.point(0.0, false, r, z, jj);
        s.cr[c] = r;
        s.cz[c] = z;
        fill_limits(cu, s.d3[c], s.d4[c], s.d8[c]);
      }
    } else if (q == 0) {
      s.cr[c] = s.cz[c] = 0.0;
    }
    const unsigned quad = 0xfu << (threadIdx.x & 28);
    same = (__ballot_sync(0xffffffffu, same) & quad) == quad;
    if (q == 0 && !same) s.d3[c] = s.d4[c] = s.d8[c] = __int_as_float(0x7f800000);
  }
}

// Stages rows i0 .. i1 - 1.
__device__ __forceinline__ void fill_rows(FillTile& s, const double* __restrict__ vertices,
                                          const uint8_t* __restrict__ types, const double* __restrict__ values,
                                          int64_t i0, int64_t i1) {
  for (int q = threadIdx.x; q < FILL_TILE; q += FILL_THREADS) {
    const int64_t i = i0 + q;
    if (i >= i1) continue;
    Cubic cu;
    cu.load(vertices + i * 12);
    double tj, nr = 0.0, nz = 0.0;
    cu.point(0.0, false, s.tr[q], s.tz[q], tj);
    const int t = types[i];
    int kind = FILL_UNKNOWN;
    if (t == VOLTAGE_FIXED || t == VOLTAGE_FUN || t == MAGNETOSTATIC_POT) {
      kind = FILL_POT;
    } else if (t == DIELECTRIC || t == MAGNETIZABLE) {
      kind = FILL_FLUX;
      cu.normal(0.0, nr, nz);
      const double f = flux_factor(values[i]) * INV_PI;
      // E_r = r0 Sr / pi, E_z = -Sz / pi (ring_field_acc)
      nr = s.tr[q] >= MIN_AXIS ? f * nr * s.tr[q] : 0.0;
      nz = -f * nz;
    }
    s.nr[q] = nr;
    s.nz[q] = nz;
    s.type[q] = kind;
  }
}

// Entry (row q, column c) of the tile; vertices, jac, pos: column j's, for the
// pairs that take all 16 rings.
__device__ __forceinline__ double fill_pair(const FillTile& s, int q, int c, const double* __restrict__ vertices,
                                            const double* __restrict__ jac, const double* __restrict__ pos, int64_t j) {
  const double tr = s.tr[q], tz = s.tz[q];
  const double dr = tr - s.cr[c], dz = tz - s.cz[c];
  const float d2 = float(fma(dr, dr, dz * dz));
  int k = 0, n = 16;
  if (d2 >= s.d3[c]) {
    n = 3;
  } else if (d2 >= s.d4[c]) {
    k = 3;
    n = 4;
  } else if (d2 >= s.d8[c]) {
    k = 7;
    n = 8;
  }
  const int kind = s.type[q];
  double a = 0.0, b = 0.0, unused = 0.0;
  if (n < 16) {
    if (kind == FILL_POT) {
#pragma unroll 1
      for (const int end = k + n; k < end; k++) a = fma(s.w[k][c], ring_pot_nopi(tr, tz, s.r[k][c], s.z[k][c]), a);
    } else {
#pragma unroll 1
      for (const int end = k + n; k < end; k++)
        ring_field_acc<false>(tr, tz, s.r[k][c], s.z[k][c], s.w[k][c], a, b, unused);
    }
  } else {
    Cubic cu;
    if (!jac) cu.load(vertices + j * 12);
#pragma unroll 2
    for (k = 0; k < NQ; k++) {
      double r, z, w;
      if (jac) {
        const int64_t g = j * NQ + k;
        r = pos[2 * g];
        z = pos[2 * g + 1];
        w = jac[g];
      } else {
        cu.point(gauss_x(k), false, r, z, w);
        w *= gauss_w(k);
      }
      if (kind == FILL_POT)
        a = fma(w, ring_pot_nopi(tr, tz, r, z), a);
      else
        ring_field_acc<false>(tr, tz, r, z, w, a, b, unused);
    }
  }
  if (kind == FILL_POT) return a * INV_PI;
  return kind == FILL_FLUX ? fma(s.nr[q], a, s.nz[q] * b) : __longlong_as_double(0x7ff8000000000000LL);
}

// ---------------------------------------------------------------- self terms
// Composite 16-point Gauss-Legendre on [-1, 0] and [0, 1], each split into
// the intervals [4^-(m+1), 4^-m], m < SELF_LEVELS, plus [0, 4^-L].  The self
// integrand is smooth + smooth * log|alpha|; over an interval whose ends are
// 1 : 4 the rule's error for the logarithm falls like 3^-32, so each piece is
// integrated to ~1e-17 relative (as with twice as many intervals 1 : 2), and
// the innermost piece contributes ~4^-L L log 4 of the total.
constexpr int SELF_LEVELS = 26;
constexpr int SELF_POINTS = 2 * (SELF_LEVELS + 1) * NQ;

// j x (potential of the ring at the offset (dr, dz) from the collocation
// point), or j x (n . E) with (fr, fz) the normal times the row's factor as in
// fill_rows; without the 1 / pi of the potential.
__device__ __forceinline__ double self_integrand(const Cubic& c, double tr, double fr, double fz, bool flux,
                                                 double alpha) {
  double dr, dz, j;
  c.point(alpha, true, dr, dz, j);
  const double rs = tr + dr, dz2 = dz * dz, rho2 = fma(dr, dr, dz2), s = rs + tr, D = fma(s, s, dz2);
  const double g = rsqrt_h3(rho2 * rho2 * D), rD = rho2 * g, t = rho2 * rD * rD, t2 = t * t, t4 = t2 * t2;
  const double L = neglog_tab(t);
  if (!flux) return j * rs * rD * fma(L, estrin8(C_KB, t, t2, t4), estrin8(C_KA, t, t2, t4));
  const double E = fma(L, estrin8(C_EB, t, t2, t4), estrin8(C_EA, t, t2, t4));
  const double G = fma(L, estrin10(C_GB, t, t2, t4), estrin10(C_GA, t, t2, t4));
  const double q = 4.0 * rs;
  return j * rs * g * fma(fr * (rD * rD), fma(q * rs * t, G, fma(-q, dr, rho2) * E), fz * (dz * E));
}

// Self term of element i by one warp (all lanes call it; every lane gets the value).
__device__ inline double self_term_warp(const double* __restrict__ vertices, const uint8_t* __restrict__ types,
                                        const double* __restrict__ values, int64_t i, int lane) {
  Cubic c;
  c.load(vertices + i * 12);
  double tr, tz, tj, nr, nz;
  c.point(0.0, false, tr, tz, tj);
  c.normal(0.0, nr, nz);
  int ty = types[i];
  bool flux = ty == DIELECTRIC || ty == MAGNETIZABLE;
  bool pot = ty == VOLTAGE_FIXED || ty == VOLTAGE_FUN || ty == MAGNETOSTATIC_POT;
  const double f = flux ? flux_factor(values[i]) * INV_PI : 0.0;
  const double fr = tr >= MIN_AXIS ? f * nr * tr : 0.0, fz = -f * nz;
  double acc = 0.0;
  for (int p = lane; p < SELF_POINTS; p += 32) {
    int k = p % NQ;
    int lvl = (p / NQ) % (SELF_LEVELS + 1);
    double sgn = (p / (NQ * (SELF_LEVELS + 1))) ? 1.0 : -1.0;
    double hi = ldexp(1.0, -2 * lvl);
    double lo = lvl == SELF_LEVELS ? 0.0 : 0.25 * hi;
    double half = 0.5 * (hi - lo), mid = 0.5 * (hi + lo);
    double a = sgn * (mid + half * gauss_x(k));
    acc += half * gauss_w(k) * self_integrand(c, tr, fr, fz, flux, a);
  }
  acc = warp_sum(acc);
  double v = flux ? acc - 1.0 : acc * INV_PI;
  if (!flux && !pot) v = __longlong_as_double(0x7ff8000000000000LL);  // unknown type: NaN
  return v;
}

}  // namespace tb
