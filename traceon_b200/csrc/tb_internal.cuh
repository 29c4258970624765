// tb_internal.cuh -- small device and host helpers shared by the kernels.
#pragma once

#include <cuda_runtime.h>
#include <atomic>
#include "tb_common.cuh"

namespace tb {

// Bounded waits inside kernels (an MMA chain's completion, a pipeline
// stage, a flag another CTA publishes) give up after this many SM clock
// cycles: ~1 s at 1.9 GHz, far beyond any wait of a healthy launch.
constexpr long long DEFAULT_WAIT_CYCLES = 2000000000LL;
// Waits that drain work already in flight before shared or tensor memory
// is given up (after a failure too) always use the default bound.
constexpr long long DRAIN_WAIT_CYCLES = DEFAULT_WAIT_CYCLES;

// The limit of the progress waits, read on the host at every launch and
// passed to the kernel (tb_set_wait_limit sets it; one value per process).
inline std::atomic<long long>& wait_limit_cycles() {
  static std::atomic<long long> v{DEFAULT_WAIT_CYCLES};
  return v;
}
inline long long wait_limit() { return wait_limit_cycles().load(std::memory_order_relaxed); }

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Distance of p from the axis, with its rounding spelled out: a point may be
// so close to a ring that the last bit of r0 shows in the field, and all sums
// at one point are to see the same one.
__device__ __forceinline__ double axis_distance(const double* p) { return sqrt(fma(p[0], p[0], p[1] * p[1])); }

// Potential and field at p from the raw sums of ring_field_acc.
__device__ __forceinline__ void finish_field(const double* p, double Sr, double Sz, double Sp, double* pot,
                                             double* field, int64_t m) {
  if (pot) pot[m] = Sp * INV_PI;
  if (field) {
    const bool off_axis = axis_distance(p) >= MIN_AXIS;  // not where a coordinate is no number
    const double er = Sr * INV_PI;                       // E_r / r
    field[3 * m] = off_axis ? p[0] * er : 0.0;
    field[3 * m + 1] = off_axis ? p[1] * er : 0.0;
    field[3 * m + 2] = -Sz * INV_PI;
  }
}

// Status of the last kernel launch on this thread.
inline int launch_status() {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? OK : CUDA_ERR;
}

// Number of SMs of the current device (cached per device).
inline int num_sms() {
  static int cache[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cache[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cache[dev] = n;
  }
  return cache[dev];
}

// Axial series (radial.c:312-384): locate the interval of z on the equally
// spaced grid zi and evaluate the derivative polynomials first .. 8 (the
// field needs 1 .. 8, the potential 0, 2, 4, 6, 8).  Returns false outside
// [zi[0], zi[Nz-1]].
//
// On the device every thread reads its own interval's rows, so a warp's loads
// touch 32 lines each and are bound by the L1's tag lookups, not by bytes:
// a row's six coefficients are read as three pairs (rows start at multiples
// of 48 bytes; a table that is not 16-byte aligned takes single loads).
// Without derivative 0 (the field) a row's other 384 bytes are read 32 at a
// time: eleven loads at the 32-byte boundaries inside and two of 16 bytes,
// 13 lookups a lane instead of 24.  Rows start at multiples of 432 bytes, so
// the boundary lies at the first byte or 16 behind it, row by row, and a
// select puts the pairs in place.
//
// grid: on the device, {z_0, z_last, dz, 1 / dz} where a kernel has them at
// hand (axial_grid), or null.
__host__ __device__ inline bool axial_eval(double z, const double* zi, const double* coeff, int64_t Nz,
                                           double* d, int first = 0, const double* grid = nullptr,
                                           bool wide = false) {
#ifdef __CUDA_ARCH__
  const double z0 = grid ? grid[0] : zi[0], zl = grid ? grid[1] : zi[Nz - 1];
  if (!(z0 <= z && z <= zl)) return false;
  int64_t idx = grid ? (int64_t)div_by(z - z0, grid[2], grid[3]) : (int64_t)((z - z0) / (zi[1] - zi[0]));
#else
  (void)grid;
  double z0 = zi[0], zl = zi[Nz - 1];
  if (!(z0 <= z && z <= zl)) return false;
  double dz = zi[1] - zi[0];
  int64_t idx = (int64_t)((z - z0) / dz);
#endif
  if (idx < 0) idx = 0;
  if (idx > Nz - 2) idx = Nz - 2;
  double x = z - zi[idx];
  const double* C = coeff + idx * NDERIV * 6;
#ifdef __CUDA_ARCH__
  if (wide && first == 1 && (reinterpret_cast<uintptr_t>(coeff) & 15) == 0) {
    const double2* row = reinterpret_cast<const double2*>(C + 6);  // 24 pairs
    const bool odd = reinterpret_cast<uintptr_t>(row) & 16;        // the boundary is behind the first pair
    const double2* quad = row + (odd ? 1 : 0);
    double2 prev = odd ? row[0] : row[22];  // the pair that the eleven loads leave out beside the last
    const double2 head = prev, last = row[23];
    double2 c[3];
    int have = 0, i = 1;
#pragma unroll
    for (int k = 0; k < 12; k++) {
      double2 lo, hi;
      if (k < 11) {
        asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                     : "=d"(lo.x), "=d"(lo.y), "=d"(hi.x), "=d"(hi.y)
                     : "l"(quad + 2 * k));
      } else {
        lo = head;
        hi = last;
      }
      const double2 even_pair{odd ? prev.x : lo.x, odd ? prev.y : lo.y};
      const double2 odd_pair = k < 11 ? double2{odd ? lo.x : hi.x, odd ? lo.y : hi.y} : last;
      prev = hi;
#pragma unroll
      for (int w = 0; w < 2; w++) {
        c[have++] = w == 0 ? even_pair : odd_pair;
        if (have == 3) {
          d[i++] = ((((c[0].x * x + c[0].y) * x + c[1].x) * x + c[1].y) * x + c[2].x) * x + c[2].y;
          have = 0;
        }
      }
    }
    return true;
  }
  if ((reinterpret_cast<uintptr_t>(coeff) & 15) == 0) {
#pragma unroll
    for (int i = 0; i < NDERIV; i++) {
      if (i < first) continue;
      const double2* c = reinterpret_cast<const double2*>(C + i * 6);
      const double2 a = c[0], b = c[1], e = c[2];
      d[i] = ((((a.x * x + a.y) * x + b.x) * x + b.y) * x + e.x) * x + e.y;
    }
    return true;
  }
#pragma unroll
#endif
  for (int i = 0; i < NDERIV; i++) {
    if (i < first) continue;
    const double* c = C + i * 6;
    d[i] = ((((c[0] * x + c[1]) * x + c[2]) * x + c[3]) * x + c[4]) * x + c[5];
  }
  return true;
}

// The grid's constants for axial_eval.
__device__ __forceinline__ void axial_grid(const double* zi, int64_t Nz, double* grid) {
  grid[0] = zi[0];
  grid[1] = zi[Nz - 1];
  grid[2] = zi[1] - zi[0];
  grid[3] = 1.0 / grid[2];
}

// potential_radial_derivs, radial.c:340-343
__host__ __device__ inline double axial_potential(const double* d, double r2) {
  return d[0] - r2 / 4 * d[2] + r2 * r2 / 64. * d[4] - r2 * r2 * r2 / 2304. * d[6] +
         r2 * r2 * r2 * r2 / 147456. * d[8];
}

// field_radial_derivs, radial.c:376-383 (192 = 64 x 3, 9216 = 1024 x 9, 2304 =
// 256 x 9: on the device the quotients by 3 and 9 in three operations each)
__host__ __device__ inline void axial_field(const double* d, const double* p, double r2, double* f) {
#ifdef __CUDA_ARCH__
  const double r4 = r2 * r2;
  const double t3 = div_by(r4, 3.0, 1.0 / 3.0), t9 = div_by(r4 * r2, 9.0, 1.0 / 9.0);
  double fr = 0.5 * (d[2] - r2 / 8 * d[4] + t3 / 64 * d[6] - t9 / 1024 * d[8]);
  double fz = -d[1] + r2 / 4 * d[3] - r4 / 64 * d[5] + t9 / 256 * d[7];
#else
  double fr = 0.5 * (d[2] - r2 / 8 * d[4] + r2 * r2 / 192 * d[6] - r2 * r2 * r2 / 9216 * d[8]);
  double fz = -d[1] + r2 / 4 * d[3] - r2 * r2 / 64 * d[5] + r2 * r2 * r2 / 2304 * d[7];
#endif
  f[0] = p[0] * fr;
  f[1] = p[1] * fr;
  f[2] = fz;
}

}  // namespace tb
