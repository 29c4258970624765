// tb_mlp_train.cu -- one training step of the surrogate network (loss and
// gradients of a batch) in one kernel and a reduction.
//
// The step was 36 launches: per layer and direction a GEMM with scalar
// staging loads, element-wise kernels with their operands in global memory,
// and weight gradients added with atomics (batch 8,192: 432 us of device
// time, 494 us a step).  Here a CTA takes 64 samples through the whole
// network and back: every weight in shared memory, activations (BF16) kept
// there for the weight gradients, pre-activations (FP32) in the registers of
// the threads that computed them -- the fragment layout of a layer's forward
// and backward products is the same.  128 CTAs at batch 8,192.  The products
// are warp-level mma.sync on ldmatrix fragments (the transposed operands of the
// backward pass come for free): at 64 rows a tile the step is latency-bound,
// 2.7 GFLOP in all, and the tensor-memory path would need a second, transposed
// copy of every operand in shared memory, which has no room for it.
//
// Every product accumulates over k in steps of 16 in ascending order, as
// k_gemm_bf16 does, and the element-wise forms are those of tb_mlp.cu, so
// activations and back-propagated gradients have the same bits; the weight
// gradients are summed per CTA, then over CTAs in a fixed order (no atomics).
#include "tb_common.cuh"
#include "tb_internal.cuh"
#include "tb_mlp.cuh"
#include "../../include/traceon_b200.h"

namespace tb {

constexpr int MT_ROWS = 64;      // samples of a tile
constexpr int MT_THREADS = 256;  // 8 warps: 4 groups of 16 rows x 2 halves of 64 columns
constexpr int MT_LD = MLP_H + 8;     // padded rows (bf16): ldmatrix without bank conflicts
constexpr int MT_LDX = MLP_IN + 8;
constexpr int MT_LDO = MLP_OUT + 8;

struct TrainSmem {
  __nv_bfloat16 wh[3][MLP_H][MT_LD];   // W2, W3, W4
  __nv_bfloat16 w1[MLP_H][MT_LDX];
  __nv_bfloat16 w5[MLP_OUT][MT_LD];
  __nv_bfloat16 x[MT_ROWS][MT_LDX];
  __nv_bfloat16 y[4][MT_ROWS][MT_LD];  // activations of the hidden layers
  __nv_bfloat16 g[MT_ROWS][MT_LD];     // gradient with respect to a layer's pre-activations
  __nv_bfloat16 g5[MT_ROWS][MT_LDO];
  float b[4][MLP_H], b5[MLP_OUT];
  float red[MT_THREADS / 32];
};
static_assert(sizeof(TrainSmem) <= 227 * 1024, "fits one CTA's shared memory");

__device__ __forceinline__ void ldm4(uint32_t (&r)[4], const __nv_bfloat16* p) {
  const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}
__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], const __nv_bfloat16* p) {
  const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}

// acc[2 t], acc[2 t + 1] (n8 tiles n0 + 16 t, + 8) += A (16 rows from a, row
// stride lda) . B over k: BT false: B(n, k) at b[n * ldb + k]; true: at
// b[k * ldb + n].  A(m, k) at a[m * lda + k], or with AT at a[k * lda + m].
template <int K, int TILES, bool AT, bool BT>
__device__ __forceinline__ void warp_gemm(float (&acc)[2 * TILES][4], const __nv_bfloat16* a, int lda,
                                          const __nv_bfloat16* b, int ldb) {
  const int lane = threadIdx.x & 31, mi = lane >> 3, l8 = lane & 7;
  // AT: matrices ordered (m, k) = (0,0) (8,0) (0,8) (8,8) either way
  const __nv_bfloat16* ap = AT ? a + ((mi >> 1) * 8 + l8) * lda + (mi & 1) * 8 : a + ((mi & 1) * 8 + l8) * lda + (mi >> 1) * 8;
  const __nv_bfloat16* bp = BT ? b + ((mi & 1) * 8 + l8) * ldb + (mi >> 1) * 8 : b + ((mi >> 1) * 8 + l8) * ldb + (mi & 1) * 8;
#pragma unroll
  for (int k = 0; k < K; k += 16) {
    uint32_t af[4];
    if (AT)
      ldm4t(af, ap + k * lda);
    else
      ldm4(af, ap + k);
#pragma unroll
    for (int t = 0; t < TILES; t++) {
      uint32_t bf[4];
      if (BT)
        ldm4t(bf, bp + k * ldb + 16 * t);
      else
        ldm4(bf, bp + 16 * t * ldb + k);
      mma_bf16_16816(acc[2 * t], af, bf);
      mma_bf16_16816(acc[2 * t + 1], af, bf + 2);
    }
  }
}

template <int N>
__device__ __forceinline__ void zero(float (&a)[N][4]) {
#pragma unroll
  for (int i = 0; i < N; i++) a[i][0] = a[i][1] = a[i][2] = a[i][3] = 0.f;
}

// Adds (or, for the CTA's first tile, stores) a warp's 16 x (8 N) block of a
// weight gradient: rows m0 .., columns n0 .. of a matrix with row stride ld.
template <int N>
__device__ __forceinline__ void store_grad(float* out, int ld, const float (&acc)[N][4], bool add) {
  const int lane = threadIdx.x & 31, gq = lane >> 2, q = lane & 3;
#pragma unroll
  for (int t = 0; t < N; t++)
#pragma unroll
    for (int hh = 0; hh < 2; hh++) {
      float2* p = reinterpret_cast<float2*>(out + (gq + 8 * hh) * ld + 8 * t + 2 * q);
      float2 v = make_float2(acc[t][2 * hh], acc[t][2 * hh + 1]);
      if (add) {
        const float2 o = *p;
        v.x += o.x;
        v.y += o.y;
      }
      *p = v;
    }
}

__device__ __forceinline__ void add_bias_grad(float* out, const __nv_bfloat16* g, int ld, int n, bool add) {
  if (threadIdx.x < n) {
    float s = 0.f;
#pragma unroll 8
    for (int r = 0; r < MT_ROWS; r++) s += __bfloat162float(g[r * ld + threadIdx.x]);
    out[threadIdx.x] = add ? out[threadIdx.x] + s : s;
  }
}

// partial: (gridDim.x, MLP_NPARAM + 4) gradient sums of each CTA, its loss at
// index MLP_NPARAM.
constexpr int64_t MT_SLOT = MLP_NPARAM + 4;

__global__ void __launch_bounds__(MT_THREADS, 1)
    k_mlp_step(const __nv_bfloat16* __restrict__ X, const float* __restrict__ T, const float* __restrict__ w, int64_t M,
               int n_out, const __nv_bfloat16* __restrict__ wb, const float* __restrict__ pf,
               float* __restrict__ partial) {
  extern __shared__ __align__(16) unsigned char mt_raw[];
  TrainSmem& s = *reinterpret_cast<TrainSmem*>(mt_raw);
  const int tid = threadIdx.x, warp = tid / 32, lane = tid & 31, gq = lane >> 2, q = lane & 3;
  const int r0 = 16 * (warp & 3), c0 = 64 * (warp >> 2);  // the warp's rows and columns of a hidden layer
  // weights, 16 bytes a thread
  const int64_t off[3] = {MLP_OFF_W2, MLP_OFF_W3, MLP_OFF_W4};
#pragma unroll
  for (int l = 0; l < 3; l++)
    for (int e = tid; e < MLP_H * MLP_H / 8; e += MT_THREADS)
      *reinterpret_cast<uint4*>(&s.wh[l][e / 16][(e % 16) * 8]) = reinterpret_cast<const uint4*>(wb + off[l])[e];
  for (int e = tid; e < MLP_H * MLP_IN / 8; e += MT_THREADS)
    *reinterpret_cast<uint4*>(&s.w1[e / 2][(e % 2) * 8]) = reinterpret_cast<const uint4*>(wb + MLP_OFF_W1)[e];
  for (int e = tid; e < MLP_OUT * MLP_H / 8; e += MT_THREADS)
    *reinterpret_cast<uint4*>(&s.w5[e / 16][(e % 16) * 8]) = reinterpret_cast<const uint4*>(wb + MLP_OFF_W5)[e];
  if (tid < MLP_H) {
    s.b[0][tid] = pf[MLP_OFF_B1 + tid];
    s.b[1][tid] = pf[MLP_OFF_B2 + tid];
    s.b[2][tid] = pf[MLP_OFF_B3 + tid];
    s.b[3][tid] = pf[MLP_OFF_B4 + tid];
  }
  if (tid < MLP_OUT) s.b5[tid] = pf[MLP_OFF_B5 + tid];
  float* out = partial + blockIdx.x * MT_SLOT;
  bool add = false;
  float loss = 0.f;
  for (int64_t m0 = blockIdx.x * (int64_t)MT_ROWS; m0 < M; m0 += (int64_t)gridDim.x * MT_ROWS) {
    __syncthreads();  // the previous tile is done with x, y and g
    for (int e = tid; e < MT_ROWS * MLP_IN; e += MT_THREADS) {
      const int r = e / MLP_IN, k = e % MLP_IN;
      s.x[r][k] = m0 + r < M ? X[(m0 + r) * MLP_IN + k] : __float2bfloat16(0.f);
    }
    __syncthreads();
    // forward: z[l] stays in registers for the backward pass
    float z[4][8][4];
#pragma unroll
    for (int l = 0; l < 4; l++) {
      zero(z[l]);
      if (l == 0)
        warp_gemm<MLP_IN, 4, false, false>(z[0], &s.x[r0][0], MT_LDX, &s.w1[c0][0], MT_LDX);
      else
        warp_gemm<MLP_H, 4, false, false>(z[l], &s.y[l > 0 ? l - 1 : 0][r0][0], MT_LD, &s.wh[l > 0 ? l - 1 : 0][c0][0], MT_LD);
#pragma unroll
      for (int t = 0; t < 8; t++) {
        const int col = c0 + 8 * t + 2 * q;
        const float b0 = s.b[l][col], b1 = s.b[l][col + 1];
        z[l][t][0] += b0;
        z[l][t][1] += b1;
        z[l][t][2] += b0;
        z[l][t][3] += b1;
        *reinterpret_cast<uint32_t*>(&s.y[l][r0 + gq][col]) = silu2_bf16(z[l][t][0], z[l][t][1]);
        *reinterpret_cast<uint32_t*>(&s.y[l][r0 + gq + 8][col]) = silu2_bf16(z[l][t][2], z[l][t][3]);
      }
      __syncthreads();
    }
    // outputs (16 columns a warp), loss, and the gradient of the mean square
    {
      float o[2][4];
      zero(o);
      const int oc = 16 * (warp >> 2);
      warp_gemm<MLP_H, 1, false, false>(o, &s.y[3][r0][0], MT_LD, &s.w5[oc][0], MT_LD);
#pragma unroll
      for (int t = 0; t < 2; t++)
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
          const int r = r0 + gq + 8 * hh, col = oc + 8 * t + 2 * q;
          const int64_t row = m0 + r;
          float gr[2] = {0.f, 0.f};
#pragma unroll
          for (int u = 0; u < 2; u++)
            if (row < M && col + u < n_out) {
              const float d = (o[t][2 * hh + u] + s.b5[col + u]) - T[row * n_out + col + u];
              const float wi = w ? w[row] : 1.f;
              gr[u] = 2.f * d * wi / float(M * n_out);
              loss += d * d * wi;
            }
          *reinterpret_cast<uint32_t*>(&s.g5[r][col]) = pack_bf16(gr[0], gr[1]);
        }
      __syncthreads();
    }
    // backward; dA of a layer has the fragment layout of its z
    float dz[8][4];
    zero(dz);
    warp_gemm<MLP_OUT, 4, false, true>(dz, &s.g5[r0][0], MT_LDO, &s.w5[0][c0], MT_LD);
    {
      float dw[4][4];  // dW5: 16 outputs x 32 inputs a warp
      zero(dw);
      const int mo = 16 * (warp & 1), no = 32 * (warp >> 1);
      warp_gemm<MT_ROWS, 2, true, true>(dw, &s.g5[0][mo], MT_LDO, &s.y[3][0][no], MT_LD);
      store_grad(out + MLP_OFF_W5 + mo * MLP_H + no, MLP_H, dw, add);
      add_bias_grad(out + MLP_OFF_B5, &s.g5[0][0], MT_LDO, MLP_OUT, add);
    }
#pragma unroll
    for (int l = 3; l >= 0; l--) {
#pragma unroll
      for (int t = 0; t < 8; t++) {
        const int col = c0 + 8 * t + 2 * q;
        *reinterpret_cast<uint32_t*>(&s.g[r0 + gq][col]) =
            pack_bf16(dz[t][0] * silu_grad(z[l][t][0]), dz[t][1] * silu_grad(z[l][t][1]));
        *reinterpret_cast<uint32_t*>(&s.g[r0 + gq + 8][col]) =
            pack_bf16(dz[t][2] * silu_grad(z[l][t][2]), dz[t][3] * silu_grad(z[l][t][3]));
      }
      __syncthreads();
      const int64_t ow = l == 0 ? MLP_OFF_W1 : l == 1 ? MLP_OFF_W2 : l == 2 ? MLP_OFF_W3 : MLP_OFF_W4;
      const int64_t ob = l == 0 ? MLP_OFF_B1 : l == 1 ? MLP_OFF_B2 : l == 2 ? MLP_OFF_B3 : MLP_OFF_B4;
      if (l > 0) {
        zero(dz);
        warp_gemm<MLP_H, 4, false, true>(dz, &s.g[r0][0], MT_LD, &s.wh[l > 0 ? l - 1 : 0][0][c0], MT_LD);
        // 16 outputs x 128 inputs a warp, in two halves
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
          float dw[8][4];
          zero(dw);
          warp_gemm<MT_ROWS, 4, true, true>(dw, &s.g[0][16 * warp], MT_LD, &s.y[l > 0 ? l - 1 : 0][0][64 * hh], MT_LD);
          store_grad(out + ow + 16 * warp * MLP_H + 64 * hh, MLP_H, dw, add);
        }
      } else {
        float dw[2][4];
        zero(dw);
        warp_gemm<MT_ROWS, 1, true, true>(dw, &s.g[0][16 * warp], MT_LD, &s.x[0][0], MT_LDX);
        store_grad(out + ow + 16 * warp * MLP_IN, MLP_IN, dw, add);
      }
      add_bias_grad(out + ob, &s.g[0][0], MT_LD, MLP_H, add);
      __syncthreads();  // g is overwritten by the next layer
    }
    add = true;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
  if (lane == 0) s.red[warp] = loss;
  __syncthreads();
  if (tid == 0) {
    float t = 0.f;
    for (int k = 0; k < MT_THREADS / 32; k++) t += s.red[k];
    out[MLP_NPARAM] = t;
  }
}

// grad = the sum of the CTAs' partial gradients, loss = the sum of theirs / (M n_out).
__global__ void __launch_bounds__(128) k_mlp_step_sum(const float* __restrict__ partial, int slots, float* __restrict__ grad,
                                                      float* __restrict__ loss, float count) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i > MLP_NPARAM) return;
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
  int k = 0;
  for (; k + 4 <= slots; k += 4) {
    s0 += partial[k * MT_SLOT + i];
    s1 += partial[(k + 1) * MT_SLOT + i];
    s2 += partial[(k + 2) * MT_SLOT + i];
    s3 += partial[(k + 3) * MT_SLOT + i];
  }
  for (; k < slots; k++) s0 += partial[k * MT_SLOT + i];
  const float t = (s0 + s1) + (s2 + s3);
  if (i < MLP_NPARAM)
    grad[i] = t;
  else
    *loss = t / count;
}

static int64_t step_slots(int64_t M) {
  const int64_t tiles = (M + MT_ROWS - 1) / MT_ROWS;
  return tiles < num_sms() ? tiles : num_sms();
}

}  // namespace tb

using namespace tb;

extern "C" int64_t tb_mlp_loss_grad_workspace(int64_t M) {
  return M <= 0 ? 0 : step_slots(M) * MT_SLOT * int64_t(sizeof(float));
}

extern "C" int tb_mlp_loss_grad(const void* X, const float* T, const float* w, int64_t M, int64_t n_out,
                                const void* weights_bf16, const float* params_f32, float* grad, float* loss, void* work,
                                int64_t work_bytes, tb_stream_t stream) {
  if (M <= 0 || n_out <= 0 || n_out > MLP_OUT || !X || !T || !weights_bf16 || !params_f32 || !grad || !loss || !work ||
      work_bytes < tb_mlp_loss_grad_workspace(M) || reinterpret_cast<uintptr_t>(weights_bf16) % 16 != 0 ||
      reinterpret_cast<uintptr_t>(work) % 16 != 0)
    return BAD_ARG;
  static bool attr[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return CUDA_ERR;
  if (dev < 0 || dev >= 64) return BAD_ARG;
  if (!attr[dev]) {
    if (cudaFuncSetAttribute(k_mlp_step, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(TrainSmem))) !=
        cudaSuccess)
      return CUDA_ERR;
    attr[dev] = true;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const int slots = int(step_slots(M));
  float* partial = static_cast<float*>(work);
  k_mlp_step<<<unsigned(slots), MT_THREADS, sizeof(TrainSmem), s>>>(static_cast<const __nv_bfloat16*>(X), T, w, M,
                                                                   int(n_out),
                                                                   static_cast<const __nv_bfloat16*>(weights_bf16),
                                                                   params_f32, partial);
  k_mlp_step_sum<<<unsigned((MLP_NPARAM + 1 + 127) / 128), 128, 0, s>>>(partial, slots, grad, loss,
                                                                       float(M * n_out));
  return launch_status();
}
