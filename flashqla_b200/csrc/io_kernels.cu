// What the operator does to its inputs before the recurrence and to the gradients after it, each
// in one pass over memory:
//   * prepare_inputs: optional L2 normalisation of the rows of q and k, and conversion of float16
//     q, k, v to the bfloat16 the tensor-core kernels read;
//   * finish_grads: sum of dq, dk over the value heads of a group, the gradient of the L2
//     normalisation, and conversion of dq, dk, dv to the caller's type.
// HBM-bound: every element is read once and written once.  A row of D elements is held by D / 8
// lanes, 16 bytes each, so a warp moves 512 contiguous bytes per instruction (the general-purpose
// conversion kernels these replace moved the float16 q, k, v of an 8192-token batch, Hv = 8, in
// 59 us over four launches; one launch of prepare_inputs takes its place).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "fqla_internal.h"

namespace fqla {
namespace {

struct Bf16x8 {
  static __device__ __forceinline__ void unpack(const uint4& raw, float (&x)[8]) {
    const bf162* p = reinterpret_cast<const bf162*>(&raw);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = __bfloat1622float2(p[e]);
      x[2 * e] = f.x;
      x[2 * e + 1] = f.y;
    }
  }
  static __device__ __forceinline__ uint4 pack(const float (&x)[8]) {
    return make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]),
                      pack_bf16(x[6], x[7]));
  }
};
struct F16x8 {
  static __device__ __forceinline__ void unpack(const uint4& raw, float (&x)[8]) {
    const __half2* p = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = __half22float2(p[e]);
      x[2 * e] = f.x;
      x[2 * e + 1] = f.y;
    }
  }
  static __device__ __forceinline__ uint4 pack(const float (&x)[8]) {
    uint4 r;
    __half2* p = reinterpret_cast<__half2*>(&r);
#pragma unroll
    for (int e = 0; e < 4; ++e) p[e] = __floats2half2_rn(x[2 * e], x[2 * e + 1]);
    return r;
  }
};

// sum over the LANES consecutive lanes that share a row
template <int LANES>
__device__ __forceinline__ float row_sum(float x) {
#pragma unroll
  for (int d = LANES / 2; d > 0; d >>= 1) x += __shfl_xor_sync(0xffffffffu, x, d);
  return x;
}

struct PrepareParams {
  const void *q, *k, *v;
  void *q_out, *k_out, *v_out;   // v_out null: v is not converted
  float *q_rstd, *k_rstd;        // null: not wanted
  long long rows_qk, rows_v;     // rows of D elements in q (and k), in v
  int normalise;
  float eps;
};

// one thread per 16 bytes; the threads of q come first, then k, then v
template <typename IN, int D>
__global__ void __launch_bounds__(256) prepare_inputs_kernel(const PrepareParams p) {
  constexpr int LANES = D / 8;
  pdl_wait();
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  const long long n_qk = p.rows_qk * LANES, n_v = p.v_out ? p.rows_v * LANES : 0;
  // which tensor, and the 16-byte piece of it (rows never straddle a warp: LANES divides 32)
  const bool is_q = i < n_qk, is_k = !is_q && i < 2 * n_qk;
  const bool in = i < 2 * n_qk + n_v;
  const long long j = is_q ? i : is_k ? i - n_qk : i - 2 * n_qk;
  const void* src = is_q ? p.q : is_k ? p.k : p.v;
  void* dst = is_q ? p.q_out : is_k ? p.k_out : p.v_out;
  float x[8];
  IN::unpack(in ? reinterpret_cast<const uint4*>(src)[j] : make_uint4(0, 0, 0, 0), x);
  if (p.normalise) {  // whole warps take part in the shuffles
    float ss = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) ss += x[e] * x[e];
    const float r = rsqrtf(row_sum<LANES>(ss) + p.eps);
    if (is_q || is_k) {
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] *= r;
      float* rstd = is_q ? p.q_rstd : p.k_rstd;
      if (rstd && in && j % LANES == 0) rstd[j / LANES] = r;
    }
  }
  if (in) reinterpret_cast<uint4*>(dst)[j] = Bf16x8::pack(x);
}

struct FinishParams {
  const void *dq_v, *dk_v, *dv_in;  // bf16, per value head; dv_in null: dv is not converted
  const void *q, *k;                // rows of the normalisation: its outputs (bf16) or inputs (type of dq)
  const float *q_rstd, *k_rstd;     // null: no normalisation
  int normalised;                   // q, k are outputs
  void *dq, *dk, *dv;
  long long rows_qk, rows_v;
  int G;                            // value heads per q/k head
};

template <typename OUT, int D>
__global__ void __launch_bounds__(256) finish_grads_kernel(const FinishParams p) {
  constexpr int LANES = D / 8;
  pdl_wait();
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  const long long n_qk = p.rows_qk * LANES, n_v = p.dv_in ? p.rows_v * LANES : 0;
  const bool is_q = i < n_qk, is_k = !is_q && i < 2 * n_qk;
  const bool in = i < 2 * n_qk + n_v;
  const long long j = is_q ? i : is_k ? i - n_qk : i - 2 * n_qk;
  const int G = is_q || is_k ? p.G : 1;
  const long long row = j / LANES;
  const int lane = (int)(j % LANES);
  const uint4* src = reinterpret_cast<const uint4*>(is_q ? p.dq_v : is_k ? p.dk_v : p.dv_in);
  float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (in) {
#pragma unroll 2
    for (int h = 0; h < G; ++h) {
      float y[8];
      Bf16x8::unpack(src[(row * G + h) * LANES + lane], y);
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] += y[e];
    }
  }
  if (p.q_rstd) {
    // y = x_in * rstd;  d x_in = (dy - <dy, y> y) * rstd
    const bool qk = in && (is_q || is_k);
    float y[8], dot = 0.f;
    const uint4 raw = qk ? reinterpret_cast<const uint4*>(is_q ? p.q : p.k)[j] : make_uint4(0, 0, 0, 0);
    const float r = qk ? (is_q ? p.q_rstd : p.k_rstd)[row] : 1.f;
    if (p.normalised) {
      Bf16x8::unpack(raw, y);
    } else {
      OUT::unpack(raw, y);
#pragma unroll
      for (int e = 0; e < 8; ++e) y[e] *= r;
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) dot += x[e] * y[e];
    dot = row_sum<LANES>(dot);
    if (qk) {
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = (x[e] - dot * y[e]) * r;
    }
  }
  if (in) reinterpret_cast<uint4*>(is_q ? p.dq : is_k ? p.dk : p.dv)[j] = OUT::pack(x);
}

}  // namespace
}  // namespace fqla

using namespace fqla;

extern "C" int fqla_prepare_inputs(const void* q, const void* k, const void* v, void* q_out,
                                   void* k_out, void* v_out, float* q_rstd, float* k_rstd,
                                   long long rows_qk, long long rows_v, int D, int is_f16,
                                   int normalise, float eps, void* stream) {
  if (!q || !k || !q_out || !k_out || (v_out && !v) || rows_qk < 0 || rows_v < 0)
    return FQLA_ERR_INVALID_ARG;
  if (D != 64 && D != 128) return FQLA_ERR_UNSUPPORTED_DIM;
  const long long n = (2 * rows_qk + (v_out ? rows_v : 0)) * (D / 8);
  if (n == 0) return FQLA_OK;
  const PrepareParams p{q, k, v, q_out, k_out, v_out, q_rstd, k_rstd, rows_qk, rows_v, normalise, eps};
  const unsigned grid = (unsigned)((n + 255) / 256);
  cudaStream_t st = (cudaStream_t)stream;
  if (D == 128) {
    if (is_f16) return launch_pdl(prepare_inputs_kernel<F16x8, 128>, dim3(grid), dim3(256), 0, st, p);
    return launch_pdl(prepare_inputs_kernel<Bf16x8, 128>, dim3(grid), dim3(256), 0, st, p);
  }
  if (is_f16) return launch_pdl(prepare_inputs_kernel<F16x8, 64>, dim3(grid), dim3(256), 0, st, p);
  return launch_pdl(prepare_inputs_kernel<Bf16x8, 64>, dim3(grid), dim3(256), 0, st, p);
}

extern "C" int fqla_finish_grads(const void* dq_v, const void* dk_v, const void* dv_in,
                                 const void* q, const void* k, const float* q_rstd,
                                 const float* k_rstd, void* dq, void* dk, void* dv,
                                 long long rows_qk, int G, int D, int types, void* stream) {
  const int is_f16 = types & FQLA_GRADS_F16;
  if (!dq_v || !dk_v || !dq || !dk || (dv_in && !dv) || G <= 0 || rows_qk < 0)
    return FQLA_ERR_INVALID_ARG;
  if (q_rstd && (!k_rstd || !q || !k)) return FQLA_ERR_INVALID_ARG;
  if (D != 64 && D != 128) return FQLA_ERR_UNSUPPORTED_DIM;
  const long long rows_v = rows_qk * G, n = (2 * rows_qk + (dv_in ? rows_v : 0)) * (D / 8);
  if (n == 0) return FQLA_OK;
  const FinishParams p{dq_v, dk_v, dv_in, q, k, q_rstd, k_rstd, types & FQLA_ROWS_NORMALISED, dq, dk, dv,
                       rows_qk, rows_v, G};
  const unsigned grid = (unsigned)((n + 255) / 256);
  cudaStream_t st = (cudaStream_t)stream;
  if (D == 128) {
    if (is_f16) return launch_pdl(finish_grads_kernel<F16x8, 128>, dim3(grid), dim3(256), 0, st, p);
    return launch_pdl(finish_grads_kernel<Bf16x8, 128>, dim3(grid), dim3(256), 0, st, p);
  }
  if (is_f16) return launch_pdl(finish_grads_kernel<F16x8, 64>, dim3(grid), dim3(256), 0, st, p);
  return launch_pdl(finish_grads_kernel<Bf16x8, 64>, dim3(grid), dim3(256), 0, st, p);
}
