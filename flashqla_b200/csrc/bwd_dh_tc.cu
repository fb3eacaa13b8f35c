// Reverse chunk recurrence of the gated delta rule (gradient of the recurrent state) on Blackwell
// tensor cores, K = V = 128.  Same mathematics and outputs as bwd_dh.cu (reference:
// tests/ref_gdr.py:302-424; the reference's kernels compute it inside
// blackwell/fused_bwd.py:336-474): one CTA walks the chunks of one (sequence or segment, value
// head) from the last to the first.
//
// The state gradient is kept transposed, dS^T [v][k], fp32 in tensor memory (128 lanes = value
// index).  Per chunk, with Kc/Qc/dOc/Ac the chunk's tiles:
//     emit dh_c = dS                                   (bf16; also the operand copy in smem)
//     X1^T = dS^T Kc^T                  [v][tok]       on the chain
//     X2^T = dOc^T Pg                   [v][tok]       Pg = scale * G .* (Qc Kc^T), lower tri.
//     dv^T = rho .* X1^T + X2^T                        -> bf16 operand, emitted as du
//     w    = (Ac diag(beta gamma)) Kc   [tok][k]
//     dS^T <- gamma_last dS^T - dv^T w + dOc^T (scale gamma .* Qc)
// Roles: warp 0 issues the products that dS depends on (X1, the update), warp 3 the others (P, w, X2), warp 1
// runs the TMA pipeline (two stages of q, k, dO, A) and the per-row vectors, warp 2 scales A, warps 4-7 own
// the state (operand copy, decay, dh / dh0 output), warps 8-11 turn X1, X2 and w into operands (and write
// du), warps 12-15 build Pg and scale q (in place).  All waits are bounded mbarrier waits.
// (One thread issued everything before, 32 instructions of some 50 cycles a chunk, and two warps scaled both A
// and q and took longer over q than the chain over a chunk: 262144 tokens x 8 heads 674 -> 587 us, 32768 packed
// x 32 heads 384 -> 360, 4096 x 8 heads 22.6 -> 21.7; with A scaled by the state group 618, 362 and 21.9.  With
// waits that pause between two tries and row-major outputs made in rolled loops (69 -> 56 KB of code) 604 -> 584 and
// 361 -> 353; with issuing warps that leave their loop where a wait is given up, 353 -> 348 to 351.)
#include <cuda.h>

#include <climits>

#include "common.cuh"
#include "fqla_internal.h"
#include "tc05.cuh"

namespace fqla {

using namespace tc;

// set to 1 when a CTA of this file's kernel abandoned a bounded wait
__device__ int g_bwd_dh_status = 0;

struct BwdDhTcParams {
  const float* g;
  const void* beta;
  int beta_is_f32;
  const float* dht;  // [*, Hv, D, D] or null; the next four: see fqla_bwd_dh_args in include/fqla.h
  const float* seg_dht;
  const int *dht_row, *dh0_row;
  int v_first;
  bf16* dh;          // [chunks, Hv, D, D] or null
  bf16* du;          // [rows, Hv, D] or null
  float* dh0;        // [*, Hv, D, D] or null
  int N, Hq, Hv;
  float scale;
  SeqLayout lay;
  int tiled;  // dh and du are written as operand tiles (dh^T, du^T per chunk) by TMA
  const int* order;  // [N] or null: block index -> sequence (longest first shortens the tail)
  // [N, Hv] or null: lead-out.  A CTA with lead > 0 starts from a ZERO state gradient `lead`
  // chunks after the end of its segment (those rows are the head of what follows it in the same
  // sequence), walks them without output and enters its own last chunk with the gradient it
  // would have been handed, up to what the gates let through of anything later.  dht is ignored
  // for such a CTA.  lead < 0: -lead chunks, to the end of the sequence that the segment is cut
  // from, and from the gradient of that one's own final state.
  const int* lead;
  // [N, Hv] or null: a CTA whose entry differs from run_value returns at once
  const int* run_mask;
  int run_value;
  // [N, Hv] or null (dh0 only): only the first warm[n,hv] chunks are walked, from a zero gradient
  // (< 0: nothing is done)
  const int* warm;
  int* zero_word;  // or null: set to zero (a counter of the kernel behind this one)
};

namespace bdtc {
constexpr int D = 128;
constexpr int TILE = 16384, TILE_A = 8192;
constexpr int STAGE_BYTES = 3 * TILE + TILE_A;  // q, k, dO, A
constexpr int OFF_STAGE = 0;
constexpr int OFF_ST = 2 * STAGE_BYTES;   // dS^T copy, 2 blocks of [128 x 128B]
constexpr int OFF_DVT = OFF_ST + 32768;   // dv^T   [128 x 128B]
constexpr int OFF_W = OFF_DVT + 16384;    // w      2 blocks of [64 x 128B]
constexpr int OFF_P = OFF_W + 16384;      // Pg     [64 x 128B]
constexpr int OFF_APP = OFF_P + 8192;     // A diag(beta gamma)
constexpr int OFF_VEC = OFF_APP + 8192;
constexpr int VEC_SLOT_FLOATS = 5 * CHUNK;
constexpr int OFF_BAR = OFF_VEC + 4 * VEC_SLOT_FLOATS * 4;
constexpr int N_BARS = 24;
constexpr int OFF_MISC = OFF_BAR + N_BARS * 8;
constexpr int SMEM_BYTES = OFF_MISC + 16 + 1024;
constexpr uint32_t TM_S = 0, TM_X1 = 128, TM_X2 = 192, TM_P = 256, TM_W = 384;
enum { FULL0 = 0, FULL1, EMPTY0, EMPTY1, S_COPY, S_DEC, X1_DONE, X2_DONE, S_DONE, P_DONE, W_DONE,
       DV_READY, W_READY, P_READY, AP_READY, QS_READY, PRIV,
       // the A tile and the per-row vectors of a chunk travel one chunk ahead of q, k, dO
       FULLA0, FULLA1, EMPTYA0, EMPTYA1, PRIVA,
       // all products have come to their end
       SETTLED };
enum { V_G = 0, V_BG = 1, V_RHO = 2, V_SGAM = 3, V_GL = 4 };
}  // namespace bdtc

__device__ __forceinline__ uint32_t scale2(uint32_t packed, float lo, float hi) {
  float2 f = __bfloat1622float2(*reinterpret_cast<const bf162*>(&packed));
  return pack_bf16(f.x * lo, f.y * hi);
}

__global__ void __launch_bounds__(512, 1)
bwd_dh_tc_kernel(const BwdDhTcParams p, const __grid_constant__ CUtensorMap map_q,
                 const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_do,
                 const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_dh,
                 const __grid_constant__ CUtensorMap map_du) {
  using namespace bdtc;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_MISC);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + OFF_MISC + 4);
  float* vec = reinterpret_cast<float*>(smem + OFF_VEC);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int hv = blockIdx.x % p.Hv;
  auto sequence = [&] { return p.order ? p.order[blockIdx.x / p.Hv] : (int)(blockIdx.x / p.Hv); };
  const int hq = hv / (p.Hv / p.Hq);
  if (p.run_mask) {
    pdl_wait();
    if (p.run_mask[sequence() * p.Hv + hv] != p.run_value) return;  // uniform per CTA
  }
  int warm = INT_MAX;
  if (p.warm) {
    pdl_wait();
    warm = p.warm[sequence() * p.Hv + hv];
    if (warm < 0) return;  // uniform per CTA
  }

  if (tid == 0) {
    mbar_init(&bars[FULL0], 1);
    mbar_init(&bars[FULL1], 1);
    mbar_init(&bars[EMPTY0], 2);  // MMA commits of the two issuing threads
    mbar_init(&bars[EMPTY1], 2);
    mbar_init(&bars[S_COPY], 128);
    mbar_init(&bars[S_DEC], 128);
    mbar_init(&bars[X1_DONE], 1);
    mbar_init(&bars[X2_DONE], 1);
    mbar_init(&bars[S_DONE], 1);
    mbar_init(&bars[P_DONE], 1);
    mbar_init(&bars[W_DONE], 1);
    mbar_init(&bars[DV_READY], 128);
    mbar_init(&bars[W_READY], 128);
    mbar_init(&bars[P_READY], 128);
    mbar_init(&bars[AP_READY], 1);
    mbar_init(&bars[QS_READY], 128);
    mbar_init(&bars[PRIV], 1);
    mbar_init(&bars[FULLA0], 1);
    mbar_init(&bars[FULLA1], 1);
    mbar_init(&bars[EMPTYA0], 1);  // the scaling warp, the only reader of the raw A tile
    mbar_init(&bars[EMPTYA1], 1);
    mbar_init(&bars[PRIVA], 1);
    mbar_init(&bars[SETTLED], 2);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_do);
    tma_prefetch_desc(&map_a);
  }
  // Pg is lower triangular: zeroed once, only the column groups that can be non-zero are rewritten
  for (int i = tid; i < 8192 / 16; i += 512)
    *reinterpret_cast<uint4*>(smem + OFF_P + i * 16) = make_uint4(0, 0, 0, 0);
  fence_proxy_async();
  if (warp == 0) tmem_alloc(tmem_slot, 512);
  // everything above overlaps the tail of the kernel before: no global memory up to here
  pdl_wait();
  if (p.zero_word && blockIdx.x == 0 && tid == 0) *p.zero_word = 0;
  const int n = sequence();
  const SeqSpan sp = p.lay.span(n);
  // iteration `it` handles chunk n_it - 1 - it of the segment; chunks >= sp.n_chunks are the
  // lead-out chunks (whole chunks, except possibly the very last one of the sequence)
  // (lead < 0: the last -lead chunks are left out)
  const int lead_out = !p.warm && p.lead && sp.n_chunks > 0 ? p.lead[n * p.Hv + hv] : 0;
  const int lead = p.warm ? min(warm, sp.n_chunks) - sp.n_chunks : abs(lead_out);
  const int n_it = sp.n_chunks + lead;
  int len_ext = sp.len;
#pragma unroll 1
  for (int i = n + 1, left = lead; left > 0 && i < p.N; ++i) {
    const SeqSpan next = p.lay.span(i);
    len_ext += min(left * CHUNK, next.len);
    left -= next.n_chunks;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
  int tries = WAIT_TRIES;  // see mbar_wait; filled up for each pass of a role's loop
  auto WAIT = [&](int idx, uint32_t parity) { mbar_wait(&bars[idx], parity, tries); };
  // (of the issuing warps: see mbar_wait_uniform; 262144 tokens x 8 heads 584 us, 590 with the plain ones)
  auto WAITU = [&](int idx, uint32_t parity) { return mbar_wait_uniform(&bars[idx], parity, tries); };
  auto fill = [&] { tries = tries > 0 ? WAIT_TRIES : tries; };
  // A thread that has given a wait up issues, signals and stores nothing more: see fwd_tc.cu.
  auto ARRIVE = [&](int idx) { mbar_arrive_if(&bars[idx], tries); };
  auto issuing = [&] { return elect_one() && tries > 0; };  // of the producer
  // At the end of a role that issues: a wait with a limit of its own.
  auto settle = [&](int idx, uint32_t parity) {
    int again = WAIT_TRIES;
    mbar_wait(&bars[idx], parity, again);
    if (again <= 0) tries = 0;
  };

  // End gradient -> tensor memory, dS^T[v][k]; zero without one and for a lead-out.  The three
  // read-out groups share the columns 2 : 1 : 1: one memory latency (see fwd_tc.cu).
  if (warp >= 4) {
    int dht_row = p.dht_row ? p.dht_row[n] : n;
    if (lead_out < 0) dht_row = ~dht_row;
    const bool edge = dht_row >= 0;
    const float* src = (p.warm ? lead != 0 : lead_out > 0) ? nullptr : edge ? p.dht : p.seg_dht;
    if (src) src += ((long long)(edge ? dht_row : n) * p.Hv + hv) * D * D;
    const int v = (warp & 3) * 32 + lane;
    auto load32 = [&](int k0, float (&x)[32]) {
      if (!src) {
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = 0.f;
      } else if (edge && p.v_first) {
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 t = *reinterpret_cast<const float4*>(src + (long long)v * D + k0 + j);
          x[j] = t.x;
          x[j + 1] = t.y;
          x[j + 2] = t.z;
          x[j + 3] = t.w;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = src[(long long)(k0 + j) * D + v];
      }
    };
    float x[32];
    if (warp < 8) {
      float y[32];
      load32(0, x);
      load32(32, y);
      tmem_st32(tmem + lane_sel + TM_S, x);
      tmem_st32(tmem + lane_sel + TM_S + 32, y);
    } else {
      load32(warp < 12 ? 64 : 96, x);
      tmem_st32(tmem + lane_sel + TM_S + (warp < 12 ? 64 : 96), x);
    }
    tmem_st_wait();
    tc_fence_before();
    if (warp < 8) {
      asm volatile("bar.sync 2, 384;" ::: "memory");  // the state group waits for the other two
      tc_fence_after();
    } else {
      asm volatile("bar.arrive 2, 384;" ::: "memory");
    }
  }

  switch (warp >> 2) {  // (and not a chain of ifs: see fwd_tc.cu)
  case 1: {
    // =============================== state group ===============================
    const int v = tid - 128;
    for (int it = 0; it < n_it; ++it, fill()) {
      const int s = it & 1, c = n_it - 1 - it;
      if (it > 0) WAIT(S_DONE, (it - 1) & 1);
      tc_fence_after();
      bf16* hdst = (p.dh && it >= lead)
                       ? p.dh + ((sp.chunk_base + c) * p.Hv + hv) * (long long)D * D : nullptr;
#pragma unroll 1
      for (int kb = 0; kb < 2; ++kb) {
        float x[32], y[32];
        tmem_ld32(tmem + lane_sel + TM_S + kb * 64, x);
        tmem_ld32(tmem + lane_sel + TM_S + kb * 64 + 32, y);
        tmem_ld_wait();
        unsigned char* row = smem + OFF_ST + kb * 16384 + v * 128;
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          *reinterpret_cast<uint4*>(row + ((cc ^ (v & 7)) << 4)) =
              make_uint4(pack_bf16(x[8 * cc + 0], x[8 * cc + 1]), pack_bf16(x[8 * cc + 2], x[8 * cc + 3]),
                         pack_bf16(x[8 * cc + 4], x[8 * cc + 5]), pack_bf16(x[8 * cc + 6], x[8 * cc + 7]));
          *reinterpret_cast<uint4*>(row + (((cc + 4) ^ (v & 7)) << 4)) =
              make_uint4(pack_bf16(y[8 * cc + 0], y[8 * cc + 1]), pack_bf16(y[8 * cc + 2], y[8 * cc + 3]),
                         pack_bf16(y[8 * cc + 4], y[8 * cc + 5]), pack_bf16(y[8 * cc + 6], y[8 * cc + 7]));
        }
      }
      fence_proxy_async();
      tc_fence_before();
      ARRIVE(S_COPY);
      if (hdst && !p.tiled) {  // row-major [k][v]: column v, from this thread's own row of the copy
#pragma unroll 1
        for (int k = 0; k < (tries > 0 ? D : 0); ++k)
          hdst[(long long)k * D + v] =
              *reinterpret_cast<const bf16*>(smem + OFF_ST + (k >> 6) * 16384 + sw128_offset(v, k & 63));
      }
      // off the chain: decay in place
      WAIT(FULL0 + s, (it >> 1) & 1);
      const float gl = vec[(it & 3) * VEC_SLOT_FLOATS + V_GL * CHUNK];
#pragma unroll 1
      for (int kb = 0; kb < 2; ++kb) {
        float x[32], y[32];
        tmem_ld32(tmem + lane_sel + TM_S + kb * 64, x);
        tmem_ld32(tmem + lane_sel + TM_S + kb * 64 + 32, y);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          x[j] *= gl;
          y[j] *= gl;
        }
        tmem_st32(tmem + lane_sel + TM_S + kb * 64, x);
        tmem_st32(tmem + lane_sel + TM_S + kb * 64 + 32, y);
      }
      tmem_st_wait();
      tc_fence_before();
      ARRIVE(S_DEC);
    }
    if (n_it > 0) WAIT(S_DONE, (n_it - 1) & 1);
    const int dh0_row = p.dh0_row ? p.dh0_row[n] : n;
    if (__all_sync(0xffffffffu, tries > 0) && p.dh0 && dh0_row >= 0) {
      float* dst = p.dh0 + ((long long)dh0_row * p.Hv + hv) * D * D;
      tc_fence_after();
#pragma unroll 1
      for (int k0 = 0; k0 < D; k0 += 32) {
        float x[32];
        tmem_ld32(tmem + lane_sel + TM_S + k0, x);
        tmem_ld_wait();
        if (p.v_first) {
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            *reinterpret_cast<float4*>(dst + (long long)v * D + k0 + j) =
                make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) dst[(long long)(k0 + j) * D + v] = x[j];
        }
      }
    }
  } break;
  case 2: {
    // =============================== dv / w group ===============================
    const int v = tid - 256;
    const int wq = warp & 3;
    const int tok_w = 16 * wq + lane;  // lanes 0-15 of each quarter hold a row of w
    auto convert_w = [&](int it) {
      // ... and the state update that reads the tile of the chunk before is complete
      WAIT(W_DONE, it & 1);
      if (it > 0) WAIT(S_DONE, (it - 1) & 1);
      tc_fence_after();
#pragma unroll 1
      for (int c0 = 0; c0 < D; c0 += 32) {
        float x[32];
        tmem_ld32(tmem + lane_sel + TM_W + c0, x);
        tmem_ld_wait();
        if (lane < 16) {
          unsigned char* row = smem + OFF_W + (c0 >> 6) * 8192 + tok_w * 128;
#pragma unroll
          for (int cc = 0; cc < 4; ++cc)
            *reinterpret_cast<uint4*>(row + (((((c0 & 63) >> 3) + cc) ^ (tok_w & 7)) << 4)) =
                make_uint4(pack_bf16(x[8 * cc + 0], x[8 * cc + 1]), pack_bf16(x[8 * cc + 2], x[8 * cc + 3]),
                           pack_bf16(x[8 * cc + 4], x[8 * cc + 5]), pack_bf16(x[8 * cc + 6], x[8 * cc + 7]));
        }
      }
      fence_proxy_async();
      tc_fence_before();
      ARRIVE(W_READY);
    };
#pragma unroll 1
    for (int it = -1; it < n_it; ++it, fill()) {  // it = -1: only w of the first iteration
     if (it >= 0) {
      const int c = n_it - 1 - it;
      const long long row0 = sp.bos + (long long)c * CHUNK;
      const int valid = min(CHUNK, len_ext - c * CHUNK);
      WAIT(FULL0 + (it & 1), (it >> 1) & 1);
      WAIT(X2_DONE, it & 1);
      WAIT(X1_DONE, it & 1);
      tc_fence_after();
      const float* rho = vec + (it & 3) * VEC_SLOT_FLOATS + V_RHO * CHUNK;
      unsigned char* row = smem + OFF_DVT + v * 128;
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {  // 32 tokens per round
        float x[32], y[32];
        tmem_ld32(tmem + lane_sel + TM_X1 + 32 * h, x);
        tmem_ld32(tmem + lane_sel + TM_X2 + 32 * h, y);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 r = *reinterpret_cast<const float4*>(rho + 32 * h + j);
          x[j] = r.x * x[j] + y[j];
          x[j + 1] = r.y * x[j + 1] + y[j + 1];
          x[j + 2] = r.z * x[j + 2] + y[j + 2];
          x[j + 3] = r.w * x[j + 3] + y[j + 3];
        }
#pragma unroll
        for (int cc = 0; cc < 4; ++cc)
          *reinterpret_cast<uint4*>(row + (((4 * h + cc) ^ (v & 7)) << 4)) =
              make_uint4(pack_bf16(x[8 * cc + 0], x[8 * cc + 1]), pack_bf16(x[8 * cc + 2], x[8 * cc + 3]),
                         pack_bf16(x[8 * cc + 4], x[8 * cc + 5]), pack_bf16(x[8 * cc + 6], x[8 * cc + 7]));
      }
      // operand complete, accumulators read: hand over before the global stores
      fence_proxy_async();
      tc_fence_before();
      ARRIVE(DV_READY);
      if (p.du && !p.tiled && it >= lead) {  // row-major: column v, from this thread's own row
        bf16* dst = p.du + (row0 * p.Hv + hv) * D + v;
#pragma unroll 1
        for (int j = 0; j < (tries > 0 ? valid : 0); ++j)
          dst[(long long)j * p.Hv * D] = *reinterpret_cast<const bf16*>(smem + OFF_DVT + sw128_offset(v, j));
      }
     }
      if (it + 1 < n_it) convert_w(it + 1);
    }
  } break;
  case 3: {
    // =============================== Pg and q group ===============================
    // Pg, then q' = scale gamma .* q (rows) over q, once P = Q K^T has read it: ready long before the state
    // update wants it.  Two threads per row, in rotated order.
    const int qr = (tid - 384) >> 1, qh = tid & 1;
    const int wq = warp & 3;
    const int row_a = 16 * wq + (lane >> 2), row_b = row_a + 8, cp = 2 * (lane & 3);
    const uint32_t lanes_p = (uint32_t)(wq * 32) << 16;
    const float log2_scale = log2f(p.scale);
    for (int it = 0; it < n_it; ++it, fill()) {
      const float* vs = vec + (it & 3) * VEC_SLOT_FLOATS;
      WAIT(FULL0 + (it & 1), (it >> 1) & 1);
      WAIT(P_DONE, it & 1);
      if (it > 0) WAIT(X2_DONE, (it - 1) & 1);  // the previous Pg tile has been consumed
      tc_fence_after();
      const float ga2 = vs[V_G * CHUNK + row_a] * 1.4426950408889634f + log2_scale;
      const float gb2 = vs[V_G * CHUNK + row_b] * 1.4426950408889634f + log2_scale;
      float x[32];
      tmem_ld_16x64(tmem + lanes_p + TM_P, x);
      tmem_ld_wait();
      unsigned char* pa = smem + OFF_P + row_a * 128 + cp * 2;
      unsigned char* pb = smem + OFF_P + row_b * 128 + cp * 2;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (i > 2 * wq + 1) continue;
        const float2 gc = *reinterpret_cast<const float2*>(vs + V_G * CHUNK + 8 * i + cp);
        const int col = 8 * i + cp;
        const float e0 = -1.4426950408889634f * gc.x, e1 = -1.4426950408889634f * gc.y;
        const float a0 = col <= row_a ? x[4 * i] * exp2f(e0 + ga2) : 0.f;
        const float a1 = col + 1 <= row_a ? x[4 * i + 1] * exp2f(e1 + ga2) : 0.f;
        const float b0 = col <= row_b ? x[4 * i + 2] * exp2f(e0 + gb2) : 0.f;
        const float b1 = col + 1 <= row_b ? x[4 * i + 3] * exp2f(e1 + gb2) : 0.f;
        *reinterpret_cast<uint32_t*>(pa + ((i ^ (row_a & 7)) << 4)) = pack_bf16(a0, a1);
        *reinterpret_cast<uint32_t*>(pb + ((i ^ (row_b & 7)) << 4)) = pack_bf16(b0, b1);
      }
      fence_proxy_async();
      tc_fence_before();
      ARRIVE(P_READY);
      // (not before the update of the chunk before has been issued: its thread waits for that chunk's q)
      if (it > 0) WAIT(S_DONE, (it - 1) & 1);
      const float sg = vs[V_SGAM * CHUNK + qr];
      unsigned char* q = smem + OFF_STAGE + (it & 1) * STAGE_BYTES + qh * 8192 + qr * 128;
#pragma unroll 4
      for (int q8 = 0; q8 < 8; ++q8) {
        uint4* x8 = reinterpret_cast<uint4*>(q + ((q8 + qr) & 7) * 16);
        const uint4 a = *x8;
        *x8 = make_uint4(scale2(a.x, sg, sg), scale2(a.y, sg, sg), scale2(a.z, sg, sg), scale2(a.w, sg, sg));
      }
      fence_proxy_async();
      ARRIVE(QS_READY);
    }
  } break;
  default: if (warp == 0 || warp == 3) {
    // =============================== MMA issuers ===============================
    // (the warps stay converged; see elect_one in tc05.cuh)  Warp 0 issues what the state gradient depends
    // on: X1 and the two products of the update; warp 3 the rest (P, w, X2 of the next iteration).
    constexpr uint32_t ID_P = idesc_bf16(64, 64, 0, 0);
    constexpr uint32_t ID_X1 = idesc_bf16(128, 64, 0, 0);
    constexpr uint32_t ID_X2 = idesc_bf16(128, 64, 1, 1);
    constexpr uint32_t ID_W = idesc_bf16(64, 128, 0, 1);
    constexpr uint32_t ID_UPD_W = idesc_bf16(128, 128, 0, 1) | (1u << 13);  // A negated
    constexpr uint32_t ID_UPD_Q = idesc_bf16(128, 128, 1, 1);
    const uint32_t q0_lo = desc_lo_kmajor(smem + OFF_STAGE), k0_lo = desc_lo_kmajor(smem + OFF_STAGE + TILE);
    const uint32_t domn0_lo = desc_lo_mnmajor(smem + OFF_STAGE + 2 * TILE, 8192);
    constexpr uint32_t STAGE_LO = STAGE_BYTES >> 4;
    if (warp == 0) {
      const uint32_t st_lo = desc_lo_kmajor(smem + OFF_ST), dvt_lo = desc_lo_kmajor(smem + OFF_DVT);
      const uint32_t wmn_lo = desc_lo_mnmajor(smem + OFF_W, 8192), qmn0_lo = desc_lo_mnmajor(smem + OFF_STAGE, 8192);
#pragma unroll 1
      for (int it = 0; it < n_it; ++it, fill()) {
        const int s = it & 1;
        const uint32_t so = s ? STAGE_LO : 0u;
        const int y_tile = (int)(((sp.chunk_base + (n_it - 1 - it)) * p.Hv + hv) * D);
        if (!(WAITU(FULL0 + s, (it >> 1) & 1) && WAITU(S_COPY, it & 1))) break;
        tc_fence_after();
        if (elect_one()) {
          // X1^T = dS^T K^T   (on the chain)
          umma_group<8, 2, 1024, 2, 512, false>(tmem + TM_X1, st_lo, k0_lo + so, ID_X1);
          tma_store_wait_read();  // du^T of the chunk before has left its tile
          umma_commit(&bars[X1_DONE]);
          if (p.tiled && p.dh && it >= lead) {  // the operand copy of dS^T is dh of this chunk
            tma_store_2d(&map_dh, 0, y_tile, smem + OFF_ST);
            tma_store_2d(&map_dh, 64, y_tile, smem + OFF_ST + 16384);
            tma_store_commit();
          }
        }
        // dS^T <- dS^T + dO^T (scale gamma q) - dv^T w; the first product while dv is on its way
        if (!(WAITU(QS_READY, it & 1) && WAITU(S_DEC, it & 1))) break;
        tc_fence_after();
        if (elect_one())
          umma_group<4, 128, 0, 128, 0, true>(tmem + TM_S, domn0_lo + so, qmn0_lo + so, ID_UPD_Q);
        if (!(WAITU(W_READY, it & 1) && WAITU(DV_READY, it & 1))) break;
        tc_fence_after();
        if (elect_one()) {
          umma_group<4, 2, 0, 128, 0, true>(tmem + TM_S, dvt_lo, wmn_lo, ID_UPD_W);
          tma_store_wait_read();  // the dS^T tile may be rewritten after this
          umma_commit(&bars[S_DONE]);
          if (p.tiled && p.du && it >= lead) {
            tma_store_2d(&map_du, 0, y_tile, smem + OFF_DVT);
            tma_store_commit();
          }
          umma_commit(&bars[EMPTY0 + s]);
        }
      }
      if (elect_one()) tma_store_wait_all();
    } else {
      const uint32_t kmn0_lo = desc_lo_mnmajor(smem + OFF_STAGE + TILE, 8192);
      const uint32_t app_lo = desc_lo_kmajor(smem + OFF_APP), pmn_lo = desc_lo_mnmajor(smem + OFF_P, 8192);
#pragma unroll 1
      for (int it = 0; it < n_it; ++it, fill()) {
        const int s = it & 1;
        const uint32_t so = s ? STAGE_LO : 0u;
        // (the Pg group has read P of the chunk before: P_READY was waited for)
        if (!WAITU(FULL0 + s, (it >> 1) & 1)) break;
        tc_fence_after();
        if (elect_one()) {
          umma_group<8, 2, 512, 2, 512, false>(tmem + TM_P, q0_lo + so, k0_lo + so, ID_P);
          umma_commit(&bars[P_DONE]);
        }
        // w, whose accumulator the dv / w group has read for the chunk before
        if (!(WAITU(AP_READY, it & 1) && (it == 0 || WAITU(W_READY, (it - 1) & 1)))) break;
        tc_fence_after();
        if (elect_one()) {
          umma_group<4, 2, 0, 128, 0, false>(tmem + TM_W, app_lo, kmn0_lo + so, ID_W);
          umma_commit(&bars[W_DONE]);
        }
        // X2^T = dO^T Pg, likewise
        if (!(WAITU(P_READY, it & 1) && (it == 0 || WAITU(DV_READY, (it - 1) & 1)))) break;
        tc_fence_after();
        if (elect_one()) {
          umma_group<4, 128, 0, 128, 0, false>(tmem + TM_X2, domn0_lo + so, pmn_lo, ID_X2);
          umma_commit(&bars[X2_DONE]);
          umma_commit(&bars[EMPTY0 + s]);
        }
      }
    }
    // no product is under way when the block goes, whoever gave up what
    if (elect_one()) umma_commit(&bars[SETTLED]);
    if (warp == 0) settle(SETTLED, 0);
  } else if (warp == 1) {
    // =============================== producer ===============================
    float g_r[2] = {0.f, 0.f}, b_r[2] = {0.f, 0.f}, gl_r = 0.f;
    auto fetch = [&](int it) {
      const int c = n_it - 1 - it;
      const long long row0 = sp.bos + (long long)c * CHUNK;
      const int valid = min(CHUNK, len_ext - c * CHUNK);
      gl_r = p.g[(row0 + valid - 1) * p.Hv + hv];
#pragma unroll
      for (int z = 0; z < 2; ++z) {
        int r = 2 * lane + z, rc = min(r, valid - 1);
        g_r[z] = p.g[(row0 + rc) * p.Hv + hv];
        b_r[z] = r < valid ? load_beta(p.beta, p.beta_is_f32, (row0 + r) * p.Hv + hv) : 0.f;
      }
    };
    // zero the rows past the sequence end in n 8 KB blocks of 64 rows, then hand the tile on
    auto zero_rows = [&](unsigned char* base, int n, int valid, uint64_t* full) {
#pragma unroll 1
      for (int i = lane; i < n * 512; i += 32)
        if (((i >> 3) & 63) >= valid) *reinterpret_cast<uint4*>(base + i * 16) = make_uint4(0, 0, 0, 0);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0 && tries > 0) mbar_arrive(full);
    };
    // As in fwd_tc.cu: q, k, dO of iteration it; vectors and A tile of iteration it + 1; the gates of
    // iteration it + 2 into registers.  Slot (it + 1) % 4 of the vectors was last read for iteration
    // it - 3, which the wait on the stage of iteration it - 2 has seen finished.
    // (A whole first chunk's q, k, dO go out at once, ahead of its gates, as in fwd_tc.cu.)
    int loads = 0, a_loads = 0;  // q, k, dO and A tiles that have been asked for
    const bool early = n_it > 0 && len_ext >= n_it * CHUNK;
    auto load = [&](int it) {
      const int s = it & 1, c = n_it - 1 - it;
      const int y = (int)(sp.bos + (long long)c * CHUNK);
      const int valid = min(CHUNK, len_ext - c * CHUNK);
      const bool partial = valid < CHUNK;
      if (it >= 2) {
        WAIT(EMPTY0 + s, ((it >> 1) - 1) & 1);
      }
      unsigned char* st = smem + OFF_STAGE + s * STAGE_BYTES;
      uint64_t* bar = &bars[partial ? PRIV : FULL0 + s];
      if (issuing()) {
        mbar_expect_tx(bar, STAGE_BYTES - TILE_A);
        if (it > 0 || !early) mbar_arrive(bar);
        tma_load_2d(st + TILE, &map_k, hq * D, y, bar);
        tma_load_2d(st + TILE + 8192, &map_k, hq * D + 64, y, bar);
        tma_load_2d(st, &map_q, hq * D, y, bar);
        tma_load_2d(st + 8192, &map_q, hq * D + 64, y, bar);
        tma_load_2d(st + 2 * TILE, &map_do, hv * D, y, bar);
        tma_load_2d(st + 2 * TILE + 8192, &map_do, hv * D + 64, y, bar);
      }
      loads = tries > 0 ? it + 1 : loads;
      if (partial) {
        WAIT(PRIV, 0);
        zero_rows(st, 6, valid, &bars[FULL0 + s]);
      }
    };
#pragma unroll 1
    for (int it = -2; it < n_it; ++it, fill()) {
      if (it > 0 || it == (early ? -2 : 0)) load(max(it, 0));
      else if (it == 0 && lane == 0) ARRIVE(FULL0);
      const int j = it + 1;
      if (j >= 0 && j < n_it) {
        const int sj = j & 1, c = n_it - 1 - j;
        const int valid = min(CHUNK, len_ext - c * CHUNK);
        const bool partial = valid < CHUNK;
        // the stage's A buffer is free once the scaling warps have read it
        if (j >= 2) {
          WAIT(EMPTYA0 + sj, ((j >> 1) - 1) & 1);
        }
        float* vs = vec + (j & 3) * VEC_SLOT_FLOATS;
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          int r = 2 * lane + z;
          float gam = fast_exp(g_r[z]);
          vs[V_G * CHUNK + r] = g_r[z];
          vs[V_BG * CHUNK + r] = b_r[z] * gam;
          vs[V_RHO * CHUNK + r] = fast_exp(gl_r - g_r[z]);
          vs[V_SGAM * CHUNK + r] = p.scale * gam;
        }
        if (lane == 0) vs[V_GL * CHUNK] = fast_exp(gl_r);
        __syncwarp();
        unsigned char* dst = smem + OFF_STAGE + sj * STAGE_BYTES + 3 * TILE;
        uint64_t* bar = &bars[partial ? PRIVA : FULLA0 + sj];
        if (issuing()) {
          mbar_arrive_expect_tx(bar, TILE_A);
          tma_load_2d(dst, &map_a, hv * CHUNK, (int)(sp.bos + (long long)c * CHUNK), bar);
        }
        a_loads = tries > 0 ? j + 1 : a_loads;
        if (partial) {
          // only the last chunk of a sequence (the first one walked) can be partial: used once
          WAIT(PRIVA, 0);
          zero_rows(dst, 1, valid, &bars[FULLA0 + sj]);
        }
      }
      if (it + 2 < n_it) fetch(it + 2);
    }
    // nor a load
#pragma unroll 1
    for (int i = 1; i <= 2; ++i) {
      if (loads >= i) settle(FULL0 + ((loads - i) & 1), ((loads - i) >> 1) & 1);
      if (a_loads >= i) settle(FULLA0 + ((a_loads - i) & 1), ((a_loads - i) >> 1) & 1);
    }
  } else {
    // =============================== scaling warp (2) ===============================
    // A'' = A diag(beta gamma) (columns): thread t owns the 8 columns 8 (t%8) .. of the rows
    // t/8 + 4 i, its scale factors stay in registers and the eight threads of a row touch one
    // 128-byte line per access.
    const int c8 = lane & 7, r0 = lane >> 3;
    for (int it = 0; it < n_it; ++it, fill()) {
      const int s = it & 1;
      WAIT(FULLA0 + s, (it >> 1) & 1);
      if (it > 0) WAIT(W_DONE, (it - 1) & 1);  // w of the chunk before has been issued and is done
      const float* vs = vec + (it & 3) * VEC_SLOT_FLOATS;
      const unsigned char* src = smem + OFF_STAGE + s * STAGE_BYTES + 3 * TILE;
      const float4 g0 = *reinterpret_cast<const float4*>(vs + V_BG * CHUNK + 8 * c8);
      const float4 g1 = *reinterpret_cast<const float4*>(vs + V_BG * CHUNK + 8 * c8 + 4);
#pragma unroll 4
      for (int i = 0; i < 16; ++i) {
        const int row = r0 + 4 * i, off = row * 128 + (c8 ^ (row & 7)) * 16;
        const uint4 a = *reinterpret_cast<const uint4*>(src + off);
        *reinterpret_cast<uint4*>(smem + OFF_APP + off) =
            make_uint4(scale2(a.x, g0.x, g0.y), scale2(a.y, g0.z, g0.w), scale2(a.z, g1.x, g1.y),
                       scale2(a.w, g1.z, g1.w));
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        ARRIVE(AP_READY);
        ARRIVE(EMPTYA0 + s);  // the A tile of this stage is no longer read
      }
    }
  }
  }  // switch

  // ---- teardown ----
  if (tries <= 0) *abort_flag = 1;
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
  if (tid == 0 && *abort_flag) atomicCAS(&g_bwd_dh_status, 0, 1);
}

int bwd_dh_tc_status(int* out, int reset) {
  int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_bwd_dh_status, sizeof(int));
  if (e != cudaSuccess) return (int)e;
  *out = v;
  if (reset && v != 0) {
    int z = 0;
    e = cudaMemcpyToSymbol(g_bwd_dh_status, &z, sizeof(int));
  }
  return (int)e;
}

// ---- host side --------------------------------------------------------------------------------
int make_tile_map(CUtensorMap* m, const void* ptr, long long rows, long long cols, int box_rows);

int launch_bwd_dh_tc(const fqla_bwd_dh_args& a, int N, SeqLayout lay, cudaStream_t st) {
  using namespace bdtc;
  CUtensorMap mq, mk, mdo, ma, mdh, mdu;
  const long long T_rows = (long long)a.B * a.T;
  int rc;
  if ((rc = make_tile_map(&mq, a.q, T_rows, (long long)a.Hq * D, 64))) return rc;
  if ((rc = make_tile_map(&mk, a.k, T_rows, (long long)a.Hq * D, 64))) return rc;
  if ((rc = make_tile_map(&mdo, a.dO, T_rows, (long long)a.Hv * D, 64))) return rc;
  if ((rc = make_tile_map(&ma, a.A, T_rows, (long long)a.Hv * CHUNK, 64))) return rc;
  mdh = mq;
  mdu = mq;
  if (a.operand_tiles) {
    // an upper bound of the chunk count: the maps only have to cover what the kernel stores
    const long long max_chunks = (T_rows + CHUNK - 1) / CHUNK + N;
    if (a.dh && (rc = make_tile_map(&mdh, a.dh, max_chunks * a.Hv * D, D, 128))) return rc;
    if (a.du && (rc = make_tile_map(&mdu, a.du, max_chunks * a.Hv * D, CHUNK, 128))) return rc;
  }
  BwdDhTcParams p;
  p.tiled = a.operand_tiles;
  p.order = a.seq_order;
  p.lead = a.lead_chunks;
  p.run_mask = a.run_mask;
  p.run_value = a.run_value;
  p.warm = a.warm_chunks;
  p.zero_word = a.zero_word;
  p.g = a.g_cum; p.beta = a.beta; p.beta_is_f32 = a.beta_is_f32;
  p.dht = a.dht; p.seg_dht = a.seg_dht; p.dht_row = a.dht_row; p.dh0_row = a.dh0_row;
  p.v_first = a.state_v_first;
  p.dh = (bf16*)a.dh; p.du = (bf16*)a.du; p.dh0 = a.dh0;
  p.N = N; p.Hq = a.Hq; p.Hv = a.Hv; p.scale = a.scale; p.lay = lay;
  static std::atomic<unsigned long long> done;
  rc = configure_smem((const void*)bwd_dh_tc_kernel, SMEM_BYTES, done);
  if (rc != 0) return rc;
  return launch_pdl(bwd_dh_tc_kernel, dim3((unsigned)(N * a.Hv)), dim3(512), (size_t)SMEM_BYTES, st, p, mq,
                    mk, mdo, ma, mdh, mdu);
}

}  // namespace fqla
