// Chunk-parallel part of the gated-delta-rule backward on Blackwell tensor cores (K = V = 128).
//
// Same mathematics and same outputs as bwd_main.cu (the reference's tests/ref_gdr.py:427-600,
// evaluated by the reference kernels inside blackwell/fused_bwd.py:595-862).  Persistent CTAs
// (one per SM) walk the work items (chunk, value head).  With v_new = A W, W = beta (V - gamma K S):
//     dW = A^T du,   dL = -dW v_new^T below the diagonal (A = (I + L)^-1: the gradient through the inverse
//                    needs no product with A but the one in dW),   X = beta G dL,   Y = dW h^T
//     ds = scale G (dO v_new^T)
//     dq = scale gamma dO h^T + ds K,   dv = beta dW
//     dk = rho v_new dh^T - beta gamma Y + ds^T q + (X + X^T) K
// and dg, dbeta from row and column sums of q dq1, k dk1, k Y, v dW, ds (Q K^T), dL (K K^T).  (As the chain
// dA = -(du h^T) (beta gamma K)^T + du (beta V)^T, dL = -A^T dA A^T it was sixteen products and six
// read-outs in a row instead of eleven and three: 262144 tokens x 8 heads 1471 -> 1340 us.  With waits that pause
// between two tries (mbar_wait in tc05.cuh) 1260 to 1280, 5.7 TB/s; 32768 packed x 32 heads 686 -> 650, 4096 x 8
// heads 30.9 -> 29.0.)
// All tile products are tcgen05.mma with M = 64 (rows = tokens) and fp32 accumulators in tensor memory;
// two M = 64 accumulators share each column range (lanes +0 and +16 of every 32-lane quarter).
//
// Roles: warp 16 issues every product and every TMA load (one elected thread).  Warps 0-7 (chain
// group) make operands of accumulators (dW, ds, X + X^T as bf16 tiles in shared memory), read in the
// 16-lane shape, and dv; warps 8-15 (bulk group) do what is off the dependent chain: the h.dh sum, the row
// sums of dq1 and dk1, and the final dq | dk, read in the 32-lane shape with 16-byte shared and global
// accesses.  The sides are coupled by one mbarrier per product group (commit -> read-out) and one per
// operand tile (written -> may be multiplied), so that the chain
//     dW -> D3 = dW v_new^T -> (X + X^T) K
// never waits for the bulk work.  Operand tiles of the next item are fetched as soon as the buffers of the
// current one are dead (k has two buffers).
#include <cuda.h>

#include <climits>
#include <mutex>

#include "common.cuh"
#include "fqla_internal.h"
#include "tc05.cuh"

namespace fqla {

using namespace tc;

// set to 1 when a CTA of this file's kernel abandoned a bounded wait; read through
// fqla_device_status together with the forward kernel's word
__device__ int g_bwd_main_status = 0;

struct BwdMainTcParams {
  const float* g;
  const void* beta;
  int beta_is_f32;
  bf16* dq;
  bf16* dk;
  bf16* dv;
  void* db;                // fp32 or (db_bf16) bf16
  float* dg;
  int dg_cumsum, db_bf16;  // see fqla_bwd_main_args
  int* next_item;          // !CLC: zero at launch; see the walk of the items below
  int Hq, Hv;
  float scale;
  SeqLayout lay;
  IndexTable chunk_indices;
  long long n_chunks;
};

namespace bmtc {
constexpr int D = 128;
constexpr int N_EPI = 512;       // read-out threads: 16 warps = 4 lane quarters x 4 column quarters
constexpr int NT = N_EPI + 32;   // + the issue warp
constexpr int ROW_TILE = 16384;  // [64 x 128] bf16 as two 64-column blocks
constexpr int SQ_TILE = 32768;   // [128 x 128] bf16 as two 64-column blocks of 128 rows
constexpr int OFF_Q = 0, OFF_K = OFF_Q + ROW_TILE;  // k: two buffers
constexpr int OFF_V = OFF_K + 2 * ROW_TILE;
constexpr int OFF_VN = OFF_V + ROW_TILE, OFF_DO = OFF_VN + ROW_TILE, OFF_DU = OFF_DO + ROW_TILE;
constexpr int OFF_H = OFF_DU + ROW_TILE;
constexpr int OFF_DH = OFF_H + SQ_TILE;
constexpr int OFF_A = OFF_DH + SQ_TILE;
constexpr int OFF_DS = OFF_A + 8192;
constexpr int OFF_X = OFF_DS + 8192;        // X + X^T, X = beta dL
constexpr int OFF_DW = OFF_X + 8192;        // dW = A^T du
// g, gamma, rho, beta of an item (64 floats each; two buffers); partial sums: of dg by row (chain group:
// 2 x 64; bulk group: 4 x 64) and by column (4 x 64), of db by row (chain and bulk group 2 x 64 each), of
// the chunk total (8) and what suffix_sum64 needs (2)
constexpr int OFF_VEC = OFF_DW + ROW_TILE;
constexpr int OFF_BAR = OFF_VEC + (2 * 256 + 128 + 3 * 256 + 18) * 4;
constexpr int N_BARS = 22;
constexpr int OFF_MISC = OFF_BAR + N_BARS * 8;
constexpr int OFF_ITEM = OFF_MISC + 32;  // ring of four items, published by the issue warp
constexpr int OFF_CLAIM = (OFF_ITEM + 4 * 32 + 15) / 16 * 16;  // CLC: two answers of 16 bytes
constexpr int SMEM_BYTES = OFF_CLAIM + 2 * 16 + 1024;
static_assert(SMEM_BYTES <= 232448, "one CTA's shared memory");
// the operand tiles of one item arrive in four groups
constexpr uint32_t TX_D = 8192 + 2 * ROW_TILE;  // A, du, v
constexpr uint32_t TX_A = 3 * ROW_TILE;         // dO, v_new, k (other buffer)
constexpr uint32_t TX_H = 2 * SQ_TILE;          // h, dh
// tensor memory: (column, lane half) of every accumulator; each has a place of its own
constexpr uint32_t HI = 16u << 16;
constexpr uint32_t T_DQ1 = 0, T_DK1 = 0 + HI;      // dO h^T | v_new dh^T
constexpr uint32_t T_DQ2 = 128, T_DK2 = 128 + HI;  // ds K | ds^T q + (X + X^T) K
constexpr uint32_t T_DW = 256, T_Y = 256 + HI;     // A^T du | dW h^T
constexpr uint32_t T_DS = 384, T_D3 = 384 + HI;    // dO v_new^T | dW v_new^T
constexpr uint32_t T_QK = 448, T_KK = 448 + HI;
enum {
  L_D = 0, L_A, L_H, L_Q,                // TMA groups landed
  C_DW, C_DSQK, C_D3, C_1B, C_2, C_5,    // product groups complete (commit)
  R_ZERO,                                // all 16 read-out warps -> issue warp (partial chunks only)
  R_DW, R_DS, R_D3,                      // the 8 warps of the chain group -> issue warp
  R_CH,                                  // ... -> bulk group: item finished
  R_HD, R_E4, R_END,                     // the 8 warps of the bulk group -> issue warp
  I_NEXT,                                // issue warp -> read-out warps: the next item is in the ring
  I_CLAIM,                               // CLC: the answer with the next item has arrived
  SETTLED                                // all products have come to their end
};
}  // namespace bmtc

__device__ __forceinline__ void epi_barrier() {  // the 16 read-out warps only
  asm volatile("bar.sync 1, 512;" ::: "memory");
}
__device__ __forceinline__ void chain_barrier() {  // warps 0-7
  asm volatile("bar.sync 4, 256;" ::: "memory");
}
__device__ __forceinline__ void bulk_barrier() {  // warps 8-15
  asm volatile("bar.sync 5, 256;" ::: "memory");
}

// Persistent: CTA b starts with work item b and takes the next one that nobody has; item w = (chunk
// w / Hv, head w % Hv), so neighbouring CTAs share q and k of a grouped-value-attention group through
// L2.  SMs differ in speed by a fifth (instruction fetch), and with a fixed share each the fast ones run
// away: a tail, and CTAs working far apart in memory.  262144 tokens x 8 heads, 7.1 GB, before the
// present algebra: 1472 us (4.8 TB/s) counted out by next_item; 1492 us where the caller brings no counter
// and the grid has a block for every item, those that run taking the items of those that have not started
// (CLC, cluster launch control: the answer takes longer than that of an atomic); 1970-2090 us with a fixed
// share, 1650 us with a fixed share and the 16 warps in step (see the end of an item).
// TILED: h, dh, vnew and du arrive in the operand layouts written by the sequential kernels
// (h^T, dh^T as [V][K] per chunk; vnew^T, du^T as [V][64] per chunk) instead of row-major.
template <bool TILED, bool CLC>
__global__ void __launch_bounds__(bmtc::NT, 1)
bwd_main_tc_kernel(const BwdMainTcParams p, const __grid_constant__ CUtensorMap map_q,
                   const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                   const __grid_constant__ CUtensorMap map_vn, const __grid_constant__ CUtensorMap map_do,
                   const __grid_constant__ CUtensorMap map_du, const __grid_constant__ CUtensorMap map_h,
                   const __grid_constant__ CUtensorMap map_dh, const __grid_constant__ CUtensorMap map_a) {
  using namespace bmtc;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_MISC);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + OFF_MISC + 4);
  volatile int* stop_flag = reinterpret_cast<volatile int*>(smem + OFF_MISC + 8);  // [group][item parity]
  // per-row vectors g, gamma, rho, beta of an item: two buffers (item parity), the second one
  // behind the column sums
  float* sVec0 = reinterpret_cast<float*>(smem + OFF_VEC);
  float* sRowDg = sVec0 + 256;
  float* sColDg = sRowDg + 128;
  float* sRowDb = sColDg + 256;
  float* sVec1 = sRowDb + 256;
  float* sRowW = sVec1 + 256;  // row terms of the 128-wide steps: [column half x lane half][row]
  float* sLast = sRowW + 256;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long total = p.n_chunks * p.Hv;

  struct Item {
    long long row0, chunk_id;
    int valid, hv, hq;
  };
  Item* ring = reinterpret_cast<Item*>(smem + OFF_ITEM);
  const int group = p.Hv / p.Hq;
  // Claiming an item and reading the tables of a packed batch are three dependent loads.  The issue
  // warp spreads them over the waits of the item before, the low words (row numbers fit) straight
  // into the registers they stay in, and hands the item to the read-out warps through a ring in
  // shared memory: read where the item begins the tables cost every warp 1500 of 14500 cycles.
  struct Raw {
    int seq, ci, begin, end, base;
  };
  auto low = [](const IndexTable& t, int i) { return reinterpret_cast<const int*>(t.ptr)[t.is64 ? 2 * i : i]; };
  auto load_index = [&](int cidx, Raw& r) {
    if (p.lay.cu.ptr) {
      r.seq = low(p.chunk_indices, 2 * cidx);
      r.ci = low(p.chunk_indices, 2 * cidx + 1);
    } else {
      const int per = (p.lay.T + CHUNK - 1) / CHUNK;
      r.seq = cidx / per;
      r.ci = cidx % per;
    }
  };
  auto load_span = [&](Raw& r) {
    if (p.lay.cu.ptr) {
      r.begin = low(p.lay.cu, r.seq);
      r.end = low(p.lay.cu, r.seq + 1);
      r.base = low(p.lay.chunk_offsets, r.seq);
    }
  };
  auto finish = [&](const Raw& r, int hv) {
    Item t;
    t.hv = hv;
    t.hq = hv / group;
    const bool packed = p.lay.cu.ptr != nullptr;
    const long long bos = packed ? r.begin : (long long)r.seq * p.lay.T;
    const int len = packed ? r.end - r.begin : p.lay.T;
    t.row0 = bos + (long long)r.ci * CHUNK;
    // clamped: a table row that does not belong to its sequence must not index outside the tiles
    t.valid = max(1, min(CHUNK, len - r.ci * CHUNK));
    t.chunk_id = (packed ? r.base : (long long)r.seq * ((p.lay.T + CHUNK - 1) / CHUNK)) + r.ci;
    return t;
  };
  if (tid == 0) {
    for (int i = L_D; i <= C_5; ++i) mbar_init(&bars[i], 1);
    mbar_init(&bars[R_ZERO], N_EPI / 32);
    for (int i = R_DW; i <= R_END; ++i) mbar_init(&bars[i], N_EPI / 64);
    mbar_init(&bars[I_NEXT], 1);
    if (CLC) mbar_init(&bars[I_CLAIM], 1);
    mbar_init(&bars[SETTLED], 1);
    *abort_flag = 0;
    for (int i = 0; i < 4; ++i) stop_flag[i] = 0;
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(tmem_slot, 512);
  pdl_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  int tries = WAIT_TRIES;  // see mbar_wait; filled up for each item; used up, a thread signals and stores no more
  auto WAIT = [&](int idx, uint32_t parity) { mbar_wait(&bars[idx], parity, tries); };

  if (warp == N_EPI / 32) {
    // ====================== issue warp: TMA loads and every tcgen05.mma ======================
    // (the warp stays converged; see elect_one in tc05.cuh)
    {
      auto WAIT = [&](int idx, uint32_t parity) { return mbar_wait_uniform(&bars[idx], parity, tries); };
      // Four groups, in the order in which their buffers become free (A and du are dead after the first
      // product of an item, q only after the bulk group has read it).
      auto load_d = [&](const Item& t) {
        const int y = (int)t.row0;
        if (!elect_one()) return;
        mbar_arrive_expect_tx(&bars[L_D], TX_D);
        tma_load_2d(smem + OFF_A, &map_a, t.hv * CHUNK, y, &bars[L_D]);
        if constexpr (TILED) {
          tma_load_2d(smem + OFF_DU, &map_du, 0, (int)((t.chunk_id * p.Hv + t.hv) * D), &bars[L_D]);
        } else {
          tma_load_2d(smem + OFF_DU, &map_du, t.hv * D, y, &bars[L_D]);
          tma_load_2d(smem + OFF_DU + 8192, &map_du, t.hv * D + 64, y, &bars[L_D]);
        }
        tma_load_2d(smem + OFF_V, &map_v, t.hv * D, y, &bars[L_D]);
        tma_load_2d(smem + OFF_V + 8192, &map_v, t.hv * D + 64, y, &bars[L_D]);
      };
      auto load_a = [&](const Item& t, int kbuf) {
        const int y = (int)t.row0, ys = (int)((t.chunk_id * p.Hv + t.hv) * D);
        if (!elect_one()) return;
        mbar_arrive_expect_tx(&bars[L_A], TX_A);
        tma_load_2d(smem + OFF_DO, &map_do, t.hv * D, y, &bars[L_A]);
        tma_load_2d(smem + OFF_DO + 8192, &map_do, t.hv * D + 64, y, &bars[L_A]);
        if constexpr (TILED) {
          tma_load_2d(smem + OFF_VN, &map_vn, 0, ys, &bars[L_A]);
        } else {
          tma_load_2d(smem + OFF_VN, &map_vn, t.hv * D, y, &bars[L_A]);
          tma_load_2d(smem + OFF_VN + 8192, &map_vn, t.hv * D + 64, y, &bars[L_A]);
        }
        tma_load_2d(smem + OFF_K + kbuf * ROW_TILE, &map_k, t.hq * D, y, &bars[L_A]);
        tma_load_2d(smem + OFF_K + kbuf * ROW_TILE + 8192, &map_k, t.hq * D + 64, y, &bars[L_A]);
        mbar_arrive_expect_tx(&bars[L_H], TX_H);
        tma_load_2d(smem + OFF_H, &map_h, 0, ys, &bars[L_H]);
        tma_load_2d(smem + OFF_H + 16384, &map_h, 64, ys, &bars[L_H]);
        tma_load_2d(smem + OFF_DH, &map_dh, 0, ys, &bars[L_H]);
        tma_load_2d(smem + OFF_DH + 16384, &map_dh, 64, ys, &bars[L_H]);
      };
      auto load_q = [&](const Item& t) {
        if (!elect_one()) return;
        mbar_arrive_expect_tx(&bars[L_Q], ROW_TILE);
        tma_load_2d(smem + OFF_Q, &map_q, t.hq * D, (int)t.row0, &bars[L_Q]);
        tma_load_2d(smem + OFF_Q + 8192, &map_q, t.hq * D + 64, (int)t.row0, &bars[L_Q]);
      };
      // descriptors (low words)
      const uint32_t q_lo = desc_lo_kmajor(smem + OFF_Q), qmn_lo = desc_lo_mnmajor(smem + OFF_Q, 8192);
      const uint32_t k_lo0 = desc_lo_kmajor(smem + OFF_K), kmn_lo0 = desc_lo_mnmajor(smem + OFF_K, 8192);
      const uint32_t vn_lo = desc_lo_kmajor(smem + OFF_VN), dumn_lo = desc_lo_mnmajor(smem + OFF_DU, 8192);
      const uint32_t do_lo = desc_lo_kmajor(smem + OFF_DO), du_lo = desc_lo_kmajor(smem + OFF_DU);
      const uint32_t h_lo = desc_lo_kmajor(smem + OFF_H), dh_lo = desc_lo_kmajor(smem + OFF_DH);
      const uint32_t amn_lo = desc_lo_mnmajor(smem + OFF_A, 8192), dw_lo = desc_lo_kmajor(smem + OFF_DW);
      const uint32_t ds_lo = desc_lo_kmajor(smem + OFF_DS), dsmn_lo = desc_lo_mnmajor(smem + OFF_DS, 8192);
      const uint32_t x_lo = desc_lo_kmajor(smem + OFF_X);
      // operand-tile layouts: [V rows][K or token columns], read MN-major, contraction over rows
      const uint32_t hT_lo = desc_lo_mnmajor(smem + OFF_H, 16384), dhT_lo = desc_lo_mnmajor(smem + OFF_DH, 16384);
      const uint32_t vnT_lo = desc_lo_mnmajor(smem + OFF_VN, 16384);
      constexpr uint32_t ID_KK_128 = idesc_bf16(64, 128, 0, 0), ID_KK_64 = idesc_bf16(64, 64, 0, 0);
      constexpr uint32_t ID_KM_128 = idesc_bf16(64, 128, 0, 1), ID_MM_128 = idesc_bf16(64, 128, 1, 1);
      constexpr uint32_t ID_KM_64 = idesc_bf16(64, 64, 0, 1), ID_MK_128 = idesc_bf16(64, 128, 1, 0);
      constexpr uint32_t KBUF_LO = ROW_TILE >> 4;

      Raw raw = {};
      int claimed = (int)blockIdx.x;  // in lane 0
      unsigned char* answers = smem + OFF_CLAIM;  // two slots, by item parity
      load_index((int)blockIdx.x / p.Hv, raw);
      load_span(raw);
      Item cur = finish(raw, (int)blockIdx.x % p.Hv);
      load_d(cur);
      load_a(cur, 0);
      load_q(cur);
      uint32_t it = 0, zero_ph = 0;
      // An accumulator or an operand tile is written again only behind a barrier that says it has been
      // read: what the chain group reads (dW, ds, qk, KK, D3) behind its own arrivals on the tiles it makes
      // of them, what the bulk group reads (dq, dk, Y) behind R_END of the item before.
#pragma unroll 1
      for (bool has_next = true; has_next; ++it) {
        tries = WAIT_TRIES;
        const uint32_t ph = it & 1;
        if (!CLC && lane == 0) claimed = (int)gridDim.x + atomicAdd(p.next_item, 1);
        const uint32_t k_lo = k_lo0 + (ph ? KBUF_LO : 0u), kmn_lo = kmn_lo0 + (ph ? KBUF_LO : 0u);
        // A partial chunk waits until the read-out warps have zeroed the rows past the sequence end (which
        // also means that all its tiles have landed).
        const bool partial = cur.valid != CHUNK;
        if (partial) {
          if (it > 0) {  // q of this item, below for a full chunk
            if (!(WAIT(C_2, ph ^ 1) && WAIT(R_E4, ph ^ 1))) break;
            load_q(cur);
          }
          if (!WAIT(R_ZERO, zero_ph)) break;
          zero_ph ^= 1;
        } else {
          if (!WAIT(L_D, ph)) break;
        }
        tc_fence_after();
        // ---- dW = A^T du: needs nothing but A and du ----
        if (elect_one()) {
          if constexpr (TILED) umma_group<4, 128, 0, 2, 0, false>(tmem + T_DW, amn_lo, du_lo, ID_MK_128);
          else umma_group<4, 128, 0, 128, 0, false>(tmem + T_DW, amn_lo, dumn_lo, ID_MM_128);
          umma_commit(&bars[C_DW]);
          if constexpr (CLC) {
            mbar_arrive_expect_tx(&bars[I_CLAIM], 16);
            clc_try_cancel(answers + 16 * ph, &bars[I_CLAIM]);
          }
        }
        if (!partial) {
          if (it > 0) {
            // q of the item before is dead: its product is complete, the bulk group has used it
            if (!(WAIT(C_2, ph ^ 1) && WAIT(R_E4, ph ^ 1))) break;
            load_q(cur);
          }
          if (!(WAIT(L_A, ph) && WAIT(L_Q, ph))) break;
          tc_fence_after();
        }
        // ---- ds, q k^T, K K^T ----
        if (elect_one()) {
          if constexpr (TILED) umma_group<8, 2, 512, 128, 512, false>(tmem + T_DS, do_lo, vnT_lo, ID_KM_64);
          else umma_group<8, 2, 512, 2, 512, false>(tmem + T_DS, do_lo, vn_lo, ID_KK_64);
          umma_group<8, 2, 512, 2, 512, false>(tmem + T_QK, q_lo, k_lo, ID_KK_64);
          umma_commit(&bars[C_DSQK]);
          umma_group<8, 2, 512, 2, 512, false>(tmem + T_KK, k_lo, k_lo, ID_KK_64);
        }
        // ---- dW is an operand now: D3 = dW v_new^T ----
        if (!WAIT(R_DW, ph)) break;
        tc_fence_after();
        if (elect_one()) {
          if constexpr (TILED) umma_group<8, 2, 512, 128, 512, false>(tmem + T_D3, dw_lo, vnT_lo, ID_KM_64);
          else umma_group<8, 2, 512, 2, 512, false>(tmem + T_D3, dw_lo, vn_lo, ID_KK_64);
          umma_commit(&bars[C_D3]);
        }
        int w_next;
        if constexpr (CLC) {
          if (!WAIT(I_CLAIM, ph)) break;
          w_next = clc_block(answers + 16 * ph);
          fence_proxy_async();  // read before the request after the next one writes the slot
          has_next = w_next >= 0;
        } else {
          w_next = __shfl_sync(0xffffffffu, claimed, 0);
          has_next = w_next < (int)total;
        }
        const int h_next = has_next ? w_next % p.Hv : 0;
        if (has_next) load_index(w_next / p.Hv, raw);
        // ---- Y = dW h^T, dq1, dk1: off the chain ----
        if (!(WAIT(L_H, ph) && (it == 0 || WAIT(R_END, ph ^ 1)))) break;
        tc_fence_after();
        if (elect_one()) {
          if constexpr (TILED) {
            umma_group<8, 2, 512, 128, 512, false>(tmem + T_Y, dw_lo, hT_lo, ID_KM_128);
            umma_group<8, 2, 512, 128, 512, false>(tmem + T_DQ1, do_lo, hT_lo, ID_KM_128);
            umma_group<8, 128, 512, 128, 512, false>(tmem + T_DK1, vnT_lo, dhT_lo, ID_MM_128);
          } else {
            umma_group<8, 2, 512, 2, 1024, false>(tmem + T_Y, dw_lo, h_lo, ID_KK_128);
            umma_group<8, 2, 512, 2, 1024, false>(tmem + T_DQ1, do_lo, h_lo, ID_KK_128);
            umma_group<8, 2, 512, 2, 1024, false>(tmem + T_DK1, vn_lo, dh_lo, ID_KK_128);
          }
          umma_commit(&bars[C_1B]);
        }
        if (has_next) load_span(raw);
        // ---- ds is an operand now ----
        if (!WAIT(R_DS, ph)) break;
        tc_fence_after();
        if (elect_one()) {
          umma_group<4, 2, 0, 128, 0, false>(tmem + T_DQ2, ds_lo, kmn_lo, ID_KM_128);
          umma_group<4, 128, 0, 128, 0, false>(tmem + T_DK2, dsmn_lo, qmn_lo, ID_MM_128);
          umma_commit(&bars[C_2]);
        }
        Item nxt = cur;
        if (has_next) {
          nxt = finish(raw, h_next);
          load_d(nxt);  // A, du and v are dead: the chain group made dW, dv and what follows of them
        } else {
          nxt.valid = 0;  // the read-out warps stop
        }
        if (lane == 0) {
          ring[(it + 1) & 3] = nxt;
          mbar_arrive(&bars[I_NEXT]);
        }
        // ---- dk += (X + X^T) K with X = beta dL, onto ds^T q ----
        if (!WAIT(R_D3, ph)) break;
        tc_fence_after();
        if (elect_one()) {
          umma_group<4, 2, 0, 128, 0, true>(tmem + T_DK2, x_lo, kmn_lo, ID_KM_128);
          umma_commit(&bars[C_5]);
        }
        // h, dh, dO, v_new are dead once their products are complete and the h.dh sum is done; the other
        // k buffer belonged to the item before, which R_END above has seen finished
        if (has_next) {
          if (!(WAIT(C_1B, ph) && WAIT(R_HD, ph))) break;
          load_a(nxt, (int)(ph ^ 1));
        }
        cur = nxt;
      }
      // No product is under way when the block goes, and no load: where this warp came through it has waited for
      // all of them, else whichever phase of theirs is open is waited for.
      if (elect_one()) umma_commit(&bars[SETTLED]);
      int again = WAIT_TRIES;
      mbar_wait(&bars[SETTLED], 0, again);
      if (again <= 0) tries = 0;
      if (tries <= 0) {
#pragma unroll 1
        for (int i = 0; i < (CLC ? 10 : 8); ++i) {
          again = WAIT_TRIES / 64;
          mbar_wait(&bars[i < 8 ? L_D + (i >> 1) : I_CLAIM], i & 1, again);
        }
      }
    }
  } else {
    // ====================== read-out warps ======================
    // Two groups of eight warps.  The CHAIN group (warps 0-7) serves the dependent chain (plus ds, which
    // it gets from the same kind of tile): it reads accumulators in the 16-lane shape (lane l of warp
    // (qd, half) owns rows 16 qd + l/4 (+8), column pairs 8 i + 2 (l%4) of half the columns).  The BULK
    // group (warps 8-15) does everything that is off the chain.  It reads the 128-wide accumulators in the
    // 32-lane shape, which returns the accumulator at lanes +0 and the one at lanes +16 of the
    // same columns at once: lane l owns row 16 qd + l%16 of the lower (l < 16) or upper one, 32
    // consecutive columns per pass; shared and global memory are touched 16 bytes at a time.
    const bool chain = warp < 8;
    const int gw = warp & 7, qd = gw & 3, half = gw >> 2;
    const int row_a = 16 * qd + (lane >> 2), row_b = row_a + 8, cp = 2 * (lane & 3);
    const int row_w = 16 * qd + (lane & 15);
    const bool hi = lane >= 16;
    const uint32_t lanes = (uint32_t)(qd * 32) << 16;
    const int c64 = 32 * half;    // first column of this warp in 64-wide tiles (chain group)
    const int c128 = 64 * half;   // first column of this warp in 128-wide tiles
    // byte offset of this thread's 16-byte piece (pass, j) (8 columns) inside a [64 x 128] row tile
    const int piece_base = half * 8192 + row_w * 128;
    auto piece = [&](int pass, int j) { return piece_base + (((4 * pass + j) ^ (row_w & 7)) << 4); };
    auto quad_sum = [&](float x) {
      x += __shfl_xor_sync(0xffffffffu, x, 1);
      x += __shfl_xor_sync(0xffffffffu, x, 2);
      return x;
    };
    auto col_sum = [&](float x) {
      x += __shfl_xor_sync(0xffffffffu, x, 4);
      x += __shfl_xor_sync(0xffffffffu, x, 8);
      x += __shfl_xor_sync(0xffffffffu, x, 16);
      return x;
    };
    auto pack8 = [&](const float* x) {
      return make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
    };
    // 32 consecutive columns of this thread's output row (bf16) go out. A thread owns a
    // row, so a plain 16-byte store per thread would touch 32 lines per instruction; the four
    // lanes of a quad first exchange their 16-byte pieces (a 4 x 4 transpose, two butterfly
    // steps), after which each store instruction writes 64 contiguous bytes of 8 rows.
    // base = offset of the row of lane 0 of the quad (+ the 32-column block), row_q = that row.
    auto store_rows = [&](bf16* out, long long base, int row_q, int valid_rows, uint4 (&pc)[4]) {  // whole warp
      const bool b0 = lane & 1, b1 = lane & 2;
      auto xchg = [&](uint4& keep_if0, uint4& keep_if1, bool bit, int mask) {
        // lanes with bit clear keep keep_if0 and send keep_if1; lanes with bit set the reverse
        uint4 snd = bit ? keep_if0 : keep_if1, rcv;
        rcv.x = __shfl_xor_sync(0xffffffffu, snd.x, mask);
        rcv.y = __shfl_xor_sync(0xffffffffu, snd.y, mask);
        rcv.z = __shfl_xor_sync(0xffffffffu, snd.z, mask);
        rcv.w = __shfl_xor_sync(0xffffffffu, snd.w, mask);
        if (bit) keep_if0 = rcv; else keep_if1 = rcv;
      };
      xchg(pc[0], pc[1], b0, 1);
      xchg(pc[2], pc[3], b0, 1);
      xchg(pc[0], pc[2], b1, 2);
      xchg(pc[1], pc[3], b1, 2);
      // pc[j] now holds piece (lane & 3) of row row_q + j
      const long long pitch = (long long)p.Hv * D;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (row_q + j < valid_rows)
          *reinterpret_cast<uint4*>(out + base + j * pitch + 8 * (lane & 3)) = pc[j];
    };
    // this warp's part of a tile (or of the accumulators) is done: tell the issue warp
    auto signal = [&](int bar) {
      fence_proxy_async();
      tc_fence_before();
      __syncwarp();
      if (lane == 0 && tries > 0) mbar_arrive(&bars[bar]);
    };
    auto zero_rows = [&](int off, int n_blocks, int valid) {
#pragma unroll 1
      for (int blk = 0; blk < n_blocks; ++blk) {
        unsigned char* base = smem + off + blk * 8192;
#pragma unroll 1
        for (int i = tid; i < (CHUNK - valid) * 8; i += N_EPI)
          *reinterpret_cast<uint4*>(base + (valid + (i >> 3)) * 128 + ((i & 7) << 4)) = make_uint4(0, 0, 0, 0);
      }
    };
    // The vectors of the next item are fetched a whole item ahead.  beta stays in its raw form
    // until it is used: a conversion right behind the load would make the thread wait for it.
    float pre_g = 0.f, pre_gl = 0.f;
    uint32_t pre_beta_raw = 0;
    auto fetch_vectors = [&](const Item& t) {
      if (tid < CHUNK) {
        const int r = min(tid, t.valid - 1);
        const long long i = (t.row0 + r) * p.Hv + t.hv;
        pre_g = p.g[i];
        pre_gl = p.g[(t.row0 + t.valid - 1) * p.Hv + t.hv];
        pre_beta_raw = p.beta_is_f32 ? reinterpret_cast<const uint32_t*>(p.beta)[i]
                                     : (uint32_t)reinterpret_cast<const unsigned short*>(p.beta)[i];
      }
    };
    // the fetched vectors of item t go to buffer `buf` (threads 0..63; published by a barrier)
    auto write_vectors = [&](const Item& t, float* buf) {
      if (tid < CHUNK) {
        buf[tid] = pre_g;
        buf[64 + tid] = fast_exp(pre_g);
        buf[128 + tid] = fast_exp(pre_gl - pre_g);
        buf[192 + tid] =
            tid < t.valid ? __uint_as_float(p.beta_is_f32 ? pre_beta_raw : pre_beta_raw << 16) : 0.f;
      }
    };
    // dg, db of a finished item from the partial sums in shared memory (threads 256..319, which
    // would otherwise idle until the first wide products are complete)
    auto combine = [&](long long first, int n_rows) {  // first = row0 * Hv + hv of the item
      const int r = tid - N_EPI / 2;
      if (r < 0 || r >= CHUNK) return;  // two whole warps go on
      float dgv = 0.f, dbv = 0.f;
      if (r < n_rows) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          dgv += sRowW[j * 64 + r] - sColDg[j * 64 + r];
          dbv += sRowDb[j * 64 + r];
        }
        dgv += sRowDg[r] + sRowDg[64 + r];
        if (r == n_rows - 1) {
#pragma unroll
          for (int j = 0; j < 8; ++j) dgv += sLast[j];
        }
      }
      if (p.dg_cumsum) dgv = suffix_sum64(dgv, r, sLast + 16);
      if (r < n_rows) {
        const long long i = first + (long long)r * p.Hv;
        p.dg[i] = dgv;
        if (p.db_bf16) reinterpret_cast<bf16*>(p.db)[i] = __float2bfloat16(dbv);
        else reinterpret_cast<float*>(p.db)[i] = dbv;
      }
    };
    Raw raw = {};
    load_index((int)blockIdx.x / p.Hv, raw);
    load_span(raw);
    Item cur = finish(raw, (int)blockIdx.x % p.Hv);
    long long prev_first = 0;
    int prev_rows = 0;
    fetch_vectors(cur);
    write_vectors(cur, sVec0);
    epi_barrier();
    uint32_t it = 0;
#pragma unroll 1
    for (;; ++it) {
      const uint32_t ph = it & 1;
      const int valid = cur.valid;
      const int koff = OFF_K + (int)ph * ROW_TILE;
      const float* sG = ph ? sVec1 : sVec0;
      const float *sGam = sG + 64, *sRho = sG + 128, *sBeta = sG + 192;
      tries = WAIT_TRIES;
      if (valid < CHUNK) {
        WAIT(L_D, ph);
        WAIT(L_A, ph);
        WAIT(L_H, ph);
        WAIT(L_Q, ph);
        zero_rows(OFF_Q, 2, valid);
        zero_rows(koff, 2, valid);
        zero_rows(OFF_A, 1, valid);
        if constexpr (TILED) zero_rows(OFF_DO, 2, valid);  // the transposed tiles already hold zeros
        else zero_rows(OFF_VN, 6, valid);                  // v_new, dO, du
        signal(R_ZERO);
      }
      Item nxt;
      // the next item, from the middle of this one on
      auto take_next = [&] {
        WAIT(I_NEXT, ph);
        nxt = ring[(it + 1) & 3];
        if (tries <= 0) nxt.valid = 0;  // not there: nothing more
      };
      float acc_last = 0.f;

      if (chain) {
        // ===================== chain group =====================
        const float beta_a = sBeta[row_a], beta_b = sBeta[row_b];
        // row sums (dg, db) and column sums (dg) of this thread; reduced across lanes once, at the end
        // of the item
        float acc_dg_a = 0.f, acc_dg_b = 0.f, acc_db_a = 0.f, acc_db_b = 0.f;
        float acc_col[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc_col[j] = 0.f;

        // ---- E1: dW = A^T du as an operand tile; dv = beta dW, made of v in place; db += dW v ----
        // the products that read the operand tile of the item before are complete (C_1B)
        WAIT(C_DW, ph);
        if (it > 0) WAIT(C_1B, ph ^ 1);
        WAIT(L_D, ph);
        {
          tc_fence_after();
          const int rows = tries > 0 ? valid : 0;  // (nothing is stored of what is not complete)
          float x[32];
          tmem_ld_16x64(tmem + lanes + T_DW + 64 * half, x);
          tmem_ld_wait();
          // 16-byte pieces 2 j, 2 j + 1 of rows 0-7 and 8-15 of this warp's [16 x 64] block: one
          // stmatrix / ldmatrix with the addresses of lane's row
          const uint32_t line = (uint32_t)(half * 8192 + (16 * qd + 8 * ((lane >> 3) & 1) + (lane & 7)) * 128);
          auto at = [&](int j) { return line + (uint32_t)(((2 * j + (lane >> 4)) ^ (lane & 7)) << 4); };
#pragma unroll
          for (int j = 0; j < 4; ++j)
            stmatrix_x4(s32(smem + OFF_DW) + at(j), pack_bf16(x[8 * j], x[8 * j + 1]), pack_bf16(x[8 * j + 2], x[8 * j + 3]),
                        pack_bf16(x[8 * j + 4], x[8 * j + 5]), pack_bf16(x[8 * j + 6], x[8 * j + 7]));
          signal(R_DW);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t vr[4];
            ldmatrix_x4_addr(vr, s32(smem + OFF_V) + at(j));
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 t = __bfloat1622float2(*reinterpret_cast<const bf162*>(&vr[e]));
              const float x0 = x[8 * j + 2 * e], x1 = x[8 * j + 2 * e + 1];
              if (e & 1) acc_db_b += x0 * t.x + x1 * t.y;
              else acc_db_a += x0 * t.x + x1 * t.y;
              const float b = e & 1 ? beta_b : beta_a;
              vr[e] = pack_bf16(b * x0, b * x1);
            }
            stmatrix_x4(s32(smem + OFF_V) + at(j), vr[0], vr[1], vr[2], vr[3]);
          }
          __syncwarp();
          // out again as whole lines: eight threads write 128 contiguous bytes of a row
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int row = 16 * qd + 4 * j + (lane >> 3);
            const uint4 w = *reinterpret_cast<const uint4*>(smem + OFF_V + half * 8192 + row * 128 +
                                                            (((lane & 7) ^ (row & 7)) << 4));
            if (row < rows)
              *reinterpret_cast<uint4*>(p.dv + ((cur.row0 + row) * p.Hv + cur.hv) * D + 64 * half + 8 * (lane & 7)) = w;
          }
        }

        // ---- E2: ds = scale * G * (dO Vn^T); ds2 = ds * (Q K^T) ----
        WAIT(C_DSQK, ph);
        if (it > 0) WAIT(C_2, ph ^ 1);
        const float g_a = sG[row_a], g_b = sG[row_b];
        // address of this lane's row in a [16 x 32] block of a 64-column tile, 16-byte piece 4 half + i
        const uint32_t line = (uint32_t)((16 * qd + 8 * ((lane >> 3) & 1) + (lane & 7)) * 128);
        {
          tc_fence_after();
          float ds[16], qk[16];
          tmem_ld_16x32(tmem + lanes + T_DS + c64, ds);
          tmem_ld_16x32(tmem + lanes + T_QK + c64, qk);
          tmem_ld_wait();
          uint32_t w[8];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int col = c64 + 8 * i + cp;
            const float gc0 = sG[col], gc1 = sG[col + 1];
            const float a0 = col <= row_a ? p.scale * ds[4 * i] * fast_exp(g_a - gc0) : 0.f;
            const float a1 = col + 1 <= row_a ? p.scale * ds[4 * i + 1] * fast_exp(g_a - gc1) : 0.f;
            const float b0 = col <= row_b ? p.scale * ds[4 * i + 2] * fast_exp(g_b - gc0) : 0.f;
            const float b1 = col + 1 <= row_b ? p.scale * ds[4 * i + 3] * fast_exp(g_b - gc1) : 0.f;
            w[2 * i] = pack_bf16(a0, a1);
            w[2 * i + 1] = pack_bf16(b0, b1);
            const float s0 = a0 * qk[4 * i], s1 = a1 * qk[4 * i + 1], s2 = b0 * qk[4 * i + 2], s3 = b1 * qk[4 * i + 3];
            acc_dg_a += s0 + s1;
            acc_dg_b += s2 + s3;
            acc_col[2 * i] += s0 + s2;
            acc_col[2 * i + 1] += s1 + s3;
          }
#pragma unroll
          for (int i = 0; i < 2; ++i)
            stmatrix_x4(s32(smem + OFF_DS) + line + (uint32_t)(((4 * half + 2 * i + (lane >> 4)) ^ (lane & 7)) << 4),
                        w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
        }
        signal(R_DS);

        // ---- E7: X = beta dL, dL = -G D3 below the diagonal, D3 = dW v_new^T; X + X^T as an operand
        //      tile; the dg and db terms of dL * (K K^T) ----
        WAIT(C_D3, ph);
        if (it > 0) WAIT(C_5, ph ^ 1);
        {
          tc_fence_after();
          float d3[16], kk[16];
          tmem_ld_16x32(tmem + lanes + T_D3 + c64, d3);
          tmem_ld_16x32(tmem + lanes + T_KK + c64, kk);
          tmem_ld_wait();
          const uint32_t tile = s32(smem + OFF_X);
          const int r8 = lane & 7, second = (lane >> 3) & 1;  // which of two matrices this lane addresses
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int cb = 4 * half + i;  // 8-column block; this warp's 8-row blocks are 2 qd, 2 qd + 1
            if (cb > 2 * qd + 1) continue;  // above the diagonal: written by the warp of the mirrored block
            const int col = c64 + 8 * i + cp;
            const float gc0 = sG[col], gc1 = sG[col + 1];
            const float a0 = col < row_a ? -d3[4 * i] * fast_exp(g_a - gc0) : 0.f;
            const float a1 = col + 1 < row_a ? -d3[4 * i + 1] * fast_exp(g_a - gc1) : 0.f;
            const float b0 = col < row_b ? -d3[4 * i + 2] * fast_exp(g_b - gc0) : 0.f;
            const float b1 = col + 1 < row_b ? -d3[4 * i + 3] * fast_exp(g_b - gc1) : 0.f;
            // db += rowsum((dL K) k) = rowsum(dL * (K K^T)); the dg terms carry the beta factor
            const float u0 = a0 * kk[4 * i], u1 = a1 * kk[4 * i + 1], u2 = b0 * kk[4 * i + 2], u3 = b1 * kk[4 * i + 3];
            acc_db_a += u0 + u1;
            acc_db_b += u2 + u3;
            const float s0 = u0 * beta_a, s1 = u1 * beta_a, s2 = u2 * beta_b, s3 = u3 * beta_b;
            acc_dg_a += s0 + s1;
            acc_dg_b += s2 + s3;
            acc_col[2 * i] += s0 + s2;
            acc_col[2 * i + 1] += s1 + s3;
            // blocks (2 qd, cb) and (2 qd + 1, cb), and mirrored (cb, 2 qd) and (cb, 2 qd + 1)
            uint32_t wa = pack_bf16(col < row_a ? beta_a * a0 : 0.f, col + 1 < row_a ? beta_a * a1 : 0.f);
            uint32_t wb = pack_bf16(col < row_b ? beta_b * b0 : 0.f, col + 1 < row_b ? beta_b * b1 : 0.f);
            const uint32_t straight = tile + (uint32_t)((16 * qd + 8 * second + r8) * 128 + ((cb ^ r8) << 4));
            const uint32_t mirrored = tile + (uint32_t)((8 * cb + r8) * 128 + (((2 * qd + second) ^ r8) << 4));
            if (cb < 2 * qd) {
              stmatrix_x2(straight, wa, wb);
              stmatrix_x2_trans(mirrored, wa, wb);
            } else if (cb == 2 * qd) {  // the upper one of the two lies on the diagonal
              stmatrix_x2(straight, wa | movmatrix_trans(wa), wb);
              stmatrix_x1_trans(tile + (uint32_t)((8 * cb + r8) * 128 + (((2 * qd + 1) ^ r8) << 4)), wb);
            } else {  // the upper one lies above the diagonal, the lower one on it
              stmatrix_x1(tile + (uint32_t)((16 * qd + 8 + r8) * 128 + ((cb ^ r8) << 4)), wb | movmatrix_trans(wb));
            }
          }
        }
        signal(R_D3);
        take_next();
        if (nxt.valid > 0) fetch_vectors(nxt);
        // The partial-sum slots were read for the previous item by two warps of the bulk group (combine), which
        // arrive on R_E4 of this item only after that: both groups wait for it before they write theirs.
        WAIT(R_E4, ph);
        // one reduction per quantity, one plain store per (warp, row or column): no atomics
        acc_dg_a = quad_sum(acc_dg_a);
        acc_dg_b = quad_sum(acc_dg_b);
        acc_db_a = quad_sum(acc_db_a);
        acc_db_b = quad_sum(acc_db_b);
        if ((lane & 3) == 0) {
          sRowDg[half * 64 + row_a] = acc_dg_a;
          sRowDg[half * 64 + row_b] = acc_dg_b;
          sRowDb[half * 64 + row_a] = acc_db_a;
          sRowDb[half * 64 + row_b] = acc_db_b;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float c = col_sum(acc_col[j]);
          if (lane < 4) sColDg[qd * 64 + c64 + 8 * (j >> 1) + cp + (j & 1)] = c;
        }
      } else {
        // ===================== bulk group =====================
        // gamma_last * sum(h * dh) over the whole 128 x 128 tiles (plain shared-memory reads)
        WAIT(L_A, ph);
        WAIT(L_H, ph);
        {
          float hd = 0.f;
#pragma unroll 2  // (unrolled as far as the compiler goes: 1 to 2 % of small launches in instruction fetches)
          for (int i = tid - N_EPI / 2; i < SQ_TILE / 16; i += N_EPI / 2) {
            const uint4 a = *reinterpret_cast<const uint4*>(smem + OFF_H + i * 16);
            const uint4 b = *reinterpret_cast<const uint4*>(smem + OFF_DH + i * 16);
            const uint32_t* pa = &a.x;
            const uint32_t* pb = &b.x;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              float2 fa = __bfloat1622float2(*reinterpret_cast<const bf162*>(&pa[e]));
              float2 fb = __bfloat1622float2(*reinterpret_cast<const bf162*>(&pb[e]));
              hd += fa.x * fb.x + fa.y * fb.y;
            }
          }
          acc_last += sGam[CHUNK - 1] * hd;
        }
        __syncwarp();
        if (lane == 0 && tries > 0) mbar_arrive(&bars[R_HD]);
        if (it > 0) combine(prev_first, prev_rows);  // fits into the wait for the first wide products
        const float f_w = hi ? sRho[row_w] : p.scale * sGam[row_w];
        const int row_q = row_w - (lane & 3);  // row of lane 0 of this quad
        const long long out_q = ((cur.row0 + row_q) * p.Hv + cur.hv) * D + c128;
        float acc_w = 0.f;

        // ---- E4: the dg terms of dq1 = scale gamma (dO h^T) on the lower lanes, dk1 = rho (Vn dh^T) on
        //      the upper ----
        WAIT(C_1B, ph);
        WAIT(L_Q, ph);
        {
          tc_fence_after();
          const unsigned char* tile = smem + (hi ? koff : OFF_Q);
#pragma unroll 1
          for (int pass = 0; pass < 2; ++pass) {
            float x[32];
            tmem_ld32(tmem + lanes + T_DQ1 + c128 + 32 * pass, x);
            tmem_ld_wait();
            float s = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint4 raw = *reinterpret_cast<const uint4*>(tile + piece(pass, j));
              const uint32_t* pr = &raw.x;
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 t = __bfloat1622float2(*reinterpret_cast<const bf162*>(&pr[e]));
                s += t.x * x[8 * j + 2 * e] + t.y * x[8 * j + 2 * e + 1];
              }
            }
            // dg += rowsum(q dq1) - rowsum(k dk1); the chunk total gets + sum(k dk1)
            s *= f_w;
            acc_w += hi ? -s : s;
            if (hi) acc_last += s;
          }
        }
        signal(R_E4);  // q is no longer read from shared memory
        take_next();   // (before R_END: the item after the next is published only behind that)

        // ---- E8: dq = dq1 + ds K (lower lanes); dk = dk1 - beta gamma Y + [ds^T q + (X + X^T) K] (upper
        //      lanes), and the dg and db terms of Y = dW h^T ----
        // (R_E4: the two warps of combine have read the sums of the item before, see the chain group)
        WAIT(R_E4, ph);
        WAIT(C_5, ph);
        {
          tc_fence_after();
          const int rows = tries > 0 ? valid : 0;
          bf16* out = hi ? p.dk : p.dq;
          const float f_y = hi ? -sBeta[row_w] * sGam[row_w] : 0.f;
          float s = 0.f;
#pragma unroll 1
          for (int pass = 0; pass < 2; ++pass) {
            uint4 pc[4];
#pragma unroll
            for (int z = 0; z < 2; ++z) {
              float x[16], y[16], w[16];
              const uint32_t col = c128 + 32 * pass + 16 * z;
              tmem_ld16(tmem + lanes + T_DQ1 + col, x);
              tmem_ld16(tmem + lanes + T_DQ2 + col, y);
              tmem_ld16(tmem + lanes + T_DW + col, w);  // upper lanes: Y; lower lanes: dW, not used
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                const uint4 raw = *reinterpret_cast<const uint4*>(smem + koff + piece(pass, 2 * z + j));
                const uint32_t* pr = &raw.x;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const float2 t = __bfloat1622float2(*reinterpret_cast<const bf162*>(&pr[e]));
                  const int c = 8 * j + 2 * e;
                  const float w0 = hi ? w[c] : 0.f, w1 = hi ? w[c + 1] : 0.f;
                  s += t.x * w0 + t.y * w1;
                  x[c] = f_w * x[c] + y[c] + f_y * w0;
                  x[c + 1] = f_w * x[c + 1] + y[c + 1] + f_y * w1;
                }
                pc[2 * z + j] = pack8(x + 8 * j);
              }
            }
            store_rows(out, out_q + 32 * pass, row_q, rows, pc);
          }
          acc_w += f_y * s;
          if (hi) sRowDb[128 + half * 64 + row_w] = -sGam[row_w] * s;
        }
        signal(R_END);  // accumulators and k of this item are free
        sRowW[(2 * half + (hi ? 1 : 0)) * 64 + row_w] = acc_w;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) acc_last += __shfl_xor_sync(0xffffffffu, acc_last, d);
        if (lane == 0) sLast[gw] = acc_last;
      }
      // The chain group goes on to the next item as soon as it is through; the bulk group, which
      // ends an item with the wide read-outs, follows at most an item behind (R_E4) and finds the
      // chain group's contributions to dg, db and the vectors of the next item (other buffer)
      // behind R_CH.  (One barrier of all sixteen warps here held the chain group for the last
      // wide read-out, 1600 of 14500 cycles per item.)  A thread that has given a wait up takes its group
      // along: each group has a stop flag of its own, by item parity, so that it is read by the whole group before
      // it can be written again, and behind the barrier all threads of a group go the same way.
      const int stop = (chain ? 0 : 2) + (int)ph;
      if (chain) {
        if (nxt.valid > 0) write_vectors(nxt, ph ? sVec0 : sVec1);
      } else {
        WAIT(R_CH, ph);
      }
      if (tries <= 0) stop_flag[stop] = 1;
      if (chain) {
        __syncwarp();
        if (lane == 0 && tries > 0) mbar_arrive(&bars[R_CH]);
        chain_barrier();
      } else {
        bulk_barrier();
      }
      prev_first = cur.row0 * p.Hv + cur.hv;
      prev_rows = cur.valid;
      cur = nxt;
      if (stop_flag[stop]) break;
      if (nxt.valid == 0) {
        combine(prev_first, prev_rows);
        break;
      }
    }
  }
  if (tries <= 0) *abort_flag = 1;
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
  if (tid == 0 && *abort_flag) atomicCAS(&g_bwd_main_status, 0, 1);
}

int bwd_main_tc_status(int* out, int reset) {
  int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_bwd_main_status, sizeof(int));
  if (e != cudaSuccess) return (int)e;
  *out = v;
  if (reset && v != 0) {
    int z = 0;
    e = cudaMemcpyToSymbol(g_bwd_main_status, &z, sizeof(int));
  }
  return (int)e;
}


// ---- host side --------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn2)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// 2-D bf16 tensor map, rows x cols (row-major), box = 64 columns x box_rows rows, 128-byte swizzle.
// Encoding a map costs about a microsecond on the host and a launch needs four to nine of them, so
// the last maps are kept in a small table keyed by (pointer, shape, box): a steady-state step that
// reuses its buffers (a framework's caching allocator, a CUDA graph's private pool) encodes nothing.
// A map only describes addresses and extents, so an entry stays valid when the buffer is freed and
// an equal allocation returns at the same address.
int make_tile_map(CUtensorMap* m, const void* ptr, long long rows, long long cols, int box_rows) {
  static EncodeTiledFn2 fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess)
      f = nullptr;
    return (EncodeTiledFn2)f;
  }();
  if (!fn) return FQLA_ERR_INVALID_ARG;
  struct Entry {
    const void* ptr;
    long long rows, cols;
    int box_rows, used;
    CUtensorMap map;
  };
  constexpr int N_ENTRIES = 128;
  static Entry table[N_ENTRIES] = {};
  static std::mutex lock;
  const uint64_t hsh = ((uint64_t)(uintptr_t)ptr >> 8) * 0x9E3779B97F4A7C15ull ^
                       ((uint64_t)rows * 0xC2B2AE3D27D4EB4Full) ^ ((uint64_t)cols << 17) ^
                       (uint64_t)box_rows;
  Entry& e = table[(hsh >> 32) % N_ENTRIES];
  {
    std::lock_guard<std::mutex> hold(lock);
    if (e.used && e.ptr == ptr && e.rows == rows && e.cols == cols && e.box_rows == box_rows) {
      *m = e.map;
      return 0;
    }
  }
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  cuuint32_t es[2] = {1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides,
                  box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return FQLA_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> hold(lock);
  e.ptr = ptr; e.rows = rows; e.cols = cols; e.box_rows = box_rows; e.map = *m; e.used = 1;
  return 0;
}

int launch_bwd_main_tc(const fqla_bwd_main_args& a, long long n_chunks, SeqLayout lay,
                       IndexTable chunk_indices, cudaStream_t st) {
  using namespace bmtc;
  CUtensorMap mq, mk, mv, mvn, mdo, mdu, mh, mdh, ma;
  const long long T_rows = (long long)a.B * a.T;
  const int Hq = a.Hq, Hv = a.Hv;
  int rc;
  if ((rc = make_tile_map(&mq, a.q, T_rows, (long long)Hq * D, 64))) return rc;
  if ((rc = make_tile_map(&mk, a.k, T_rows, (long long)Hq * D, 64))) return rc;
  if ((rc = make_tile_map(&mv, a.v, T_rows, (long long)Hv * D, 64))) return rc;
  if (a.operand_tiles) {
    if ((rc = make_tile_map(&mvn, a.vnew, n_chunks * Hv * D, CHUNK, 128))) return rc;
    if ((rc = make_tile_map(&mdu, a.du, n_chunks * Hv * D, CHUNK, 128))) return rc;
  } else {
    if ((rc = make_tile_map(&mvn, a.vnew, T_rows, (long long)Hv * D, 64))) return rc;
    if ((rc = make_tile_map(&mdu, a.du, T_rows, (long long)Hv * D, 64))) return rc;
  }
  if ((rc = make_tile_map(&mdo, a.dO, T_rows, (long long)Hv * D, 64))) return rc;
  if ((rc = make_tile_map(&mh, a.h, n_chunks * Hv * D, D, 128))) return rc;
  if ((rc = make_tile_map(&mdh, a.dh, n_chunks * Hv * D, D, 128))) return rc;
  if ((rc = make_tile_map(&ma, a.A, T_rows, (long long)Hv * CHUNK, 64))) return rc;
  BwdMainTcParams p;
  p.g = a.g_cum; p.beta = a.beta; p.beta_is_f32 = a.beta_is_f32;
  p.dq = (bf16*)a.dq; p.dk = (bf16*)a.dk; p.dv = (bf16*)a.dv; p.db = a.db; p.dg = a.dg;
  p.dg_cumsum = a.dg_cumsum; p.db_bf16 = a.db_is_bf16;
  p.Hq = Hq; p.Hv = Hv; p.scale = a.scale; p.lay = lay; p.chunk_indices = chunk_indices;
  p.n_chunks = n_chunks;
  p.next_item = a.next_item;
  const long long total = n_chunks * Hv;
  if (total > INT_MAX) return FQLA_ERR_TOO_LARGE;
  auto launch = [&](auto kernel, std::atomic<unsigned long long>& done, long long blocks) {
    int err = configure_smem((const void*)kernel, SMEM_BYTES, done);
    if (err != 0) return err;
    return launch_pdl(kernel, dim3((unsigned)blocks), dim3(NT), (size_t)SMEM_BYTES, st, p, mq, mk, mv, mvn, mdo,
                      mdu, mh, mdh, ma);
  };
  static std::atomic<unsigned long long> done[4];
  if (!p.next_item)
    return a.operand_tiles ? launch(bwd_main_tc_kernel<true, true>, done[0], total)
                           : launch(bwd_main_tc_kernel<false, true>, done[1], total);
  const long long n_sm = sm_count(), blocks = total < n_sm ? total : n_sm;
  return a.operand_tiles ? launch(bwd_main_tc_kernel<true, false>, done[2], blocks)
                         : launch(bwd_main_tc_kernel<false, false>, done[3], blocks);
}

}  // namespace fqla
