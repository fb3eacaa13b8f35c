// Sequential forward recurrence of the gated delta rule on Blackwell tensor cores:
// TMA-fed tcgen05.mma with all accumulators in tensor memory, warp-specialised.
//
// One CTA (640 threads; 512 without outputs) walks the chunks of one (sequence or segment, value head),
// K = V = 128.
// Per chunk, with S [K x V] the fp32 state entering the chunk, A the gated inverse from
// kkt_solve, g the chunk-local cumulative log gate (gamma = exp g, rho = exp(g_last - g)):
//
//   off the serial chain, prepared one chunk ahead (WY form, FLA's w and u):
//     A'  = A diag(beta),  A'' = A diag(beta gamma)                               (prep group)
//     u^T [v x tok] = V^T A'^T          (A operand = V tile read MN-major)        -> TM_UV
//     w^T [k x tok] = K^T A''^T         (A operand = K tile read MN-major)        -> TM_W -> smem
//     P   [tok x tok'] = Q K^T,  Pg = s P exp(g_tok - g_tok') for tok >= tok'     (prep group)
//   on the chain (two products):
//     Vn^T [v x tok] = u^T - S^T w^T    (A = bf16 copy of S^T, negated; accumulates onto u^T)
//     S^T  [v x k]   = gamma_last S^T + (rho Vn)^T K     (B = K tile read MN-major)
//   output, transposed so that it shares the A operands of the chain:
//     O1^T [v x tok] = S^T Q^T,   O2^T [v x tok] = Vn^T Pg^T,   o = s gamma_tok O1 + O2
//
// The state path is kept TRANSPOSED: the 128-wide value dimension sits on the MMA M axis
// (tensor-memory lane = value index, one thread per lane), so every product but P has M = 128.
// Every operand that a read-out warp derives from an accumulator - the bf16 copy of S^T, Vn^T and
// rho Vn^T - goes back into TENSOR MEMORY (two bf16 per 32-bit column) and is consumed as the A
// operand of the next product straight from there (tcgen05.mma with A in tensor memory): the
// chunk-to-chunk chain never touches shared memory, and the tensor pipe, which is bound by the
// shared-memory fetch of its operands, reads half as much.  This is the algebra of the
// reference's blackwell/fused_fwd.py:349-596 (and the X/Y form of prepare_h.py:312-318) with the
// gate folded into A.
//
// Warp roles:
//     warps 4-7,   S group : fp32 master state in tensor memory; per chunk packs the bf16 operand copy of S^T
//                            into tensor memory (on the chain), then decays S^T in place
//     warps 8-11,  V group : Vn^T -> rho-scaled and plain bf16 operand copies (tensor memory, on the chain);
//                            w^T -> bf16 operand tile (shared memory)
//     warps 12-15, O group : output epilogue o = s gamma O1 + O2
//     warps 16-19, prep group : A', A'' of the next chunk, P -> Pg   (warps 12-15 where nothing is output)
//     warp 0 issues the two products of the chain, warp 1 those of the output (none where nothing is output),
//     warp 3 u^T and w^T
//     warp 2, producer: per-chunk gate vectors (fetched one chunk ahead), TMA loads of the q, k, v, A tiles
//                       (2 stages), zero-fill of rows past the end of a partial chunk
//
// What bounds it: the chain of a chunk (3230 cycles on an idle chip: state copy 530, Vn^T 770, its read-out 780,
// state update 700, and the arrivals between them) and, with all SMs at work, HBM: 262144 tokens x 8 heads 454 us,
// 5.3 TB/s.  Two things had made it 4830 and 516 us (4 x 8192 x 16 heads 151 -> 131 us, 32768 packed x 32 heads with
// tiles 392 -> 353).  (1) Roles that waited for one another in a ring: one thread that issued everything off the
// chain, and an output group that built Pg between two epilogues.  No role waits here for another one's work off the
// chain, and w^T and P, which share their columns, are read out of them at once.  (2) Code: the instruction cache of
// an SM holds some 28 KB (straight code of one warp per scheduler, measured: full speed up to there, 2.5 cycles an
// instruction beyond, 10 with all SMs at it), and a chunk runs every role's loop once.  So loops are rolled to
// rounds of one tensor-memory load, and a wait is six instructions (tc05.cuh): 57 -> 49 KB, with tiles 72 -> 54.  (The
// issuing warps wait as one instead, which lets them leave where a wait is given up: 55 and 61 KB, and no slower, as
// this code is not on the way of the others: 262144 tokens x 8 heads 457 -> 454 us, 64 prompts of 135161 tokens
// 266 -> 264.5.)
//
// The state-only pass of the exact hand-off (end states and transition matrices of segments) is a
// chain of its own, because its roundings go into every segment behind the hand-off: A diag(beta),
// A diag(beta gamma) and w, each rounded to bf16, are not formed.  Instead
//     U^T [v x tok] = S^T K^T,  W^T = beta (V^T - gamma U^T),  Vn^T = W^T A^T
// three products deep, W^T and rho Vn^T made by the V and the O group together (32 tokens each), warp 0
// issuing everything.  W^T goes into its product as bf16; as the diagonal of A is one, what that rounding
// left out is simply added to Vn^T.  (Error of o of the heads that never forget, against 64 bits, 8192 to
// 16384 tokens: see the figures at the dispatch in fwd_seq.cu.)
// Synchronisation is by mbarriers only; every wait is bounded and reports through a status word.
#include <cuda.h>
#include <cuda_fp16.h>

#include <climits>
#include <cstdlib>

#include "common.cuh"
#include "fqla_internal.h"
#include "tc05.cuh"

namespace fqla {

using namespace tc;

// 0 = ok; 1 after some kernel abandoned a bounded wait (its outputs are then invalid)
__device__ int g_device_status = 0;

#ifdef FQLA_DIAGNOSTICS
// Development builds only: clock stamps of the role leaders of CTA 0 over a window of chunks,
// [role 0..5][chunk in window 0..15][tag 0..9].
__device__ long long g_fwd_trace[6 * 16 * 10];
__device__ int g_trace_cta = 0;               // which CTA records the role trace
__device__ long long g_cta_cycles[2 * 1024];  // per CTA: SM id, cycles from entry to exit
// chain issuer of CTA 0 and CTA 77: clock at the start of every chunk, [cta 0/1][chunk 0..127];
// entries 126, 127: kernel entry and exit of that CTA
__device__ long long g_fwd_chunk_clock[2 * 128];
#define FQLA_CHUNK_CLOCK(idx)                                                              \
  do {                                                                                     \
    if ((blockIdx.x == 0 || blockIdx.x == 77) && (idx) < 128)                              \
      g_fwd_chunk_clock[(blockIdx.x == 0 ? 0 : 128) + (idx)] = clock64();                  \
  } while (0)
#define FQLA_TRACE(role, tag)                                                         \
  do {                                                                                \
    if (blockIdx.x == g_trace_cta && it >= 24 && it < 40)                             \
      g_fwd_trace[((role) * 16 + (it - 24)) * 10 + (tag)] = clock64();               \
  } while (0)
#else
#define FQLA_TRACE(role, tag) do { } while (0)
#define FQLA_CHUNK_CLOCK(idx) do { } while (0)
#endif

struct FwdTcParams {
  const float* g;
  const void* beta;
  int beta_is_f32;
  const float* h0;
  const float* seg_h0;            // see fqla_fwd_args in include/fqla.h for these five
  const int *h0_row, *ht_row;
  int v_first;
  float* ht;
  bf16* o;
  bf16* h;
  bf16* vnew;
  int N, Hq, Hv;
  long long T_rows;
  float scale;
  SeqLayout lay;
  int tiled;  // h and vnew are written as operand tiles (h^T per chunk, v_new^T per chunk) by TMA
  // [N, Hv] or null: lead-in.  A CTA with lead > 0 starts from a ZERO state `lead` chunks before
  // its sequence (segment) and walks those chunks state-only (no q, no output, nothing stored):
  // the rows just before a segment are the tail of the segment before it, whose influence dies
  // out within `lead` chunks.  h0 is ignored for such a CTA.  lead < 0: -lead chunks, back to the
  // start of the sequence that the segment is cut from, and from that one's own initial state.
  const int* lead;
  // [N, Hv] or null: a CTA whose entry differs from run_value returns at once, reading and
  // writing nothing (two launches can share one set of outputs, each taking its own pairs)
  const int* run_mask;
  int run_value;
  // [N] or null: the CTAs of block index i / Hv walk sequence order[i].  Blocks start in index
  // order, so a table that lists the longest sequences first shortens the tail of a ragged batch.
  const int* order;
  // State-only variant: the blocks from m_first on compute the transition matrix M [N, Hv, D, D] (the
  // same walk from the identity with v = 0), the ones before it the end state.  warm [N, Hv] or
  // null: only the last warm[n,hv] chunks are walked, from a zero state (< 0: nothing is done);
  // m_mask [N, Hv] or null: M only where non-zero, and there of the whole sequence, whatever warm says.
  float* M;
  const int *warm, *m_mask;
  int m_first;
};

namespace fwdtc {
constexpr int D = 128;
constexpr int threads(bool no_o) { return no_o ? 512 : 640; }
constexpr int TILE_QK = 16384, TILE_V = 16384, TILE_A = 8192;
constexpr int STAGE_BYTES = 2 * TILE_QK + TILE_V + TILE_A;  // 57344
constexpr int OFF_STAGE = 0;
constexpr int OFF_W = 2 * STAGE_BYTES;           // w^T   [128 k rows x 128B (64 tokens)]
constexpr int OFF_P = OFF_W + 16384;             // Pg    [64 x 128B]
constexpr int OFF_AP = OFF_P + 8192;             // A diag(beta)
constexpr int OFF_APP = OFF_AP + 8192;           // A diag(beta gamma)
constexpr int OFF_O = OFF_APP + 8192;            // o tile [64 tok x 128 v] bf16, source of its TMA store
constexpr int OFF_VEC = OFF_O + 16384;           // 4 slots x 6 vectors x 64 floats
constexpr int VEC_SLOT_FLOATS = 6 * CHUNK;
constexpr int OFF_BAR = OFF_VEC + 4 * VEC_SLOT_FLOATS * 4;
constexpr int N_BARS = 32;
constexpr int OFF_MISC = OFF_BAR + N_BARS * 8;
// only the variants that hand per-chunk tiles to the backward pass keep shared-memory copies of
// S^T and Vn^T (the sources of their TMA stores)
constexpr int OFF_ST = (OFF_MISC + 16 + 1023) / 1024 * 1024;  // S^T copy, 2 blocks of [128 x 128B]
constexpr int OFF_VNT = OFF_ST + 32768;                       // Vn^T  [128 x 128B]
constexpr int SMEM_BYTES = OFF_ST + 1024;  // + slack for 1024-byte alignment of the base
constexpr int SMEM_BYTES_EXTRA = OFF_VNT + 16384 + 1024;
// tensor-memory columns (512).  The bf16 operands hold two elements per column.
constexpr uint32_t TM_S = 0;      // S^T fp32                      128 columns
constexpr uint32_t TM_SB = 128;   // S^T bf16 (A operand, K = 128)  64 columns
constexpr uint32_t TM_UV = 192;   // u^T, then Vn^T fp32            64 columns
constexpr uint32_t TM_VNB = 256;  // Vn^T bf16 (A operand, K = 64)  32 columns
constexpr uint32_t TM_VRB = 288;  // rho Vn^T bf16                  32 columns
constexpr uint32_t TM_O1 = 320;   // O1^T fp32                      64 columns
constexpr uint32_t TM_O2 = 384;   // O2^T fp32                      64 columns
// w^T of a chunk (M = 128) and, once the value group has made its operand tile of it, P (M = 64: lanes
// 0-15 of each quarter) take turns in the same columns.
constexpr uint32_t TM_W = 448, TM_P = TM_W;
// state-only pass
constexpr uint32_t TM_U = TM_UV;    // U^T fp32                   64 columns
constexpr uint32_t TM_WB = TM_VNB;  // W^T bf16 (A operand)       32 columns
constexpr uint32_t TM_VN = TM_O1;   // Vn^T fp32                  64 columns
// barrier indices
enum { FULL0 = 0, FULL1, EMPTY0, EMPTY1, S_COPY, S_DEC, VN_DONE, S_DONE, P_DONE, O_DONE,
       // w^T, u^T of a chunk are complete (state-only pass: U^T)
       W_DONE, U_DONE,
       VB_READY, W_READY, P_READY, O_FREE, AP_READY, PRIV,
       // the A tile and the per-row vectors of a chunk travel one chunk ahead of q, k, v
       FULLA0, FULLA1, EMPTYA0, EMPTYA1, PRIVA,
       // tile outputs: the shared-memory copies of S^T / Vn^T are complete
       ST_READY, VN_READY,
       // the output product that reads the packed copy of S^T has completed
       SB_FREE,
       // P has been read
       P_FREE,
       // all products have come to their end
       SETTLED,
       // state-only pass: W^T, made by the V and the O group, is there
       WB_READY = P_READY };
// vectors inside a slot; V_GL holds gamma_last at [0], V_BG -beta gamma instead of beta gamma in
// the state-only pass
enum { V_G = 0, V_BETA = 1, V_BG = 2, V_RHO = 3, V_SGAM = 4, V_GL = 5 };
}  // namespace fwdtc

__device__ __forceinline__ uint32_t scale_bf16x2(uint32_t packed, float lo, float hi) {
  float2 f = __bfloat1622float2(*reinterpret_cast<const bf162*>(&packed));
  return pack_bf16(f.x * lo, f.y * hi);
}

template <bool F16>
__device__ __forceinline__ uint32_t pack_out(float lo, float hi) {
  if constexpr (F16) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  } else {
    return pack_bf16(lo, hi);
  }
}

// EXTRA: per-chunk state and v_new outputs (compiled out of the common instantiation, whose code
// does not fit the instruction cache as it is).  NO_O: state-only walk, no q, no output products: with EXTRA the
// recomputation for the backward pass (the output warps have nothing to do), without it (STATE) the end states
// and M of the exact hand-off.  O_F16: o leaves as fp16 instead of bf16.
template <bool EXTRA, bool NO_O, bool O_F16>
__global__ void __launch_bounds__(fwdtc::threads(NO_O), 1)
fwd_tc_kernel(const FwdTcParams p, const __grid_constant__ CUtensorMap map_q,
              const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
              const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_h,
              const __grid_constant__ CUtensorMap map_vn, const __grid_constant__ CUtensorMap map_o) {
  using namespace fwdtc;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_MISC);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + OFF_MISC + 4);
  float* vec = reinterpret_cast<float*>(smem + OFF_VEC);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr bool STATE = NO_O && !EXTRA;
  constexpr int NT = threads(NO_O);
  constexpr int PREP = NO_O ? 12 : 16;  // first warp of the prep group
  const bool m_pass = STATE && (int)blockIdx.x >= p.m_first;
  const int block = m_pass ? (int)blockIdx.x - p.m_first : (int)blockIdx.x;
  const int hv = block % p.Hv;
  auto sequence = [&] { return p.order ? p.order[block / p.Hv] : block / p.Hv; };
  const int hq = hv / (p.Hv / p.Hq);
  if (p.run_mask) {
    pdl_wait();
    if (p.run_mask[sequence() * p.Hv + hv] != p.run_value) return;  // uniform per CTA
  }
  int warm = INT_MAX;
  if (STATE && (p.warm || p.m_mask)) {
    pdl_wait();
    const int item = sequence() * p.Hv + hv;
    const int masked = m_pass && p.m_mask ? p.m_mask[item] : 1;
    if (p.warm) warm = p.warm[item];
    if (warm < 0 || masked == 0) return;  // uniform per CTA
    if (m_pass && p.m_mask) warm = INT_MAX;
  }
  const bool tile_h = EXTRA && p.tiled && p.h, tile_vn = EXTRA && p.tiled && p.vnew;

  if (tid == 0) FQLA_CHUNK_CLOCK(126);
#ifdef FQLA_DIAGNOSTICS
  const long long g_fwd_chunk_clock_entry = clock64();
#endif
  if (tid == 0) {
    mbar_init(&bars[FULL0], 1);
    mbar_init(&bars[FULL1], 1);
    mbar_init(&bars[EMPTY0], STATE ? 1 : NO_O ? 2 : 3);  // MMA commits of the issuing threads
    mbar_init(&bars[EMPTY1], STATE ? 1 : NO_O ? 2 : 3);
    mbar_init(&bars[SB_FREE], 1);
    mbar_init(&bars[P_FREE], 128);
    mbar_init(&bars[SETTLED], STATE ? 1 : NO_O ? 2 : 3);
    mbar_init(&bars[U_DONE], 1);
    mbar_init(&bars[FULLA0], 1);
    mbar_init(&bars[FULLA1], 1);
    // the only reader of the raw A tile: the prep group, or (STATE) a product
    mbar_init(&bars[EMPTYA0], STATE ? 1 : 128);
    mbar_init(&bars[EMPTYA1], STATE ? 1 : 128);
    mbar_init(&bars[PRIVA], 1);
    mbar_init(&bars[S_COPY], 128);
    mbar_init(&bars[S_DEC], 128);
    mbar_init(&bars[VN_DONE], 1);
    mbar_init(&bars[S_DONE], 1);
    mbar_init(&bars[P_DONE], 1);
    mbar_init(&bars[O_DONE], 1);
    mbar_init(&bars[W_DONE], 1);
    mbar_init(&bars[VB_READY], STATE ? 256 : 128);
    mbar_init(&bars[W_READY], 128);
    mbar_init(&bars[P_READY], STATE ? 256 : 128);
    mbar_init(&bars[O_FREE], 128);
    mbar_init(&bars[AP_READY], 128);
    mbar_init(&bars[PRIV], 1);
    mbar_init(&bars[ST_READY], 128);
    mbar_init(&bars[VN_READY], 128);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    tma_prefetch_desc(&map_a);
  }
  // Pg is lower triangular: its tile is zeroed once, the prep group only ever rewrites the column
  // groups that can be non-zero for its rows
  for (int i = tid; i < 8192 / 16; i += NT)
    *reinterpret_cast<uint4*>(smem + OFF_P + i * 16) = make_uint4(0, 0, 0, 0);
  if (m_pass) {  // v stays zero: its tiles are never loaded
    for (int i = tid; i < 2 * TILE_V / 16; i += NT)
      *reinterpret_cast<uint4*>(smem + OFF_STAGE + 2 * TILE_QK + (i & 1023) * 16 + (i >> 10) * STAGE_BYTES) =
          make_uint4(0, 0, 0, 0);
  }
  fence_proxy_async();
  if (warp == 0) tmem_alloc(tmem_slot, 512);
  // everything above overlaps the tail of the kernel before: no global memory up to here
  pdl_wait();
  const int n = sequence();
  const SeqSpan sp = p.lay.span(n);
  // iteration j handles chunk c = j - lead of the sequence; c < 0 are the lead-in chunks
  // (lead < 0: the first -lead chunks are left out)
  const int lead_in = !STATE && p.lead ? p.lead[n * p.Hv + hv] : 0;
  const int lead = STATE ? min(warm, sp.n_chunks) - sp.n_chunks : abs(lead_in);
  const int n_it = sp.n_chunks == 0 ? 0 : sp.n_chunks + lead;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;  // this warp's lane quarter
  int tries = WAIT_TRIES;  // see mbar_wait; filled up for each pass of a role's loop
  auto WAIT = [&](int idx, uint32_t parity) { mbar_wait(&bars[idx], parity, tries); };
  auto WAITU = [&](int idx, uint32_t parity) { return mbar_wait_uniform(&bars[idx], parity, tries); };
  auto fill = [&] { tries = tries > 0 ? WAIT_TRIES : tries; };
  // A thread that has given a wait up issues, signals and stores nothing more.  An issuing warp leaves its loop as one.
  // The others walk theirs to the end, as their lanes each count for themselves and what follows are instructions of
  // whole warps (a vote on the way out, once a chunk, cost 1 %: three prompts of 985 tokens x 64 heads 30.8 us
  // instead of 30.5), one try a wait.
  auto ARRIVE = [&](int idx) { mbar_arrive_if(&bars[idx], tries); };
  auto issuing = [&] { return elect_one() && tries > 0; };  // of the producer
  // At the end of a role that issues: a wait with a limit of its own.
  auto settle = [&](int idx, uint32_t parity) {
    int again = WAIT_TRIES;
    mbar_wait(&bars[idx], parity, again);
    if (again <= 0) tries = 0;
  };

  // Initial state -> tensor memory, S^T[v][k]; zero without one and for a lead-in.  The three
  // read-out groups share the columns 2 : 1 : 1, each thread with its whole part in flight at once:
  // one memory latency (four in turn, 3 us of an 11 us launch over two chunks, when the state group
  // loaded 32 columns at a time by itself).
  if (warp >= 4 && warp < 16) {
    int h0_row = p.h0_row ? p.h0_row[n] : n;
    if (lead_in < 0) h0_row = ~h0_row;
    const bool edge = h0_row >= 0;  // starts its sequence; else it is handed a state, if any
    const float* src = (STATE ? lead != 0 || m_pass : lead_in > 0) ? nullptr : edge ? p.h0 : p.seg_h0;
    if (src) src += ((long long)(edge ? h0_row : n) * p.Hv + hv) * D * D;
    const int v = (warp & 3) * 32 + lane;
    auto load32 = [&](int k0, float (&x)[32]) {
      if (!src) {
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = m_pass && k0 + j == v ? 1.f : 0.f;
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

  // The single-thread roles are warps 0 to 3 on purpose: among the warps of one scheduler the oldest
  // (lowest id) wins when several are ready, and these must never queue behind the compute groups.
  // A switch and not a chain of ifs: every test of a chain stands behind the code of the role before it, a line to
  // fetch from L2 each at the start of a launch (the last role came to its loop 2400 cycles behind the first barrier).
  const int role = STATE && warp >= 8 ? 5 : NO_O && warp >= 12 ? 4 : warp >> 2;
  switch (role) {
  case 1: {
    // =============================== S group ===============================
    const int v = tid - 128;  // lane of tensor memory = value index
#pragma unroll 1
    for (int it = 0; it < n_it; ++it, fill()) {
      const int s = it & 1;
      if (v == 0) FQLA_TRACE(0, 0);
      if (it > 0) WAIT(S_DONE, (it - 1) & 1);
      // the output product of the chunk before, issued by another thread, has read the copy (in a lead-in
      // there is none, but its issuer signals all the same: see there)
      if (!NO_O && it > 0) WAIT(SB_FREE, (it - 1) & 1);
      tc_fence_after();
      if (v == 0) FQLA_TRACE(0, 1);
      // on the chain: the bf16 operand copy of S^T, packed back into tensor memory.  (Of the products that read
      // the copy of the chunk before, Vn^T came ahead of the state update, issued by the same thread; O1^T has
      // signalled SB_FREE.)
#pragma unroll 1
      for (int k0 = 0; k0 < D; k0 += 32) {
        float x[32];
        tmem_ld32(tmem + lane_sel + TM_S + k0, x);
        tmem_ld_wait();
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) pk[i] = pack_bf16(x[2 * i], x[2 * i + 1]);
        tmem_st16(tmem + lane_sel + TM_SB + (k0 >> 1), pk);
      }
      tmem_st_wait();
      tc_fence_before();
      ARRIVE(S_COPY);
      if (v == 0) FQLA_TRACE(0, 2);
      if constexpr (EXTRA) {
        // off the chain: the state entering this chunk as an output, from the operand copy
        if (p.h && it >= lead) {
          unsigned char* row = smem + OFF_ST + v * 128;
#pragma unroll 1
          for (int kb = 0; kb < 2; ++kb) {  // 64 columns (one operand block) per round
            float x[32];
            tmem_ld32(tmem + lane_sel + TM_SB + kb * 32, x);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 8; ++c)
              *reinterpret_cast<float4*>(row + kb * 16384 + ((c ^ (v & 7)) << 4)) =
                  make_float4(x[4 * c], x[4 * c + 1], x[4 * c + 2], x[4 * c + 3]);
          }
          if (p.tiled) {
            fence_proxy_async();
            ARRIVE(ST_READY);
          } else {  // row-major [k][v]: column v, from this thread's own row
            bf16* hdst = p.h + ((sp.chunk_base + (it - lead)) * p.Hv + hv) * (long long)D * D + v;
#pragma unroll 1
            for (int k = 0; k < (tries > 0 ? D : 0); ++k)
              hdst[(long long)k * D] =
                  *reinterpret_cast<const bf16*>(smem + OFF_ST + (k >> 6) * 16384 + sw128_offset(v, k & 63));
          }
        }
      }
      // off the chain: decay in place, needed only by the state update at the end of the chunk
      WAIT(FULL0 + s, (it >> 1) & 1);
      if (v == 0) FQLA_TRACE(0, 3);
      const float gl = vec[(it & 3) * VEC_SLOT_FLOATS + V_GL * CHUNK];
#pragma unroll 1
      for (int k0 = 0; k0 < D; k0 += 32) {
        float x[32];
        tmem_ld32(tmem + lane_sel + TM_S + k0, x);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] *= gl;
        tmem_st32(tmem + lane_sel + TM_S + k0, x);
      }
      tmem_st_wait();
      tc_fence_before();
      ARRIVE(S_DEC);
      if (v == 0) FQLA_TRACE(0, 4);
    }
    if (n_it > 0) WAIT(S_DONE, (n_it - 1) & 1);
    const int ht_row = p.ht_row && !m_pass ? p.ht_row[n] : n;
    float* end = m_pass ? p.M : p.ht;
    if (__all_sync(0xffffffffu, tries > 0) && end && ht_row >= 0) {
      float* dst = end + ((long long)ht_row * p.Hv + hv) * D * D;
      tc_fence_after();
#pragma unroll 1
      for (int k0 = 0; k0 < D; k0 += 32) {
        float x[32];
        tmem_ld32(tmem + lane_sel + TM_S + k0, x);
        tmem_ld_wait();
        if (p.v_first && !m_pass) {
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
  case 5: if constexpr (STATE) {
    // =============================== V and O group, state-only pass ===============================
    // Each takes 32 tokens of a chunk: U^T -> W^T = beta (V^T - gamma U^T), Vn^T -> rho Vn^T, both bf16
    // operands in tensor memory.
    const int v = (warp & 3) * 32 + lane;  // tensor-memory lane = value index
    const int t0 = warp < 12 ? 0 : 32;
    for (int it = 0; it < n_it; ++it, fill()) {
      const int s = it & 1;
      WAIT(FULL0 + s, (it >> 1) & 1);
      const float* vs = vec + (it & 3) * VEC_SLOT_FLOATS + t0;
      // off the chain: beta V^T, this thread's value index of its 32 tokens, and -beta gamma
      const unsigned char* vt = smem + OFF_STAGE + s * STAGE_BYTES + 2 * TILE_QK + (v >> 6) * 8192;
      auto load32 = [&](const float* src, float (&a)[32]) {
#pragma unroll
        for (int i = 0; i < 8; ++i) *reinterpret_cast<float4*>(a + 4 * i) = *reinterpret_cast<const float4*>(src + 4 * i);
      };
      float x[32], y[32], f[32];
      load32(vs + V_BETA * CHUNK, y);
      load32(vs + V_BG * CHUNK, f);
#pragma unroll
      for (int j = 0; j < 32; ++j)
        y[j] = __fmul_rn(y[j], __bfloat162float(*reinterpret_cast<const bf16*>(vt + sw128_offset(t0 + j, v & 63))));
      WAIT(U_DONE, it & 1);
      tc_fence_after();
      tmem_ld32(tmem + lane_sel + TM_U + t0, x);
      tmem_ld_wait();
      uint32_t pk[16];
#pragma unroll
      for (int j = 0; j < 32; ++j) y[j] = __fmaf_rn(f[j], x[j], y[j]);
#pragma unroll
      for (int i = 0; i < 16; ++i) pk[i] = pack_bf16(y[2 * i], y[2 * i + 1]);
      tmem_st16(tmem + lane_sel + TM_WB + (t0 >> 1), pk);
      tmem_st_wait();
      tc_fence_before();
      ARRIVE(WB_READY);
      // off the chain: rho, and rho times what the rounding of the operand left out
      load32(vs + V_RHO * CHUNK, f);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        y[2 * i] = f[2 * i] * (y[2 * i] - __uint_as_float(pk[i] << 16));
        y[2 * i + 1] = f[2 * i + 1] * (y[2 * i + 1] - __uint_as_float(pk[i] & 0xffff0000u));
      }
      WAIT(VN_DONE, it & 1);
      tc_fence_after();
      tmem_ld32(tmem + lane_sel + TM_VN + t0, x);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; ++i)
        pk[i] = pack_bf16(f[2 * i] * x[2 * i] + y[2 * i], f[2 * i + 1] * x[2 * i + 1] + y[2 * i + 1]);
      tmem_st16(tmem + lane_sel + TM_VRB + (t0 >> 1), pk);
      tmem_st_wait();
      tc_fence_before();
      ARRIVE(VB_READY);
    }
  } break;
  case 2: if constexpr (!STATE) {
    // =============================== V group ===============================
    const int v = tid - 256;  // tensor-memory lane: value index for Vn^T, key index for w^T
    // w^T of chunk `it` (tensor memory, [k][tok]) -> bf16 operand tile, row k = 64 tokens
    auto convert_w = [&](int it) {
      WAIT(W_DONE, it & 1);
      tc_fence_after();
      unsigned char* row = smem + OFF_W + v * 128;
#pragma unroll 1
      for (int h = 0; h < 8; h += 4) {  // 32 tokens, four 16-byte pieces per round
        float x[32];
        tmem_ld32(tmem + lane_sel + TM_W + 8 * h, x);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 4; ++c)
          *reinterpret_cast<uint4*>(row + (((h + c) ^ (v & 7)) << 4)) =
              make_uint4(pack_bf16(x[8 * c], x[8 * c + 1]), pack_bf16(x[8 * c + 2], x[8 * c + 3]),
                         pack_bf16(x[8 * c + 4], x[8 * c + 5]), pack_bf16(x[8 * c + 6], x[8 * c + 7]));
      }
      tc_fence_before();
      fence_proxy_async();
      ARRIVE(W_READY);
    };
#pragma unroll 1
    for (int it = -1; it < n_it; ++it, fill()) {  // it = -1: only w^T of the first iteration
     if (it >= 0) {
      const int c = it - lead;
      if (v == 0) FQLA_TRACE(1, 0);
      WAIT(FULL0 + (it & 1), (it >> 1) & 1);
      WAIT(VN_DONE, it & 1);
      // the output product that reads Vn^T of the chunk before is issued by the other thread
      if (!NO_O && c >= 1) WAIT(O_DONE, (c - 1) & 1);
      tc_fence_after();
      if (v == 0) FQLA_TRACE(1, 1);
      const float* rho = vec + (it & 3) * VEC_SLOT_FLOATS + V_RHO * CHUNK;
      // on the chain: Vn^T as the two bf16 operands (rho-scaled for the state update, plain for
      // the output product), 32 tokens = 16 packed columns at a time
#pragma unroll 1
      for (int t0 = 0; t0 < CHUNK; t0 += 32) {
        float x[32];
        tmem_ld32(tmem + lane_sel + TM_UV + t0, x);
        float4 r[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) r[i] = *reinterpret_cast<const float4*>(rho + t0 + 4 * i);
        tmem_ld_wait();
        uint32_t pr[16], pn[16];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          pr[2 * i] = pack_bf16(r[i].x * x[4 * i], r[i].y * x[4 * i + 1]);
          pr[2 * i + 1] = pack_bf16(r[i].z * x[4 * i + 2], r[i].w * x[4 * i + 3]);
          pn[2 * i] = pack_bf16(x[4 * i], x[4 * i + 1]);
          pn[2 * i + 1] = pack_bf16(x[4 * i + 2], x[4 * i + 3]);
        }
        tmem_st16(tmem + lane_sel + TM_VRB + (t0 >> 1), pr);
        tmem_st16(tmem + lane_sel + TM_VNB + (t0 >> 1), pn);
      }
      tmem_st_wait();
      tc_fence_before();
      ARRIVE(VB_READY);
      if (v == 0) FQLA_TRACE(1, 2);
      if constexpr (EXTRA) {
        // off the chain: v_new as an output, from the operand copy (the store of the chunk before has
        // read the tile: the thread that issued this chunk's Vn^T waited for it)
        if (p.vnew && c >= 0) {
          unsigned char* row = smem + OFF_VNT + v * 128;
          float x[32];
          tmem_ld32(tmem + lane_sel + TM_VNB, x);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 8; ++q)
            *reinterpret_cast<float4*>(row + ((q ^ (v & 7)) << 4)) =
                make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
          if (p.tiled) {
            fence_proxy_async();
            ARRIVE(VN_READY);
          } else {  // row-major [row][v]: column v, from this thread's own row
            const long long row0 = sp.bos + (long long)c * CHUNK;
            const int valid = tries > 0 ? min(CHUNK, sp.len - c * CHUNK) : 0;
            bf16* dst = p.vnew + (row0 * p.Hv + hv) * D + v;
#pragma unroll 1
            for (int j = 0; j < valid; ++j)
              dst[(long long)j * p.Hv * D] = *reinterpret_cast<const bf16*>(smem + OFF_VNT + sw128_offset(v, j));
          }
        }
      }
     }
      if (it + 1 < n_it) convert_w(it + 1);
      if (v == 0) FQLA_TRACE(1, 3);
    }
  } break;
  case 3: if constexpr (!NO_O) {
    // =============================== O group ===============================
    const int wq = warp & 3;
    const int v = tid - 384;
    // c counts the chunks of the sequence itself; the lead-in chunks (iterations j < lead) have no
    // output products, so the barriers of this group's products are phased by c, while stages and
    // vector slots follow the iteration j = c + lead
    // The output tile leaves through shared memory and one TMA store per 64-column box: a
    // read-out thread owns one value index of all 64 tokens, and global stores of that shape (two
    // 64-byte pieces per warp instruction) are an order of magnitude slower than the rest of the
    // chunk.  Only a sequence's ragged last chunk is written with plain stores, row by row.
    auto epilogue = [&](int c) {
      const int it = c + lead;  // (trace window index)
      const float* sg = vec + (it & 3) * VEC_SLOT_FLOATS + V_SGAM * CHUNK;
      const long long row0 = sp.bos + (long long)c * CHUNK;
      const int valid = min(CHUNK, sp.len - c * CHUNK);
      // The accumulators hold o transposed ([value index][token]).  Read with the 16-lane shape, a
      // lane gets mma-style fragments: rows l/4 and l/4 + 8 of a 16-row half, token pairs
      // 8 i + 2 (l%4), +1.  stmatrix with .trans writes each 8 x 8 fragment block transposed, i.e.
      // as eight 16-byte pieces "8 value indices of one token": the tile comes out token-major
      // without a single shuffle.
      // Rounds of 16 lanes (value indices) x 32 tokens.
      const int l4 = lane & 3, mtx = lane >> 3, r8 = lane & 7;
#pragma unroll 1
      for (int h = 0; h < 4; ++h) {
        const int t0 = 32 * (h & 1);
        const uint32_t at = tmem + ((uint32_t)(wq * 32 + 8 * (h & 2)) << 16) + (uint32_t)t0;
        float a[16], b[16];
        tmem_ld_16x32(at + TM_O1, a);
        tmem_ld_16x32(at + TM_O2, b);
        float2 s2[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) s2[i] = *reinterpret_cast<const float2*>(sg + t0 + 8 * i + 2 * l4);
        tmem_ld_wait();
        if (h == 3) {  // all tensor-memory reads of this chunk's output are done
          tc_fence_before();
          ARRIVE(O_FREE);
        }
        // this lane supplies the address of row r8 of matrix mtx of every store: matrices 0, 1 are
        // the two 8-row blocks of token block i, matrices 2, 3 those of token block i + 1
        const int pv = (wq & 1) * 4 + (h & 2);  // 16-byte piece of rows 0-7 inside the box
        const uint32_t base = s32(smem + OFF_O + (wq >> 1) * 8192) +
                              (uint32_t)((t0 + 8 * (mtx >> 1) + r8) * 128 + (((pv + (mtx & 1)) ^ r8) << 4));
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
          uint32_t w[4];
#pragma unroll
          for (int z = 0; z < 2; ++z) {
            const float* aa = a + 4 * (i + z);
            const float* bb = b + 4 * (i + z);
            w[2 * z] = pack_out<O_F16>(s2[i + z].x * aa[0] + bb[0], s2[i + z].y * aa[1] + bb[1]);
            w[2 * z + 1] = pack_out<O_F16>(s2[i + z].x * aa[2] + bb[2], s2[i + z].y * aa[3] + bb[3]);
          }
          stmatrix_x4_trans(base + (uint32_t)(i * 1024), w[0], w[1], w[2], w[3]);
        }
      }
      fence_proxy_async();
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (valid == CHUNK) {
        if (wq == 0 && elect_one()) {
          tma_store_2d(&map_o, hv * D, (int)row0, smem + OFF_O);
          tma_store_2d(&map_o, hv * D + 64, (int)row0, smem + OFF_O + 8192);
          tma_store_commit();
        }
      } else {
        // 16 pieces of 16 bytes per row; piece pc of row r sits at pc ^ (r & 7) inside its box
#pragma unroll 1
        for (int i = v; i < valid * 16; i += 128) {
          const int r = i >> 4, pc = i & 15;
          const uint4 w = *reinterpret_cast<const uint4*>(smem + OFF_O + (pc >> 3) * 8192 + r * 128 +
                                                          (((pc & 7) ^ (r & 7)) << 4));
          *reinterpret_cast<uint4*>(p.o + ((row0 + r) * p.Hv + hv) * D + pc * 8) = w;
        }
      }
    };
#pragma unroll 1
    for (int c = 0; c < n_it - lead; ++c, fill()) {
      if (v == 0) { const int it = c + lead; FQLA_TRACE(2, 0); }
      WAIT(O_DONE, c & 1);
      if (wq == 0 && elect_one()) tma_store_wait_read();  // the store of the chunk before has read the tile
      // nothing is stored of what is not complete, and the four warps, which meet again behind this, go as one
      if (!bar_all<1, 128>(tries > 0)) break;
      tc_fence_after();
      if (v == 0) { const int it = c + lead; FQLA_TRACE(2, 1); }
      epilogue(c);
      if (v == 0) { const int it = c + lead; FQLA_TRACE(2, 2); }
    }
    if (wq == 0 && elect_one()) tma_store_wait_all();
    // rows of o past the end of the last packed sequence come out zero
    if (p.o && p.lay.cu.ptr && n == p.N - 1) {
      const long long end = sp.bos + sp.len;
#pragma unroll 1
      for (long long i = tid - 384; i < (p.T_rows - end) * 16; i += 128)
        *reinterpret_cast<uint4*>(p.o + ((end + (i >> 4)) * p.Hv + hv) * D + (i & 15) * 8) =
            make_uint4(0, 0, 0, 0);
    }
  } break;
  case 4: if constexpr (!STATE) {
    // =============================== prep group ===============================
    // A' = A diag(beta), A'' = A diag(beta gamma) of the next chunk, then Pg of this one.
    const int v = tid - 32 * PREP, wq = warp & 3;
    // A', A'': thread t owns the 8 columns 8 (t%8) .. of the rows t/8 + 16 i: its 16 scale factors stay in
    // registers, and the eight threads of a row touch the eight 16-byte pieces of that row (one 128-byte line
    // per access, conflict-free).
    const int c8 = v & 7, r0 = v >> 3;
    // Pg: P is an M = 64 accumulator read with the 16-lane shape: lane l of warp q owns rows
    // 16q + l/4 and 16q + l/4 + 8, and in every group of 8 columns the pair 2*(l%4), +1.
    const int row_a = 16 * wq + (lane >> 2), row_b = row_a + 8, cp = 2 * (lane & 3);
    const uint32_t lanes_p = (uint32_t)(wq * 32) << 16;  // lanes 0-15 of the quarter
    const float log2_scale = log2f(p.scale);
#pragma unroll 1
    for (int it = -1; it < n_it; ++it, fill()) {  // it = -1: only A of the first iteration
      if (v == 0) FQLA_TRACE(2, 3);
      if (it + 1 < n_it) {
        const int j = it + 1, sj = j & 1;
        WAIT(FULLA0 + sj, (j >> 1) & 1);
        if (j > 0) WAIT(U_DONE, (j - 1) & 1);  // u of the chunk before, and w ahead of it, are done
        const float* vs = vec + (j & 3) * VEC_SLOT_FLOATS + 8 * c8;
        const float4 b0 = *reinterpret_cast<const float4*>(vs + V_BETA * CHUNK);
        const float4 b1 = *reinterpret_cast<const float4*>(vs + V_BETA * CHUNK + 4);
        const float4 g0 = *reinterpret_cast<const float4*>(vs + V_BG * CHUNK);
        const float4 g1 = *reinterpret_cast<const float4*>(vs + V_BG * CHUNK + 4);
        // physical piece: rows r0 + 16 i all have (row & 7) == r0 & 7
        unsigned char* dst = smem + OFF_AP + r0 * 128 + (c8 ^ (r0 & 7)) * 16;
        const unsigned char* src = dst + (OFF_STAGE + 2 * TILE_QK + TILE_V - OFF_AP) + sj * STAGE_BYTES;
        uint4 next = *reinterpret_cast<const uint4*>(src);
#pragma unroll 1
        for (int i = 0; i < 4 * 2048; i += 2048) {
          const uint4 a = next;
          next = *reinterpret_cast<const uint4*>(src + ((i + 2048) & 0x1fff));
          *reinterpret_cast<uint4*>(dst + i) =
              make_uint4(scale_bf16x2(a.x, b0.x, b0.y), scale_bf16x2(a.y, b0.z, b0.w),
                         scale_bf16x2(a.z, b1.x, b1.y), scale_bf16x2(a.w, b1.z, b1.w));
          *reinterpret_cast<uint4*>(dst + (OFF_APP - OFF_AP) + i) =
              make_uint4(scale_bf16x2(a.x, g0.x, g0.y), scale_bf16x2(a.y, g0.z, g0.w),
                         scale_bf16x2(a.z, g1.x, g1.y), scale_bf16x2(a.w, g1.z, g1.w));
        }
        fence_proxy_async();
        ARRIVE(AP_READY);
        ARRIVE(EMPTYA0 + sj);  // the A tile of this stage is no longer read here
      }
      if (v == 0) FQLA_TRACE(2, 4);
      if (!NO_O && it >= 0 && it >= lead) {
        const float* vs = vec + (it & 3) * VEC_SLOT_FLOATS + V_G * CHUNK;
        WAIT(P_DONE, (it - lead) & 1);
        if (it > lead) WAIT(O_DONE, (it - lead - 1) & 1);  // the tile of the chunk before has been read
        tc_fence_after();
        if (v == 0) FQLA_TRACE(2, 5);
        // Pg = s P exp(g_row - g_col) = P exp2((g_row - g_col) log2e + log2 s), col <= row; 16 columns a
        // round (column groups entirely above this warp's rows stay zero, written once at start)
        const float ga2 = vs[row_a] * 1.4426950408889634f + log2_scale;
        const float gb2 = vs[row_b] * 1.4426950408889634f + log2_scale;
        unsigned char* pa = smem + OFF_P + row_a * 128 + cp * 2;  // rows b: 8 rows below, the same swizzle
        float x[32];
        tmem_ld_16x64(tmem + lanes_p + TM_P, x);
        tmem_ld_wait();
        tc_fence_before();
        ARRIVE(P_FREE);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (i > 2 * wq + 1) continue;
          const int col = 8 * i + cp;
          const float2 gc = *reinterpret_cast<const float2*>(vs + col);
          const float e0 = -1.4426950408889634f * gc.x, e1 = -1.4426950408889634f * gc.y;
          const float a0 = col <= row_a ? x[4 * i] * exp2f(e0 + ga2) : 0.f;
          const float a1 = col + 1 <= row_a ? x[4 * i + 1] * exp2f(e1 + ga2) : 0.f;
          const float b0 = col <= row_b ? x[4 * i + 2] * exp2f(e0 + gb2) : 0.f;
          const float b1 = col + 1 <= row_b ? x[4 * i + 3] * exp2f(e1 + gb2) : 0.f;
          unsigned char* at = pa + ((i ^ (row_a & 7)) << 4);
          *reinterpret_cast<uint32_t*>(at) = pack_bf16(a0, a1);
          *reinterpret_cast<uint32_t*>(at + 1024) = pack_bf16(b0, b1);
        }
        fence_proxy_async();
        ARRIVE(P_READY);
        if (v == 96) FQLA_TRACE(2, 6);
      }
    }
  } break;
  default: if (warp != 2) {
    // =============================== MMA issuers ===============================
    // Three warps issue, each with its own waits and, from one elected lane, its own products and
    // tcgen05.commit (a commit covers the MMAs of the committing thread only).  The tensor pipe runs products
    // in the order in which they come, whoever issued them: what is off the chain is issued behind the
    // chain's product of the moment and runs while the read-out groups work on that one's result.
    constexpr uint32_t ID_P = idesc_bf16(64, 64, 0, 0);
    constexpr uint32_t ID_UT = idesc_bf16(128, 64, 1, 0);            // A = V / K tile, MN-major
    constexpr uint32_t ID_VN = idesc_bf16(128, 64, 0, 1) | (1u << 13);  // A negated; B = w^T tile
    constexpr uint32_t ID_OT = idesc_bf16(128, 64, 0, 0);            // A from tensor memory
    constexpr uint32_t ID_S = idesc_bf16(128, 128, 0, 1);
    constexpr uint32_t STAGE_LO = STAGE_BYTES >> 4;
    const bool idle = STATE ? warp != 0 : NO_O && warp == 1;
    if constexpr (STATE) {
      const uint32_t k0_lo = desc_lo_kmajor(smem + OFF_STAGE + TILE_QK);
      const uint32_t kmn0_lo = desc_lo_mnmajor(smem + OFF_STAGE + TILE_QK, 8192);
      const uint32_t a0_lo = desc_lo_kmajor(smem + OFF_STAGE + 2 * TILE_QK + TILE_V);
#pragma unroll 1
      for (int it = 0; it < n_it && warp == 0; ++it, fill()) {
        const int s = it & 1, ph = (it >> 1) & 1;
        const uint32_t so = s ? STAGE_LO : 0u;
        if (!(WAITU(FULL0 + s, ph) && WAITU(S_COPY, it & 1))) break;
        tc_fence_after();
        if (elect_one()) {
          // U^T = S^T K^T   (A = packed S^T; B = K tile, K-major)
          umma_ts_group_kmajor_b<8>(tmem + TM_U, tmem + TM_SB, k0_lo + so, ID_OT);
          umma_commit(&bars[U_DONE]);
        }
        if (!(WAITU(FULLA0 + s, ph) && WAITU(WB_READY, it & 1))) break;
        tc_fence_after();
        if (elect_one()) {
          // Vn^T = W^T A^T   (A = packed W^T; B = A tile, K-major)
          umma_ts_group<4, 8, 2, false>(tmem + TM_VN, tmem + TM_WB, a0_lo + so, ID_OT);
          umma_commit(&bars[VN_DONE]);
          umma_commit(&bars[EMPTYA0 + s]);
        }
        if (!(WAITU(VB_READY, it & 1) && WAITU(S_DEC, it & 1))) break;
        tc_fence_after();
        if (elect_one()) {
          // S^T += (rho Vn)^T K
          umma_ts_group<4, 8, 128, true>(tmem + TM_S, tmem + TM_VRB, kmn0_lo + so, ID_S);
          umma_commit(&bars[S_DONE]);
          umma_commit(&bars[EMPTY0 + s]);
        }
      }
    } else if (warp == 0) {
      // low descriptor words of every operand tile (see umma_lo); steps are 32-bit adds
      const uint32_t wmn_lo = desc_lo_mnmajor(smem + OFF_W, 16384);
      const uint32_t kmn0_lo = desc_lo_mnmajor(smem + OFF_STAGE + TILE_QK, 8192);
#pragma unroll 1
      for (int it = 0; it < n_it; ++it, fill()) {
        const int s = it & 1, c = it - lead;  // c < 0: lead-in chunk
        const uint32_t so = s ? STAGE_LO : 0u;
        if (lane == 0) FQLA_TRACE(3, 0);
        if (lane == 0 && it < 126) FQLA_CHUNK_CLOCK(it);
        if (!(WAITU(U_DONE, it & 1) && WAITU(W_READY, it & 1) && WAITU(S_COPY, it & 1))) break;
        tc_fence_after();
        if (lane == 0) FQLA_TRACE(3, 1);
        if (elect_one()) {
          // Vn^T = u^T - S^T w^T   (accumulates onto u^T; A = packed S^T in tensor memory)
          umma_ts_group<8, 8, 128, true>(tmem + TM_UV, tmem + TM_SB, wmn_lo, ID_VN);
          if constexpr (EXTRA) tma_store_wait_read();  // v_new^T of the chunk before has left its tile
          umma_commit(&bars[VN_DONE]);
        }
        if (lane == 0) FQLA_TRACE(3, 2);
        if constexpr (EXTRA) {
          if (tile_h && c >= 0) {  // the state entering this chunk, as an operand tile
            if (!WAITU(ST_READY, c & 1)) break;
            if (elect_one()) {
              const int y = (int)(((sp.chunk_base + c) * p.Hv + hv) * D);
              tma_store_2d(&map_h, 0, y, smem + OFF_ST);
              tma_store_2d(&map_h, 64, y, smem + OFF_ST + 16384);
              tma_store_commit();
            }
          }
        }
        if (lane == 0) FQLA_TRACE(3, 3);
        if (!(WAITU(VB_READY, it & 1) && WAITU(S_DEC, it & 1))) break;
        tc_fence_after();
        if (lane == 0) FQLA_TRACE(3, 4);
        if (elect_one()) {
          // S^T += (rho Vn)^T K      (A = packed rho Vn^T; B = K tile read MN-major)
          umma_ts_group<4, 8, 128, true>(tmem + TM_S, tmem + TM_VRB, kmn0_lo + so, ID_S);
          if constexpr (EXTRA) tma_store_wait_read();  // the S^T tile may be rewritten after this
          umma_commit(&bars[S_DONE]);
          umma_commit(&bars[EMPTY0 + s]);  // this thread's last product that reads the stage
        }
        if (lane == 0) FQLA_TRACE(3, 5);
        if constexpr (EXTRA) {
          if (tile_vn && c >= 0) {
            if (!WAITU(VN_READY, c & 1)) break;
            if (elect_one()) {  // the v_new^T tile is complete
              tma_store_2d(&map_vn, 0, (int)(((sp.chunk_base + c) * p.Hv + hv) * D), smem + OFF_VNT);
              tma_store_commit();
            }
          }
        }
        if (lane == 0) FQLA_TRACE(3, 8);
      }
      if constexpr (EXTRA) {
        if (elect_one()) tma_store_wait_all();
      }
    } else if (warp == 1) {
     if constexpr (!NO_O) {
      const uint32_t p_lo = desc_lo_kmajor(smem + OFF_P);
      const uint32_t q0_lo = desc_lo_kmajor(smem + OFF_STAGE);
      const uint32_t k0_lo = desc_lo_kmajor(smem + OFF_STAGE + TILE_QK);
      // A parity tells a phase from its neighbours only, so nothing may run two chunks ahead of this warp.  Its
      // products see to that; in a lead-in, where it has none, SB_FREE does, which the next state copy waits for,
      // and it waits only for VN_DONE, which that copy comes before (and which implies W_READY of the same chunk
      // and VB_READY of the one before).
#pragma unroll 1
      for (int it = 0; it < n_it; ++it, fill()) {
        const int s = it & 1, c = it - lead;
        const uint32_t so = s ? STAGE_LO : 0u;
        if (lane == 0) FQLA_TRACE(4, 0);
        // P = Q K^T, over w^T; the prep group turns it into Pg
        if (c >= 0) {
          if (!(WAITU(FULL0 + s, (it >> 1) & 1) && WAITU(W_READY, it & 1))) break;
          tc_fence_after();
          if (lane == 0) FQLA_TRACE(4, 1);
          if (elect_one()) {
            umma_loop<2, 2, 512, 2, 512>(tmem + TM_P, q0_lo + so, k0_lo + so, ID_P);
            umma_commit(&bars[P_DONE]);
          }
        }
        // O1^T = S^T Q^T   (A = packed S^T; B = q tile, K-major), behind Vn^T of the chain
        if (lane == 0) FQLA_TRACE(4, 2);
        if (!(WAITU(VN_DONE, it & 1) && (c <= 0 || WAITU(O_FREE, (c - 1) & 1)))) break;
        tc_fence_after();
        if (lane == 0) FQLA_TRACE(4, 3);
        if (elect_one()) {
          if (c >= 0) umma_ts_loop8<2, 512>(tmem + TM_O1, tmem + TM_SB, q0_lo + so, ID_OT);
          umma_commit(&bars[SB_FREE]);
          umma_commit(&bars[EMPTY0 + s]);  // this thread's products that read the stage
        }
        if (lane == 0) FQLA_TRACE(4, 4);
        // O2^T = Vn^T Pg^T   (A = packed Vn^T; B = Pg, K-major)
        if (c >= 0) {
          if (!(WAITU(VB_READY, it & 1) && WAITU(P_READY, c & 1))) break;
          tc_fence_after();
          if (lane == 0) FQLA_TRACE(4, 5);
          if (elect_one()) {
            umma_ts_group<4, 8, 2, false>(tmem + TM_O2, tmem + TM_VNB, p_lo, ID_OT);
            umma_commit(&bars[O_DONE]);
          }
        }
        if (lane == 0) FQLA_TRACE(4, 6);
      }
     }
    } else {
      // w^T of iteration it + 1, behind Vn^T of iteration `it`, which stands on the chain (and for which w^T of
      // `it` has been made an operand), and behind Pg, made of P in the same columns.
      const uint32_t ap_lo = desc_lo_kmajor(smem + OFF_AP), app_lo = desc_lo_kmajor(smem + OFF_APP);
      const uint32_t vmn0_lo = desc_lo_mnmajor(smem + OFF_STAGE + 2 * TILE_QK, 8192);
      const uint32_t kmn0_lo = desc_lo_mnmajor(smem + OFF_STAGE + TILE_QK, 8192);
#pragma unroll 1
      for (int it = -1; it + 1 < n_it; ++it, fill()) {
        const int s = (it + 1) & 1;
        if (!(WAITU(FULL0 + s, ((it + 1) >> 1) & 1) && WAITU(AP_READY, (it + 1) & 1))) break;
        if (it >= 0 && !WAITU(VN_DONE, it & 1)) break;
        if (!NO_O && it >= 0 && it >= lead && !WAITU(P_FREE, (it - lead) & 1)) break;
        tc_fence_after();
        if (lane == 0) FQLA_TRACE(5, 0);
        if (elect_one()) {
          umma_group<4, 128, 0, 2, 0, false>(tmem + TM_W, kmn0_lo + (s ? STAGE_LO : 0u), app_lo, ID_UT);
          umma_commit(&bars[W_DONE]);
        }
        if (lane == 0) FQLA_TRACE(5, 1);
        // u^T over Vn^T, which has been read, behind the state update
        if (it >= 0 && !WAITU(S_DONE, it & 1)) break;
        tc_fence_after();
        if (lane == 0) FQLA_TRACE(5, 2);
        if (elect_one()) {
          umma_group<4, 128, 0, 2, 0, false>(tmem + TM_UV, vmn0_lo + (s ? STAGE_LO : 0u), ap_lo, ID_UT);
          umma_commit(&bars[U_DONE]);
          umma_commit(&bars[EMPTY0 + s]);
        }
        if (lane == 0) FQLA_TRACE(5, 3);
      }
    }
    // no product is under way when the block goes, whoever gave up what
    if (!idle && elect_one()) umma_commit(&bars[SETTLED]);
    if (warp == 0) settle(SETTLED, 0);
  } else {
    // =============================== producer ===============================
    // zero the rows past the sequence end in n 8 KB blocks of 64 rows (they belong to the next
    // sequence), then hand the tile on
    auto zero_rows = [&](unsigned char* base, int n, int valid, uint64_t* full) {
#pragma unroll 1
      for (int i = lane; i < n * 512; i += 32)
        if (((i >> 3) & 63) >= valid) *reinterpret_cast<uint4*>(base + i * 16) = make_uint4(0, 0, 0, 0);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0 && tries > 0) mbar_arrive(full);
    };
    // Iteration `it`: q, k, v of chunk it; vectors and A tile of chunk it + 1, a whole chunk before
    // its q, k, v (whose stage is still in use, but the prep warps can start on A early); the gates
    // of chunk it + 2 into registers.  (Slot (it + 1) % 4 of the vectors was last read for chunk
    // it - 3, which the wait on the stage of chunk it - 2 has seen finished.)
    float g_r[2] = {0.f, 0.f}, b_r[2] = {0.f, 0.f}, gl_r = 0.f;
    // (A whole first chunk's q, k, v go out at once, ahead of its gates: it = -2.  The arrival on their barrier,
    // which stands for the vectors too, follows in its place.  100 tokens x 8 heads 13.1 -> 12.3 us.)
    int loads = 0, a_loads = 0;  // q, k, v and A tiles that have been asked for
    const bool early = n_it > 0 && (lead > 0 || sp.len + lead * CHUNK >= CHUNK);
    auto load = [&](int it) {
      const int s = it & 1, c = it - lead;
      const int y = (int)sp.bos + c * CHUNK;
      const int valid = c < 0 ? CHUNK : min(CHUNK, sp.len - c * CHUNK);
      const bool with_q = !NO_O && c >= 0, partial = valid < CHUNK;
      if (it >= 2) WAIT(EMPTY0 + s, ((it >> 1) - 1) & 1);
      unsigned char* st = smem + OFF_STAGE + s * STAGE_BYTES;
      uint64_t* bar = &bars[partial ? PRIV : FULL0 + s];
      if (issuing()) {
        mbar_expect_tx(bar, STAGE_BYTES - TILE_A - (with_q ? 0 : TILE_QK) - (m_pass ? TILE_V : 0));
        if (it > 0 || !early) mbar_arrive(bar);
        tma_load_2d(st + TILE_QK, &map_k, hq * D, y, bar);
        tma_load_2d(st + TILE_QK + 8192, &map_k, hq * D + 64, y, bar);
        if (!m_pass) {
          tma_load_2d(st + 2 * TILE_QK, &map_v, hv * D, y, bar);
          tma_load_2d(st + 2 * TILE_QK + 8192, &map_v, hv * D + 64, y, bar);
        }
        if (with_q) {
          tma_load_2d(st, &map_q, hq * D, y, bar);
          tma_load_2d(st + 8192, &map_q, hq * D + 64, y, bar);
        }
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
        const int sj = j & 1, c = j - lead;
        const int valid = c < 0 ? CHUNK : min(CHUNK, sp.len - c * CHUNK);
        const bool partial = valid < CHUNK;
        // the stage's A buffer is free once the prep warps have read it
        if (j >= 2) WAIT(EMPTYA0 + sj, ((j >> 1) - 1) & 1);
        float* vs = vec + (j & 3) * VEC_SLOT_FLOATS + lane;
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          const float gam = fast_exp(g_r[z]);
          vs[V_G * CHUNK + 32 * z] = g_r[z];
          vs[V_BETA * CHUNK + 32 * z] = b_r[z];
          vs[V_BG * CHUNK + 32 * z] = STATE ? -b_r[z] * gam : b_r[z] * gam;
          vs[V_RHO * CHUNK + 32 * z] = fast_exp(gl_r - g_r[z]);
          vs[V_SGAM * CHUNK + 32 * z] = p.scale * gam;
        }
        vs[V_GL * CHUNK] = fast_exp(gl_r);
        __syncwarp();
        unsigned char* dst = smem + OFF_STAGE + sj * STAGE_BYTES + 2 * TILE_QK + TILE_V;
        uint64_t* bar = &bars[partial ? PRIVA : FULLA0 + sj];
        if (issuing()) {
          mbar_arrive_expect_tx(bar, TILE_A);
          tma_load_2d(dst, &map_a, hv * CHUNK, (int)sp.bos + c * CHUNK, bar);
        }
        a_loads = tries > 0 ? j + 1 : a_loads;
        if (partial) {
          // only the last chunk of a sequence can be partial: the private barrier is used once
          WAIT(PRIVA, 0);
          zero_rows(dst, 1, valid, &bars[FULLA0 + sj]);
        }
      }
      if (it + 2 < n_it) {
        // (lead-in chunks, c < 0, are whole chunks of the rows before the sequence)
        const int c = it + 2 - lead, last = (c < 0 ? CHUNK : min(CHUNK, sp.len - c * CHUNK)) - 1;
        const long long at = (sp.bos + (long long)c * CHUNK) * p.Hv + hv;
        gl_r = p.g[at + last * p.Hv];
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          const int r = lane + 32 * z;
          const long long i = at + min(r, last) * p.Hv;
          g_r[z] = p.g[i];
          b_r[z] = load_beta(p.beta, p.beta_is_f32, i);
          if (r > last) b_r[z] = 0.f;
        }
      }
    }
    // nor a load
#pragma unroll 1
    for (int i = 1; i <= 2; ++i) {
      if (loads >= i) settle(FULL0 + ((loads - i) & 1), ((loads - i) >> 1) & 1);
      if (a_loads >= i) settle(FULLA0 + ((a_loads - i) & 1), ((a_loads - i) >> 1) & 1);
    }
  }

  }  // switch

  // ---- teardown: everybody meets, then the allocating warp frees tensor memory
  if (tries <= 0) *abort_flag = 1;
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
  if (tid == 0 && *abort_flag) atomicCAS(&g_device_status, 0, 1);
  if (tid == 0) FQLA_CHUNK_CLOCK(127);
#ifdef FQLA_DIAGNOSTICS
  if (tid == 0 && blockIdx.x < 1024) {
    unsigned smid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    g_cta_cycles[2 * blockIdx.x] = smid;
    g_cta_cycles[2 * blockIdx.x + 1] = clock64() - g_fwd_chunk_clock_entry;
  }
#endif
}

// ---- host side --------------------------------------------------------------------------------
// 2-D bf16 tensor [rows][cols] (row pitch = cols), box = 64 columns x box_rows rows, 128-byte
// swizzle; recently used maps are served from a small host-side table (bwd_main_tc.cu).
int make_tile_map(CUtensorMap* m, const void* ptr, long long rows, long long cols, int box_rows);

static int make_map(CUtensorMap* m, const void* ptr, long long rows, long long cols) {
  return make_tile_map(m, ptr, rows, cols, 64);
}

int launch_fwd_tc(const fqla_fwd_args& a, int N, SeqLayout lay, cudaStream_t st) {
  using namespace fwdtc;
  CUtensorMap mq, mk, mv, ma, mh, mvn, mo;
  const long long T_rows = (long long)a.B * a.T;
  int rc;
  // without q (recomputation of h and v_new for the backward pass) the state-only variant runs;
  // its q map is never used and only has to be a valid map
  if ((rc = make_map(&mq, a.q ? a.q : a.k, T_rows, (long long)a.Hq * D))) return rc;
  if ((rc = make_map(&mk, a.k, T_rows, (long long)a.Hq * D))) return rc;
  if ((rc = make_map(&mv, a.v, T_rows, (long long)a.Hv * D))) return rc;
  if ((rc = make_map(&ma, a.A, T_rows, (long long)a.Hv * CHUNK))) return rc;
  mh = mq;
  mvn = mq;
  mo = mq;
  if (a.o && (rc = make_map(&mo, a.o, T_rows, (long long)a.Hv * D))) return rc;
  if (a.operand_tiles) {
    // an upper bound of the chunk count: the maps only have to cover what the kernel stores
    const long long max_chunks = (T_rows + CHUNK - 1) / CHUNK + N;
    if (a.h && (rc = make_tile_map(&mh, a.h, max_chunks * a.Hv * D, D, 128))) return rc;
    if (a.vnew && (rc = make_tile_map(&mvn, a.vnew, max_chunks * a.Hv * D, CHUNK, 128))) return rc;
  }
  FwdTcParams p;
  p.g = a.g_cum; p.beta = a.beta; p.beta_is_f32 = a.beta_is_f32;
  p.h0 = a.h0; p.seg_h0 = a.seg_h0; p.h0_row = a.h0_row; p.ht_row = a.ht_row;
  p.v_first = a.state_v_first; p.ht = a.ht;
  p.o = (bf16*)a.o; p.h = (bf16*)a.h; p.vnew = (bf16*)a.vnew;
  p.N = N; p.Hq = a.Hq; p.Hv = a.Hv; p.T_rows = T_rows; p.scale = a.scale; p.lay = lay;
  p.tiled = a.operand_tiles; p.lead = a.lead_chunks; p.run_mask = a.run_mask;
  p.run_value = a.run_value; p.order = a.seq_order;
  p.M = a.M; p.warm = a.warm_chunks; p.m_mask = a.m_mask; p.m_first = INT_MAX;
  int blocks = N * a.Hv;
  const bool no_o = !a.q && !a.o;
  auto launch = [&](auto kernel, int smem_bytes, std::atomic<unsigned long long>& done) {
    int err = configure_smem((const void*)kernel, smem_bytes, done);
    if (err != 0) return err;
    return launch_pdl(kernel, dim3((unsigned)blocks), dim3(threads(no_o)), (size_t)smem_bytes, st, p, mq, mk,
                      mv, ma, mh, mvn, mo);
  };
  static std::atomic<unsigned long long> done[6];
  if (!a.q && !a.o && !a.h && !a.vnew) {  // end states and transition matrices
    if (a.M) {
      p.m_first = a.ht ? blocks : 0;
      blocks += p.m_first;
    }
    return launch(fwd_tc_kernel<false, true, false>, SMEM_BYTES, done[5]);
  }
  if (!a.q && !a.o)  // recomputation of h, v_new
    return launch(fwd_tc_kernel<true, true, false>, SMEM_BYTES_EXTRA, done[0]);
  if (a.h || a.vnew)
    return a.o_is_f16 ? launch(fwd_tc_kernel<true, false, true>, SMEM_BYTES_EXTRA, done[1])
                      : launch(fwd_tc_kernel<true, false, false>, SMEM_BYTES_EXTRA, done[2]);
  return a.o_is_f16 ? launch(fwd_tc_kernel<false, false, true>, SMEM_BYTES, done[3])
                    : launch(fwd_tc_kernel<false, false, false>, SMEM_BYTES, done[4]);
}

}  // namespace fqla

#ifdef FQLA_DIAGNOSTICS
extern "C" int fqla_debug_fwd_trace(long long* out960) {
  return (int)cudaMemcpyFromSymbol(out960, fqla::g_fwd_trace, sizeof(long long) * 960);
}
extern "C" int fqla_debug_cta_cycles(long long* out2048, int trace_cta) {
  cudaMemcpyToSymbol(fqla::g_trace_cta, &trace_cta, sizeof(int));
  return (int)cudaMemcpyFromSymbol(out2048, fqla::g_cta_cycles, sizeof(long long) * 2048);
}
extern "C" int fqla_debug_fwd_chunk_clock(long long* out256) {
  return (int)cudaMemcpyFromSymbol(out256, fqla::g_fwd_chunk_clock, sizeof(long long) * 256);
}
#endif

namespace fqla {
// Self-test of the bounded-wait path: one thread waits on an mbarrier that nobody ever arrives
// at, with a budget of `tries` tries.  The wait gives up, the kernel sets the device status word exactly as a product kernel does, and returns.
__global__ void wait_timeout_selftest_kernel(int tries) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    mbar_wait(&bar, 0, tries);
    if (tries <= 0) atomicCAS(&g_device_status, 0, 1);
  }
}
}  // namespace fqla

extern "C" int fqla_selftest_wait_timeout(int tries, void* stream) {
  if (tries < 1 || tries > 100) return FQLA_ERR_INVALID_ARG;
  fqla::wait_timeout_selftest_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(tries);
  return (int)cudaGetLastError();
}

namespace fqla {
int bwd_main_tc_status(int* out, int reset);
int bwd_dh_tc_status(int* out, int reset);
int kkt_status(int* out, int reset);
}

extern "C" int fqla_device_status(int* out, int reset) {
  int v = 0, w = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, fqla::g_device_status, sizeof(int));
  if (e != cudaSuccess) return (int)e;
  int u = 0;
  int rc = fqla::bwd_main_tc_status(&w, reset);
  if (rc != 0) return rc;
  rc = fqla::bwd_dh_tc_status(&u, reset);
  if (rc != 0) return rc;
  int x = 0;
  rc = fqla::kkt_status(&x, reset);
  if (rc != 0) return rc;
  if (out) *out = v | w | u | x;
  if (reset && v != 0) {
    int z = 0;
    e = cudaMemcpyToSymbol(fqla::g_device_status, &z, sizeof(int));
  }
  return (int)e;
}
