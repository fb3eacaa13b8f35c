// Chunk-parallel preparation kernels of the gated-delta-rule path:
//   * chunk-local cumulative sum of the log gates (forward, and reversed for the gate gradient)
//   * A = (I + strict_lower(diag(beta) K K^T * exp(g_s - g_t)))^-1 per (chunk, value head)
//   * sum of per-value-head dq/dk over each grouped-value-attention group
// These replace the reference's ops/utils/cumsum.py:14-134, blackwell/kkt_solve.py:19-281 and
// ops/utils/group_reduce.py:12-57.
#include <cuda.h>

#include "common.cuh"
#include "fqla_internal.h"
#include "tc05.cuh"

namespace fqla {

int make_tile_map(CUtensorMap* m, const void* ptr, long long rows, long long cols, int box_rows);

// ------------------------------------------------------------------------------------------
// Chunk-local cumsum.  One CTA per chunk, one warp per head (looping), two rows per lane.
// HBM-bound: 8 bytes per (token, head).
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) cumsum_kernel(const float* __restrict__ g,
                                                     float* __restrict__ out, int H, int T_rows,
                                                     SeqLayout lay, IndexTable chunk_indices,
                                                     int N, int reverse) {
  pdl_wait();
  int seq, ci;
  if (lay.cu.ptr) {
    seq = (int)chunk_indices[2 * blockIdx.x];
    ci = (int)chunk_indices[2 * blockIdx.x + 1];
  } else {
    int per = (lay.T + CHUNK - 1) / CHUNK;
    seq = blockIdx.x / per;
    ci = blockIdx.x % per;
  }
  SeqSpan sp = lay.span(seq);
  long long row0 = sp.bos + (long long)ci * CHUNK;
  int valid = min(CHUNK, sp.len - ci * CHUNK);
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int h = warp; h < H; h += 4) {
    // lane owns rows 2*lane, 2*lane+1 (forward) or their mirror images (reverse)
    int r0 = 2 * lane, r1 = 2 * lane + 1;
    if (reverse) { r0 = valid - 1 - r0; r1 = valid - 1 - r1; }
    bool ok0 = reverse ? r0 >= 0 : r0 < valid;
    bool ok1 = reverse ? r1 >= 0 : r1 < valid;
    float a = ok0 ? g[(row0 + r0) * H + h] : 0.f;
    float b = ok1 ? g[(row0 + r1) * H + h] : 0.f;
    float pair = a + b, incl = pair;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      float t = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += t;
    }
    float excl = incl - pair;
    if (ok0) out[(row0 + r0) * H + h] = excl + a;
    if (ok1) out[(row0 + r1) * H + h] = excl + a + b;
  }
  // Rows past the last sequence's end (packed input shorter than the buffer) come out zero.
  if (lay.cu.ptr && seq == N - 1 && ci == sp.n_chunks - 1) {
    long long end = sp.bos + sp.len;
    for (long long i = end * H + threadIdx.x; i < (long long)T_rows * H; i += blockDim.x)
      out[i] = 0.f;
  }
}

// ------------------------------------------------------------------------------------------
// kkt + solve:  A = (I + L)^-1,  L = strict_lower(diag(beta) K K^T exp(g_s - g_t)),  one 64 x 64
// problem per (chunk, value head).
//
// ONE WARP solves one problem, in registers: there is no block-wide barrier on the way, and what
// hides the latencies is that a dozen warps with a problem each sit on an SM.  (The form before
// spread a problem over four warps and met eight block barriers per head with two of the four
// warps idle in the forward substitution: 79 us for 8192 problems against 31 us of HBM time.)
// A block is min(G, 4) warps sharing the K tile of one (chunk, q head); warp w takes the value
// heads w, w + 4, ... of the group.
//
// All 64 x 64 matrices are 16 x 16 blocks in the fragment layout of mma.sync (lane l = 4 g + t:
// element e of column half h is row g + 8 (e >> 1), column 8 h + 2 t + (e & 1)):
//   1. K K^T: the 10 blocks on and below the diagonal (bf16 products, fp32 sums).  A fragment of
//      rows loaded by ldmatrix serves as left operand and, for the transposed product, as right
//      operand, so each is loaded once.
//   2. L in place; the four 16 x 16 diagonal blocks go through shared memory.
//   3. D_i = (I + L_ii)^-1 by forward substitution in fp32, a lane = one column of two blocks.
//   4. The blocks of X = A below the diagonal, from  X_ij = -D_i (sum_{j<=k<i} L_ik X_kj),  are
//      computed TRANSPOSED (Y_ji = X_ij^T = -(sum_k Y_jk L_ik^T) D_i^T, Y_jj = D_j^T): then every left
//      operand is a result in fragment layout and every right operand L_ik^T, D_i^T is, read
//      element for element, the fragment of L_ik, D_i: no shuffle, no shared memory.  tf32 inputs
//      rounded to nearest, fp32 sums.  (tf32 k index t / t + 4 stands for column 2 t / 2 t + 1.)
//   5. bf16 tile through shared memory (stmatrix undoes the transposition), one TMA store.
// L is kept NEGATED throughout, so that every step is an addition.
//
// What bounds it: instruction issue and the latency of one warp's chain.  4 x 8192 tokens, 16 heads
// (8192 problems): the four-warp form 79 us; this one with scalar fp32, cvt.rna and per-thread
// copies 58 us (3090 instructions per problem); with packed fp32 pairs, TMA both ways and cvt.rn
// 46 us.
// ------------------------------------------------------------------------------------------
// set to 1 when a block of kkt_solve_kernel abandoned its bounded wait; read through
// fqla_device_status
__device__ int g_kkt_status = 0;

struct Block16 {  // 16 x 16 fp32 fragment
  float c[2][4];
};
// the same block as tf32 operand.  The conversion keeps infinities and NaN; adding half an ulp to the bits,
// which rounds as well and takes as long, makes -0 of the NaN of arithmetic (0x7fffffff).
// (cvt.rna, ties away instead of to even: 3 us of 46 more on the 8192 problems below.)
struct Op16 {
  uint32_t c[2][4];
};
__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rn.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ Op16 to_op(const Block16& b) {
  Op16 o;
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int e = 0; e < 4; ++e) o.c[h][e] = to_tf32(b.c[h][e]);
  return o;
}
// d (+)= a * b^T
template <bool ADD>
__device__ __forceinline__ void mma_abt(Block16& d, const Op16& a, const Op16& b) {
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (ADD || s > 0)
        asm volatile(
            "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
            "{%0,%1,%2,%3};"
            : "+f"(d.c[h][0]), "+f"(d.c[h][1]), "+f"(d.c[h][2]), "+f"(d.c[h][3])
            : "r"(a.c[s][0]), "r"(a.c[s][2]), "r"(a.c[s][1]), "r"(a.c[s][3]), "r"(b.c[s][2 * h]),
              "r"(b.c[s][2 * h + 1]));
      else
        asm volatile(
            "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
            "{%10,%10,%10,%10};"
            : "=f"(d.c[h][0]), "=f"(d.c[h][1]), "=f"(d.c[h][2]), "=f"(d.c[h][3])
            : "r"(a.c[s][0]), "r"(a.c[s][2]), "r"(a.c[s][1]), "r"(a.c[s][3]), "r"(b.c[s][2 * h]),
              "r"(b.c[s][2 * h + 1]), "f"(0.f));
    }
}
template <bool ADD>
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if (ADD)
    mma_bf16_16816(d, a, b0, b1);
  else
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// packed pairs of fp32 (one instruction for two lanes of arithmetic)
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
      "add.rn.ftz.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
      "mul.rn.ftz.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, w, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 w, {%6, %7};\n\t"
      "fma.rn.ftz.f32x2 z, x, y, w;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}

namespace kkt {
constexpr int MAX_WARPS = 4;
// The diagonal blocks 0 | 2 and 1 | 3 sit in shared memory as two matrices of pairs, so that one
// packed operation serves both blocks.  Row stride 52 words (16-byte rows, at most two-way bank
// conflicts for fragments and transposed fragments), pair stride 16 banks apart (the two
// half-warps read one pair each).
constexpr int LD_DIAG = 52, DIAG_STRIDE = 16 * LD_DIAG + 16;
constexpr int WARP_BYTES = CHUNK * CHUNK * 2;  // 8192: the output tile, and before it the diagonal blocks
constexpr int VEC_BYTES = 2 * CHUNK * 4;       // g, -beta of a warp's head
static_assert(2 * DIAG_STRIDE * 4 <= WARP_BYTES, "diagonal blocks fit the output tile");
template <int D>
constexpr int k_bytes() { return CHUNK * D * 2; }
// a single-warp block builds its output over the K tile, dead by then; + barrier, + alignment
template <int D>
constexpr int smem_bytes(int warps) {
  return k_bytes<D>() + warps * VEC_BYTES + (warps > 1 ? warps * WARP_BYTES : 0) + 16 + 1024;
}
}  // namespace kkt

template <int D>
__global__ void __launch_bounds__(32 * kkt::MAX_WARPS, 3) kkt_solve_kernel(
    const void* __restrict__ beta, int beta_is_f32, const float* __restrict__ g,
    float* __restrict__ g_cum_out, bf16* __restrict__ A, int Hq, int Hv, SeqLayout lay,
    IndexTable chunk_indices, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_a) {
  using namespace kkt;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, n_warps = blockDim.x >> 5;
  // per-warp scratch (1024-byte aligned): diagonal blocks (fp32), then the output tile (bf16)
  unsigned char* scratch = n_warps == 1 ? smem : smem + k_bytes<D>() + warp * WARP_BYTES;
  float* sD = reinterpret_cast<float*>(scratch);
  unsigned char* vecs = smem + k_bytes<D>() + (n_warps > 1 ? n_warps * WARP_BYTES : 0);
  float* sG = reinterpret_cast<float*>(vecs + warp * VEC_BYTES);  // g log2(e)
  float* sB = sG + CHUNK;                                         // -beta
  uint64_t* bar = reinterpret_cast<uint64_t*>(vecs + n_warps * VEC_BYTES);
  const int q8 = lane >> 2, t4 = lane & 3, l7 = lane & 7;  // fragment row, column pair; row mod 8
  const int hq = blockIdx.y, G = Hv / Hq;
  if (tid == 0) {
    tc::mbar_init(bar, 1);
    tc::fence_mbar_init();
  }
  pdl_wait();
  int seq, ci;
  if (lay.cu.ptr) {
    seq = (int)chunk_indices[2 * blockIdx.x];
    ci = (int)chunk_indices[2 * blockIdx.x + 1];
  } else {
    int per = (lay.T + CHUNK - 1) / CHUNK;
    seq = blockIdx.x / per;
    ci = blockIdx.x % per;
  }
  const SeqSpan sp = lay.span(seq);
  const long long row0 = sp.bos + (long long)ci * CHUNK;
  const int valid = min(CHUNK, sp.len - ci * CHUNK);
  if (n_warps > 1) __syncthreads();
  else __syncwarp();
  if (tid == 0) {
    // rows past the end of the sequence hold other rows of k: what they give is masked below
    tc::mbar_arrive_expect_tx(bar, k_bytes<D>());
#pragma unroll
    for (int b = 0; b < D / 64; ++b)
      tc::tma_load_2d(smem + b * 8192, &map_k, hq * D + 64 * b, (int)row0, bar);
  }
  int tries = tc::WAIT_TRIES;

#pragma unroll 1
  for (int gi = warp; gi < G; gi += n_warps) {
    const int hv = hq * G + gi;
    {  // gates and beta of the rows lane, lane + 32
      float x[2];
#pragma unroll
      for (int z = 0; z < 2; ++z) {
        const int r = lane + 32 * z;
        const long long i = (row0 + min(r, valid - 1)) * Hv + hv;
        x[z] = g[i];
        sB[r] = r < valid ? -load_beta(beta, beta_is_f32, i) : 0.f;
      }
      if (g_cum_out) {
        // g is the raw log gate: chunk-local inclusive prefix sum over the valid rows (rows past
        // the end repeat the last value, as the clamped read does)
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          if (lane + 32 * z >= valid) x[z] = 0.f;
#pragma unroll
          for (int d = 1; d < 32; d <<= 1) {
            const float y = __shfl_up_sync(0xffffffffu, x[z], d);
            if (lane >= d) x[z] += y;
          }
        }
        x[1] += __shfl_sync(0xffffffffu, x[0], 31);
#pragma unroll
        for (int z = 0; z < 2; ++z)
          if (lane + 32 * z < valid) g_cum_out[(row0 + lane + 32 * z) * Hv + hv] = x[z];
      }
      sG[lane] = x[0] * 1.4426950408889634f;
      sG[lane + 32] = x[1] * 1.4426950408889634f;
    }
    tc::mbar_wait(bar, 0, tries);
    if (!__all_sync(0xffffffffu, tries > 0)) break;
    __syncwarp();

    // ---- 1. K K^T, lower blocks (rb, cb), index rb (rb + 1) / 2 + cb
    Block16 L[10];
    {
      // 16-byte chunk c of row r of a 64-column block sits at chunk c ^ (r & 7)
      const uint32_t frag = smem_u32(smem) + (uint32_t)((l7 + ((lane >> 3) & 1) * 8) * 128);
      uint32_t col[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) col[i] = (uint32_t)(((2 * i + (lane >> 4)) ^ l7) << 4);
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        uint32_t a[4][4];
#pragma unroll
        for (int rb = 0; rb < 4; ++rb)
          ldmatrix_x4_addr(a[rb], frag + col[ks & 3] + (uint32_t)((ks >> 2) * 8192 + rb * 2048));
#pragma unroll
        for (int rb = 0; rb < 4; ++rb)
#pragma unroll
          for (int cb = 0; cb <= rb; ++cb) {
            Block16& d = L[rb * (rb + 1) / 2 + cb];
            if (ks == 0) {
              mma_bf16<false>(d.c[0], a[rb], a[cb][0], a[cb][2]);
              mma_bf16<false>(d.c[1], a[rb], a[cb][1], a[cb][3]);
            } else {
              mma_bf16<true>(d.c[0], a[rb], a[cb][0], a[cb][2]);
              mma_bf16<true>(d.c[1], a[rb], a[cb][1], a[cb][3]);
            }
          }
      }
    }
    // ---- 2. -L
    {
      float gr[8], br[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        gr[i] = sG[8 * i + q8];
        br[i] = sB[8 * i + q8];
      }
      const bool below0 = q8 > 2 * t4, below1 = q8 > 2 * t4 + 1;  // inside an 8 x 8 diagonal block
#pragma unroll
      for (int cb = 0; cb < 4; ++cb)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float2 gc = *reinterpret_cast<const float2*>(sG + 16 * cb + 8 * h + 2 * t4);
          const float2 ngc = make_float2(-gc.x, -gc.y);
#pragma unroll
          for (int rb = cb; rb < 4; ++rb)
#pragma unroll
            for (int z = 0; z < 2; ++z) {
              float* c = L[rb * (rb + 1) / 2 + cb].c[h] + 2 * z;
              if (rb == cb && h > z) {  // above the diagonal
                c[0] = c[1] = 0.f;
                continue;
              }
              const int ri = 2 * rb + z;
              const float2 d = add2(make_float2(gr[ri], gr[ri]), ngc);
              const float2 x = mul2(make_float2(c[0], c[1]), make_float2(br[ri], br[ri]));
              const float2 v = mul2(x, make_float2(exp2f(d.x), exp2f(d.y)));
              c[0] = v.x;
              c[1] = v.y;
              if (rb == cb && h == z) {
                if (!below0) c[0] = 0.f;
                if (!below1) c[1] = 0.f;
              }
            }
        }
      if (valid < CHUNK) {  // rows past the end: whatever their k holds, L is zero there
#pragma unroll
        for (int rb = 0; rb < 4; ++rb)
#pragma unroll
          for (int cb = 0; cb <= rb; ++cb)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (16 * rb + q8 + 8 * (e >> 1) >= valid) L[rb * (rb + 1) / 2 + cb].c[h][e] = 0.f;
      }
    }
    // ---- 3. inverses of the diagonal blocks
    // the K tile (single-warp blocks) and the output tile of the head before are dead
    if (lane == 0) tc::tma_store_wait_read();
    __syncwarp();
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          const float *lo = L[b * (b + 3) / 2].c[h] + 2 * z, *hi = L[(b + 2) * (b + 5) / 2].c[h] + 2 * z;
          *reinterpret_cast<float4*>(sD + b * DIAG_STRIDE + (q8 + 8 * z) * LD_DIAG + 16 * h + 4 * t4) =
              make_float4(lo[0], hi[0], lo[1], hi[1]);
        }
    __syncwarp();
    {
      const int c = lane & 15;  // column c of the blocks b, b + 2 with b = lane / 16
      float* d = sD + (lane >> 4) * DIAG_STRIDE;
      float2 x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float one = i == c ? 1.f : 0.f;
        float2 s = make_float2(one, one), s1 = make_float2(0.f, 0.f);  // two chains
#pragma unroll
        for (int j = 0; j < i; j += 2) {
          const float4 l = *reinterpret_cast<const float4*>(d + i * LD_DIAG + 2 * j);
          s = fma2(make_float2(l.x, l.y), x[j], s);
          if (j + 1 < i) s1 = fma2(make_float2(l.z, l.w), x[j + 1], s1);
        }
        x[i] = i > 1 ? add2(s, s1) : s;
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 16; ++i) *reinterpret_cast<float2*>(d + i * LD_DIAG + 2 * c) = x[i];
      __syncwarp();
    }
    // D_i and D_j^T as operands, D_i packed for the output
    Op16 Dop[4], Y[4][4];  // Y[j][i], j <= i: X_ij^T
    uint32_t dpack[4][4];
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          const float4 v = *reinterpret_cast<const float4*>(sD + b * DIAG_STRIDE + (q8 + 8 * z) * LD_DIAG + 16 * h + 4 * t4);
          dpack[b][2 * h + z] = pack_bf16(v.x, v.z);
          dpack[b + 2][2 * h + z] = pack_bf16(v.y, v.w);
          Dop[b].c[h][2 * z] = to_tf32(v.x);
          Dop[b].c[h][2 * z + 1] = to_tf32(v.z);
          Dop[b + 2].c[h][2 * z] = to_tf32(v.y);
          Dop[b + 2].c[h][2 * z + 1] = to_tf32(v.w);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float2 w = *reinterpret_cast<const float2*>(sD + b * DIAG_STRIDE + (8 * h + 2 * t4 + e) * LD_DIAG + 2 * (q8 + 8 * z));
            Y[b][b].c[h][2 * z + e] = to_tf32(w.x);
            Y[b + 2][b + 2].c[h][2 * z + e] = to_tf32(w.y);
          }
        }
    __syncwarp();  // the diagonal blocks have been read: the output tile goes over them
    // ---- 4. and 5.: blocks below the diagonal, row by row, each stored as soon as it is known
    const uint32_t out = smem_u32(scratch);
    const int mtx = lane >> 3;  // stmatrix: this lane addresses row l7 of matrix mtx
#pragma unroll
    for (int i = 1; i < 4; ++i) {
      Op16 Lop[3];
#pragma unroll
      for (int kk = 0; kk < i; ++kk) Lop[kk] = to_op(L[i * (i + 1) / 2 + kk]);
#pragma unroll
      for (int j = 0; j < i; ++j) {
        Block16 t, y;
        mma_abt<false>(t, Y[j][j], Lop[j]);
#pragma unroll
        for (int kk = j + 1; kk < i; ++kk) mma_abt<true>(t, Y[j][kk], Lop[kk]);
        mma_abt<false>(y, to_op(t), Dop[i]);
        if (i < 3) Y[j][i] = to_op(y);
        // 8 x 8 matrices (Y rows 8 a, columns 8 h; mtx = 2 h + a) go, transposed, to X rows 8 h,
        // columns 8 a of the block
        tc::stmatrix_x4_trans(
            out + (uint32_t)((16 * i + 8 * (mtx >> 1) + l7) * 128 + (((2 * j + (mtx & 1)) ^ l7) << 4)),
            pack_bf16(y.c[0][0], y.c[0][1]), pack_bf16(y.c[0][2], y.c[0][3]),
            pack_bf16(y.c[1][0], y.c[1][1]), pack_bf16(y.c[1][2], y.c[1][3]));
      }
    }
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int z = 0; z < 2; ++z)
          *reinterpret_cast<uint32_t*>(scratch + (16 * b + q8 + 8 * z) * 128 + (((2 * b + h) ^ q8) << 4) + 4 * t4) =
              dpack[b][2 * h + z];
    // blocks above the diagonal: zero (lane: row lane / 2 of the block, 16-byte half lane % 2)
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = i + 1; j < 4; ++j) {
        const int r = 16 * i + (lane >> 1);
        *reinterpret_cast<uint4*>(scratch + r * 128 + (((2 * j + (lane & 1)) ^ (r & 7)) << 4)) =
            make_uint4(0, 0, 0, 0);
      }
    if (valid == CHUNK) {
      tc::fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        tc::tma_store_2d(&map_a, hv * CHUNK, (int)row0, scratch);
        tc::tma_store_commit();
      }
    } else {
      __syncwarp();
      for (int i = lane; i < valid * 8; i += 32) {
        const int r = i >> 3, c = i & 7;
        *reinterpret_cast<uint4*>(A + ((row0 + r) * Hv + hv) * CHUNK + 8 * c) =
            *reinterpret_cast<const uint4*>(scratch + r * 128 + ((c ^ (r & 7)) << 4));
      }
    }
  }  // value heads of this warp
  if (lane == 0) tc::tma_store_wait_read();  // shared memory outlives the stores' reads
  if (tries <= 0) atomicCAS(&g_kkt_status, 0, 1);
}

// ------------------------------------------------------------------------------------------
// Grouped-value-attention reduce: out[row, hq, :] = sum_{i<G} in[row, hq*G+i, :], fp32 adds.
// HBM-bound: reads 2*D*G bytes and writes 2*D bytes per (token, q head).
// ------------------------------------------------------------------------------------------
__global__ void group_reduce_kernel(const bf16* __restrict__ in, bf16* __restrict__ out,
                                    long long n_vec, int G, int D8) {
  // one thread per 8-element (16-byte) segment of an output row
  pdl_wait();
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_vec) return;
  long long row_hq = i / D8;
  int seg = (int)(i % D8);
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int j = 0; j < G; ++j) {
    uint4 raw = *reinterpret_cast<const uint4*>(in + ((row_hq * G + j) * D8 + seg) * 8);
    const bf162* p = reinterpret_cast<const bf162*>(&raw);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float2 f = __bfloat1622float2(p[e]);
      acc[2 * e] += f.x;
      acc[2 * e + 1] += f.y;
    }
  }
  uint4 res;
  uint32_t* pr = reinterpret_cast<uint32_t*>(&res);
#pragma unroll
  for (int e = 0; e < 4; ++e) pr[e] = pack_bf16(acc[2 * e], acc[2 * e + 1]);
  *reinterpret_cast<uint4*>(out + i * 8) = res;
}

int kkt_status(int* out, int reset) {
  int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_kkt_status, sizeof(int));
  if (e != cudaSuccess) return (int)e;
  *out = v;
  if (reset && v != 0) {
    int z = 0;
    e = cudaMemcpyToSymbol(g_kkt_status, &z, sizeof(int));
  }
  return (int)e;
}

}  // namespace fqla

using namespace fqla;

extern "C" int fqla_chunk_local_cumsum(const float* g, float* out, int B, int T, int H,
                                       const void* cu_seqlens, int idx_is64, int N,
                                       const void* chunk_indices, long long num_chunks,
                                       int reverse, void* stream) {
  if (!g || !out || B <= 0 || T < 0 || H <= 0) return FQLA_ERR_INVALID_ARG;
  if (cu_seqlens && (!chunk_indices || B != 1)) return FQLA_ERR_INVALID_ARG;
  SeqLayout lay{{cu_seqlens, idx_is64}, {nullptr, idx_is64}, T};
  long long n = cu_seqlens ? num_chunks : (long long)B * ((T + CHUNK - 1) / CHUNK);
  if (n <= 0) return FQLA_OK;
  return launch_pdl(cumsum_kernel, dim3((unsigned)n), dim3(128), 0, (cudaStream_t)stream,
      g, out, H, B * T, lay, IndexTable{chunk_indices, idx_is64}, cu_seqlens ? N : B, reverse);
}

template <int D>
static int launch_kkt(const void* k, const void* beta, int beta_is_f32, const float* g,
                      float* g_cum_out, void* A, int Hq, int Hv, SeqLayout lay, IndexTable ci,
                      long long n, long long T_rows, cudaStream_t st) {
  const int G = Hv / Hq, warps = G < kkt::MAX_WARPS ? G : kkt::MAX_WARPS;
  static std::atomic<unsigned long long> done;
  int rc = configure_smem((const void*)kkt_solve_kernel<D>, kkt::smem_bytes<D>(kkt::MAX_WARPS), done);
  if (rc != 0) return rc;
  CUtensorMap mk, ma;
  if ((rc = make_tile_map(&mk, k, T_rows, (long long)Hq * D, 64))) return rc;
  if ((rc = make_tile_map(&ma, A, T_rows, (long long)Hv * CHUNK, 64))) return rc;
  return launch_pdl(kkt_solve_kernel<D>, dim3((unsigned)n, Hq), dim3(32 * warps),
                    (size_t)kkt::smem_bytes<D>(warps), st, beta, beta_is_f32, g, g_cum_out, (bf16*)A, Hq, Hv,
                    lay, ci, mk, ma);
}

extern "C" int fqla_kkt_solve(const void* k, const void* beta, int beta_is_f32,
                              const float* g_cum, float* g_cum_out, void* A, int B, int T, int Hq,
                              int Hv, int D,
                              const void* cu_seqlens, int idx_is64, const void* chunk_indices,
                              long long num_chunks, void* stream) {
  if (!k || !beta || !g_cum || !A || Hq <= 0 || Hv % Hq) return FQLA_ERR_INVALID_ARG;
  if (cu_seqlens && (!chunk_indices || B != 1)) return FQLA_ERR_INVALID_ARG;
  SeqLayout lay{{cu_seqlens, idx_is64}, {nullptr, idx_is64}, T};
  IndexTable ci{chunk_indices, idx_is64};
  long long n = cu_seqlens ? num_chunks : (long long)B * ((T + CHUNK - 1) / CHUNK);
  if (n <= 0) return FQLA_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (D == 128) return launch_kkt<128>(k, beta, beta_is_f32, g_cum, g_cum_out, A, Hq, Hv, lay, ci, n, (long long)B * T, st);
  if (D == 64) return launch_kkt<64>(k, beta, beta_is_f32, g_cum, g_cum_out, A, Hq, Hv, lay, ci, n, (long long)B * T, st);
  return FQLA_ERR_UNSUPPORTED_DIM;
}

extern "C" int fqla_group_reduce(const void* in, void* out, long long rows, int Hq, int G, int D,
                                 void* stream) {
  if (!in || !out || G <= 0 || D % 8) return FQLA_ERR_INVALID_ARG;
  long long n_vec = rows * Hq * (D / 8);
  if (n_vec <= 0) return FQLA_OK;
  return launch_pdl(group_reduce_kernel, dim3((unsigned)((n_vec + 255) / 256)), dim3(256), 0,
                    (cudaStream_t)stream, (const bf16*)in, (bf16*)out, n_vec, G, D / 8);
}
