// Blackwell (sm_100a) building blocks: mbarrier, TMA (cp.async.bulk.tensor), tensor memory and
// tcgen05.mma wrappers, shared-memory matrix descriptors and the 128-byte swizzle used for every
// tensor-core operand tile in this library.
//
// Operand tile convention ("SW128 tile"): rows of 64 bf16 (128 bytes); 8 consecutive rows form a
// 1024-byte swizzle atom in which the 16-byte chunk c of row r is stored at chunk c ^ (r & 7).
// A tile base must be 1024-byte aligned.  This is exactly what TMA writes for a box of 64 bf16
// columns with CU_TENSOR_MAP_SWIZZLE_128B.  Wider matrices are stored as consecutive 64-column
// blocks (block stride = rows * 128 bytes).
//   * As a K-major operand (contraction along the 64 columns): SBO = 1024; a K step of 16
//     elements advances the start address by 32 bytes inside the block.
//   * As an MN-major operand (contraction along the rows): LBO = block stride, SBO = 1024; a
//     K step of 16 rows advances the start address by 2048 bytes.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <stdint.h>

namespace fqla {
namespace tc {

__device__ __forceinline__ uint32_t s32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// ---- swizzle -------------------------------------------------------------------------------
// byte offset inside an SW128 tile of element (row, col), col in [0,64)
__device__ __forceinline__ uint32_t sw128_offset(int row, int col) {
  return (uint32_t)(row * 128 + ((((col >> 3) ^ (row & 7)) << 4) | ((col & 7) << 1)));
}

// ---- mbarrier ------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s32(bar)) : "memory");
}
// ... of a thread that has given no wait up (see mbar_wait)
__device__ __forceinline__ void mbar_arrive_if(uint64_t* bar, int tries) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(s32(bar)),
      "r"(tries)
      : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {  // without an arrival
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(s32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s32(bar)),
               "r"(bytes)
               : "memory");
}
// One try: the thread may be suspended by the hardware until the phase completes or a system limit runs out (4 us
// in a block where nothing else happens, sooner in a busy one); no instructions are issued meanwhile.
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(s32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait.  `tries` is the thread's own count, WAIT_TRIES at the start of each pass of its loop; a wait that
// uses it up falls through, and every wait after it does so after one try: looks with a result at each of the dozens
// of wait sites were a fifth of the kernels' code.  Such a thread issues, signals and stores nothing more, so that the
// threads that wait for it run out too, and the block ends after two limits or so, with its values lost and the status
// word set.  The lanes of a warp count each for themselves: only a vote may take a warp out of a loop.
// The limit: a try of a block that stands still takes 4.07 us with its pause (100 of them 408 us), so 2^18 a second.
// (It was 2^24, more than a minute.)
// The thread is suspended by the hardware meanwhile, but comes back early and often: trying again at once takes
// issue slots from the warps that have work, hence the pause (chunk-parallel backward, 262144 tokens x 8 heads:
// 1510 us without it, 1260 with, whether 20 or 400 ns; 1340 with a look at an abort flag in its place).  Polling with
// test_wait instead, or once before it, costs more (forward recurrence 467 us, 484 with a test at the waits that are
// mostly over).
constexpr int WAIT_TRIES = 1 << 18;
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity, int& tries) {
  asm volatile(
      "{\n\t.reg .pred p;\n"
      "W%=:\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "@p bra D%=;\n\t"
      "nanosleep.u32 20;\n\tadd.s32 %0, %0, -1;\n\tsetp.gt.s32 p, %0, 0;\n\t@p bra W%=;\n"
      "D%=:\n\t}"
      : "+r"(tries)
      : "r"(s32(bar)), "r"(parity)
      : "memory");
}

// The same for a warp that issues products: it stays converged in the compiler's eyes, which keeps what is
// computed between its waits in uniform registers, and may leave its loop right where a wait has been given up
// (false), which costs nothing where it has not.
__device__ __forceinline__ bool mbar_wait_uniform(uint64_t* bar, uint32_t parity, int& tries) {
#pragma unroll 1
  while (!__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) {
    if (--tries <= 0) return false;
    __nanosleep(20);
  }
  return true;
}

// Named barrier ID of N threads that tells all of them alike whether `ok` holds for each: a group that meets at
// barriers leaves its loop as one, although each thread counts its own tries.
template <int ID, int N>
__device__ __forceinline__ bool bar_all(bool ok) {
  uint32_t all;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.and.pred q, %2, %3, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(all)
      : "r"((uint32_t)ok), "n"(ID), "n"(N)
      : "memory");
  return all != 0;
}

// Four 8 x 8 bf16 matrices from registers to shared memory, each stored TRANSPOSED: register i of
// lane l carries the elements (row l/4, columns 2(l%4), +1) of matrix i - the layout of an
// mma / 16x256b tensor-memory fragment - and lands at (row 2(l%4) + {0,1}, column l/4) of the
// stored matrix, whose row r (16 bytes) starts at the address given by lane 8i + r.
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t saddr, uint32_t r0, uint32_t r1,
                                                  uint32_t r2, uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(saddr),
               "r"(r0), "r"(r1), "r"(r2), "r"(r3)
               : "memory");
}

// One, two or four 8 x 8 matrices as they are, or one or two transposed; lane 8 i + r gives the address of
// row r of matrix i.
__device__ __forceinline__ void stmatrix_x4(uint32_t saddr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "r"(r0), "r"(r1),
               "r"(r2), "r"(r3)
               : "memory");
}
__device__ __forceinline__ void stmatrix_x2(uint32_t saddr, uint32_t r0, uint32_t r1) {
  asm volatile("stmatrix.sync.aligned.m8n8.x2.shared.b16 [%0], {%1, %2};" ::"r"(saddr), "r"(r0), "r"(r1) : "memory");
}
__device__ __forceinline__ void stmatrix_x1(uint32_t saddr, uint32_t r0) {
  asm volatile("stmatrix.sync.aligned.m8n8.x1.shared.b16 [%0], {%1};" ::"r"(saddr), "r"(r0) : "memory");
}
__device__ __forceinline__ void stmatrix_x2_trans(uint32_t saddr, uint32_t r0, uint32_t r1) {
  asm volatile("stmatrix.sync.aligned.m8n8.x2.trans.shared.b16 [%0], {%1, %2};" ::"r"(saddr), "r"(r0), "r"(r1)
               : "memory");
}
__device__ __forceinline__ void stmatrix_x1_trans(uint32_t saddr, uint32_t r0) {
  asm volatile("stmatrix.sync.aligned.m8n8.x1.trans.shared.b16 [%0], {%1};" ::"r"(saddr), "r"(r0) : "memory");
}
// an 8 x 8 matrix in fragment form, transposed across the warp
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t r) {
  uint32_t t;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(t) : "r"(r));
  return t;
}

// ---- issuing warps -----------------------------------------------------------------------------
// A warp that issues tcgen05 and TMA instructions stays CONVERGED: all its lanes run the loop and
// the waits, and only the instructions themselves sit behind elect_one().  The compiler then keeps
// descriptors in uniform registers: six instructions per MMA.  Inside a divergent `lane == 0` branch
// it cannot know that one thread is active and emits a loop over distinct operand values for every
// MMA, 49 instructions (790 bytes of code) each: 58 of the forward recurrence kernel's 93 KB,
// streamed through instruction caches that the SMs of a GPC share (a chunk took 4.3 k cycles on an
// otherwise idle GPC and 7.3 k with all its SMs busy).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(p));
  return p != 0;
}
// ---- cluster launch control ----------------------------------------------------------------------
// Asks for a block of this grid that has not started yet.  It then never starts, and the block that asked
// does its work: dynamic hand-out of a grid without a counter in memory.  The answer (16 bytes, written
// by the async proxy) lands in `slot` and counts on `bar`, which expects 16 bytes.  After an answer
// without a block a CTA must not ask again.
__device__ __forceinline__ void clc_try_cancel(void* slot, uint64_t* bar) {
  asm volatile(
      "clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
          s32(slot)),
      "r"(s32(bar))
      : "memory");
}
// The answer: the block's index in a one-dimensional grid, or -1.
__device__ __forceinline__ int clc_block(const void* slot) {
  uint32_t found, x;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 answer;\n\t"
      "ld.shared.b128 answer, [%2];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, answer;\n\t"
      "selp.u32 %0, 1, 0, p;\n\tmov.u32 %1, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, answer;\n\t}"
      : "=r"(found), "=r"(x)
      : "r"(s32(slot))
      : "memory");
  return found ? (int)x : -1;
}

// ---- proxy / tcgen05 fences ------------------------------------------------------------------
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// ---- TMA -----------------------------------------------------------------------------------
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, int x, int y,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, "
      "{%2, %3}], [%4];" ::"r"(s32(smem_dst)),
      "l"(map), "r"(x), "r"(y), "r"(s32(bar))
      : "memory");
}
// Tile store shared -> global (bulk async group of the issuing thread).  The shared-memory tile
// must have been written, fenced (fence.proxy.async) and handed over to the issuing thread.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int x, int y,
                                             const void* smem_src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map),
               "r"(x), "r"(y), "r"(s32(smem_src))
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// every store group committed so far by this thread has finished READING shared memory
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
// ... and has been written to global memory
__device__ __forceinline__ void tma_store_wait_all() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// ---- tensor memory ---------------------------------------------------------------------------
// One warp allocates `ncols` (power of two >= 32) columns; the base address lands in *slot.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(slot)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}

// 32 lanes x 32 consecutive columns -> 32 registers per thread (thread = lane of its warp's
// quarter of the tensor memory: warp w may only touch lanes 32*(w%4) .. 32*(w%4)+31).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// 16 lanes x 64 consecutive columns spread over the 32 threads of a warp (the natural read of an
// M = 64 accumulator quarter): register 4i+e of lane l holds row l/4 + 8*(e>>1), column
// 8*i + 2*(l%4) + (e&1).  `taddr` names the first of the 16 lanes.
__device__ __forceinline__ void tmem_ld_16x64(uint32_t taddr, float (&v)[32]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// The same over 32 columns (x4).
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, float (&v)[16]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// 32 lanes x 16 consecutive columns -> 16 registers per thread
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float (&v)[32]) {
  const uint32_t* r = reinterpret_cast<const uint32_t*>(v);
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};" ::"r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
      "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
      "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
      "r"(r[30]), "r"(r[31]), "r"(taddr)
      : "memory");
}
// 32 lanes x 16 consecutive columns from 16 registers per thread (e.g. 32 packed bf16 per lane)
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};" ::"r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
      "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// ---- descriptors -----------------------------------------------------------------------------
// Instruction descriptor for kind::f16 with bf16 inputs and fp32 accumulation.
//   bits [4,6) D format (1 = f32), [7,10) A format (1 = bf16), [10,13) B format, 15 A major
//   (0 = K, 1 = MN), 16 B major, [17,23) N >> 3, [24,29) M >> 4.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N, int a_mn_major, int b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn_major << 15) |
         ((uint32_t)b_mn_major << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Shared-memory matrix descriptor for an SW128 tile (see the convention at the top):
//   bits [0,14) start address >> 4, [16,30) leading byte offset >> 4, [32,46) stride byte offset
//   >> 4, [46,48) version = 1, [61,64) layout type = 2 (128-byte swizzle).
// All of them have the same high word (SBO = 1024, version 1, 128-byte swizzle); the low word is
// (address >> 4) | (LBO >> 4) << 16, so a K step is one 32-bit add on a per-tile base kept in a register.
// Few, mutually independent instructions per MMA matter: the issuing thread shares its scheduler with three busy
// warps and pays a scheduling delay for every dependent instruction.
constexpr uint32_t DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_lo_kmajor(const void* tile) {
  return ((s32(tile) >> 4) & 0x3FFF) | (1u << 16);
}
__device__ __forceinline__ uint32_t desc_lo_mnmajor(const void* tile, uint32_t block_stride_bytes) {
  return ((s32(tile) >> 4) & 0x3FFF) | ((block_stride_bytes >> 4) << 16);
}
// D[tmem] (+)= A[smem] * B[smem]; issued by one thread.
template <bool ACCUMULATE>
__device__ __forceinline__ void umma_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo,
                                        uint32_t idesc) {
  if (ACCUMULATE) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 p, 1, 0;\n\t"
        "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}" ::"r"(d_tmem),
        "r"(a_lo), "r"(b_lo), "r"(DESC_HI), "r"(idesc)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 p, 0, 0;\n\t"
        "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}" ::"r"(d_tmem),
        "r"(a_lo), "r"(b_lo), "r"(DESC_HI), "r"(idesc)
        : "memory");
  }
}
// ... onto the accumulator where acc is not zero
__device__ __forceinline__ void umma_acc(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, int acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}" ::"r"(d_tmem),
      "r"(a_lo), "r"(b_lo), "r"(DESC_HI), "r"(idesc), "r"(acc)
      : "memory");
}
// One product: NK K-steps; operand low words advance by A_STEP / B_STEP (units of 16 bytes) per
// step, plus A_BLK / B_BLK after every fourth step (next 64-column block of a K-major operand).
template <int NK, int A_STEP, int A_BLK, int B_STEP, int B_BLK, bool ACC_FIRST>
__device__ __forceinline__ void umma_group(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo,
                                           uint32_t idesc) {
#pragma unroll
  for (int j = 0; j < NK; ++j) {
    const uint32_t a = a_lo + (uint32_t)((j & 3) * A_STEP + (j >> 2) * A_BLK);
    const uint32_t b = b_lo + (uint32_t)((j & 3) * B_STEP + (j >> 2) * B_BLK);
    if (j == 0 && !ACC_FIRST) umma_lo<false>(d_tmem, a, b, idesc);
    else umma_lo<true>(d_tmem, a, b, idesc);
  }
}

// The same as NB passes of a loop over four unrolled steps: the operand words advance by A_BLK / B_BLK a pass.
template <int NB, int A_STEP, int A_BLK, int B_STEP, int B_BLK>
__device__ __forceinline__ void umma_loop(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc) {
#pragma unroll 1
  for (int b = 0; b < NB; ++b) {
    umma_acc(d_tmem, a_lo, b_lo, idesc, b);
#pragma unroll
    for (int j = 1; j < 4; ++j) umma_lo<true>(d_tmem, a_lo + (uint32_t)(j * A_STEP), b_lo + (uint32_t)(j * B_STEP), idesc);
    a_lo += A_BLK;
    b_lo += B_BLK;
  }
}

// ---- A operand in tensor memory ("TS" form) -------------------------------------------------------
// The A matrix [M = 128 rows][K] sits in tensor memory: lane = row, one 32-bit column holds the
// two bf16 elements k = 2c (low half) and k = 2c + 1 (high half); a K step of 16 elements is 8
// columns.  It is written there with tcgen05.st by the thread that owns the lane.  B comes from
// shared memory as usual.  The product reads no shared memory for A: the tensor pipe, whose rate
// in the SS form is set by the 128 B/clk operand fetch, runs at its arithmetic rate.
template <bool ACCUMULATE>
__device__ __forceinline__ void umma_ts_lo(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo,
                                           uint32_t idesc) {
  if (ACCUMULATE) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
        "setp.ne.b32 p, 1, 0;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "r"(b_lo), "r"(DESC_HI), "r"(idesc)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
        "setp.ne.b32 p, 0, 0;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "r"(b_lo), "r"(DESC_HI), "r"(idesc)
        : "memory");
  }
}
// Eight K-steps as two passes of a loop, fresh accumulator: B advances by B_STEP a step, by B_BLK a pass.
template <int B_STEP, int B_BLK>
__device__ __forceinline__ void umma_ts_loop8(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc) {
#pragma unroll 1
  for (int b = 0; b < 2; ++b) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "r"(b_lo), "r"(DESC_HI), "r"(idesc), "r"(b)
        : "memory");
#pragma unroll
    for (int j = 1; j < 4; ++j)
      umma_ts_lo<true>(d_tmem, a_tmem + (uint32_t)(8 * j), b_lo + (uint32_t)(j * B_STEP), idesc);
    a_tmem += 32;
    b_lo += B_BLK;
  }
}
// NK K-steps; A advances A_COLS columns per step, B by B_STEP descriptor units (16 bytes) per step
// (an MN-major B tile: 128 = 16 rows; a K-major B tile of one 64-column block: 2).
template <int NK, int A_COLS, int B_STEP, bool ACC_FIRST>
__device__ __forceinline__ void umma_ts_group(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo,
                                              uint32_t idesc) {
#pragma unroll
  for (int j = 0; j < NK; ++j) {
    if (j == 0 && !ACC_FIRST) umma_ts_lo<false>(d_tmem, a_tmem, b_lo, idesc);
    else umma_ts_lo<true>(d_tmem, a_tmem + (uint32_t)(j * A_COLS), b_lo + (uint32_t)(j * B_STEP), idesc);
  }
}
// B = a K-major tile of NK / 4 blocks of 64 columns (block stride 8192 bytes), fresh accumulator.
template <int NK>
__device__ __forceinline__ void umma_ts_group_kmajor_b(uint32_t d_tmem, uint32_t a_tmem,
                                                       uint32_t b_lo, uint32_t idesc) {
#pragma unroll
  for (int j = 0; j < NK; ++j) {
    const uint32_t b = b_lo + (uint32_t)((j & 3) * 2 + (j >> 2) * 512);
    if (j == 0) umma_ts_lo<false>(d_tmem, a_tmem, b, idesc);
    else umma_ts_lo<true>(d_tmem, a_tmem + (uint32_t)(j * 8), b, idesc);
  }
}

// mbarrier arrives (count 1) once every tcgen05.mma issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   s32(bar))
               : "memory");
}

}  // namespace tc
}  // namespace fqla
