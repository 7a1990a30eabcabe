// tcgen05 / TMA / mbarrier primitives shared by the tensor-core projection kernels (gemm_tc.cu: fp16 and int8 weights,
// dense_tc.cu: bf16), and the tensor-map encoder behind them.  K-major operand tiles of 64 16-bit elements per row in
// 128-byte swizzled shared memory, fp32 accumulators in tensor memory.
#pragma once
#include <cuda.h>

#include "common.cuh"

// Tensor memory.  A kernel lets its successor start (pdl_launch) only behind its own tcgen05.alloc.  That waits, without a limit, until the
// SM has enough columns free, and a successor's CTA that shares the SM and was first to take them keeps them until the kernel it
// waits for has ended: all 512 columns of the prompt attention beside the 32 of a half-ring projection would wait for ever.

// Polls of one mbarrier phase before a wait gives up.  A try_wait that fails returns after the hardware's own
// suspend time (up to ~1 us), so the limit is of the order of seconds; every wait starts after the kernel's dependency
// wait, i.e. it only ever measures this kernel's own TMA / MMA progress.
constexpr uint32_t TC_SPIN_LIMIT = 1u << 24;

#ifdef __CUDACC__
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// The warp's index, known to the compiler as the same in all lanes.
__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }
// One lane of a converged warp.  The roles that issue tcgen05.mma, tcgen05.commit and TMA run their loops with all lanes and
// put only these instructions behind it: their operands then stay in uniform registers.  Loops behind `lane == 0` had them
// moved there lane by lane, some 84 cycles for each MMA and 264 for a stage's wait and commit (600 per 64-wide k-block of
// 256 x 128 as of 256 x 256, where the MMAs themselves take 256 and 512).
__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok)::"memory");
  return ok != 0;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait of a converged warp for the phase with the given parity; false = gave up.  The lanes poll together and leave
// together: a verdict of each lane's own would let some go on to elect.sync, __syncwarp or a tcgen05 .aligned instruction
// that waits for all of them.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (uint32_t i = 0; i < TC_SPIN_LIMIT; i++)
    if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
  return false;
}
// The same for a loop that one lane runs.
__device__ __forceinline__ bool mbar_wait_lane(uint64_t* bar, uint32_t parity) {
  for (uint32_t i = 0; i < TC_SPIN_LIMIT; i++)
    if (mbar_try(bar, parity)) return true;
  return false;
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
// K-major operand tile in 128-byte swizzled shared memory: rows of 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc(const void* tile) {
  const uint32_t lo = ((smem_u32(tile) & 0x3FFFFu) >> 4) | (1u << 16);  // start address, leading byte offset = 1 (unused)
  const uint32_t hi = 64u | (1u << 14) | (2u << 29);                    // stride 1024 B, descriptor version 1, SWIZZLE_128B
  return (uint64_t)lo | ((uint64_t)hi << 32);
}
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&r)[16]) {
  uint32_t u[16];
  tmem_ld16(taddr, u);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 16; j++) r[j] = __uint_as_float(u[j]);
}
// Cluster-wide barrier with release / acquire semantics (orders the distributed-shared-memory traffic around it).
__device__ __forceinline__ void cluster_barrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Shared-memory address `local` as seen in the CTA of rank `rank` of this cluster.
__device__ __forceinline__ uint32_t map_to_rank(uint32_t local, uint32_t rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  return remote;
}
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
#endif

// Tensor map of a row-major [rows][cols] matrix of 16-bit elements (or int8 when bytes == 1) with `ld` elements between
// rows, cut into boxes of box_rows x 64; out-of-range elements read as zero.  Maps are kept per argument set; `out` is a
// copy, because the next call may reuse the slot this one came from.
// groups > 0: boxes of box_rows x `groups` runs of 128 bytes, [run][row][128 bytes] in shared memory (rows of a whole number of
// runs); groups < 0: boxes of box_rows x -groups elements, as they lie.  slice > 0: a row is slices of that many runs, one more
// dimension, and the box's groups are spread evenly over `slices` of them.
int jg_tensor_map(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows,
                  const char* what, int bytes = 2, bool bf16 = false, int groups = 0,
                  int slice = 0, int slices = 1);
