// Dense projection on the 5th-generation tensor cores for 3 rows and more (batched decode, prompt processing):
// Y[m][n] = epilogue( sum_k X[m][k] * W[n][k] ) with tcgen05.mma, the accumulator in tensor memory and both operands
// brought into 128-byte swizzled shared memory by TMA (cp.async.bulk.tensor).  Fp16 weights of more than 64 rows (gate and up: 32) mostly
// go to pairs of CTAs instead (gemm_pair.cuh, launch_tc_rows).
//
// The roles of the MMA are swapped with respect to the usual GEMM picture so that both operands are K-major exactly as
// they lie in memory (nn.Linear keeps W as [out][in], jsgrad/nn/index.ts:403-412): A = 128 weight rows x 64 k,
// B = TN activation rows x 64 k (TN = 16 ... 256), D[128 lanes = weight rows][TN columns = activation rows] in fp32.
// With few activation rows the kernel is a weight stream: every weight byte crosses HBM once, the pipeline is as deep
// as shared memory allows, and the first weight tiles are requested before the kernel waits for its predecessor.
// Warp roles: warp 0 issues the TMA loads, warp 1 owns tensor memory and issues the MMAs,
// warps 2-9 read the accumulator back (tcgen05.ld; a warp may touch the 32-lane quarter given by its id modulo 4, so
// two warps share a quarter and split its columns) and apply the epilogue.
//
// Split-K over a thread-block cluster: when the output tiles alone do not fill the GPU, the CTAs of a cluster
// (1,1,ks) share one output tile, each accumulating a slice of K; ranks > 0 then write their accumulators into rank 0's
// (by then idle) pipeline buffers through distributed shared memory and rank 0 adds them in rank order before the
// epilogue.  No cluster multicast is used anywhere: every CTA fetches its own tiles.
// int8 weights (Int8Linear with many rows, jsgrad/models/llama3.ts:35): the weight tile arrives by TMA as int8 (8 KB
// instead of 16), and the warps that will later run the epilogue — idle during the main loop — turn it into the fp16
// tile the MMA reads: thread = one weight row of the tile, half(q) * scale rounded once per element, written in the
// 128-byte swizzle pattern TMA would have produced (16-byte chunk c of row r lands at chunk c ^ (r % 8)), followed by a
// proxy fence.  The weights cross HBM as int8 once per pass; no fp16 copy of a matrix is ever written.
// Every mbarrier wait is bounded: a wait that does not complete sets an error word and the CTA winds down (cluster
// barriers are still reached, tensor memory is released in every case); the host reports JG_ETIMEDOUT at the next
// synchronisation.
#include <stdlib.h>
#include <string.h>

#include "common.cuh"
#include "gemm_pair.cuh"
#include "quant.cuh"
#include "transcendental.cuh"

enum { TC_STORE = 0, TC_RESIDUAL = 1, TC_SWIGLU = 2, TC_PARTIAL = 4 };

constexpr int TC_BM = 128;  // weight rows per CTA (MMA M)
constexpr int TC_BK = 64;   // k per stage: 64 halves = one 128-byte swizzle row
// Threads of a CTA: warp 0 TMA, warp 1 MMA, then EPW epilogue warps for each 32-lane quarter of tensor memory.
constexpr int tc_threads(int epw) { return 64 + 128 * epw; }
struct TcArgs {
  __half* y;
  float* y32;
  const __half* residual;
  int* err;  // device word: 0 = fine, otherwise the code of the first wait that gave up
  int M, N, K;
  int w_late;  // the weights were written by the preceding kernel: no load before the dependency wait
  const __half* s0;  // int8 weights: per-output-row scales of the (first / second) matrix
  const __half* s1;
};

template <int TN, int EPI, bool W8 = false, bool HALF = false>
struct TcCfg {
  static constexpr int NW = (EPI == TC_SWIGLU) ? 2 : 1;
  static constexpr uint32_t RAW_BYTES = W8 ? TC_BM * TC_BK : 0;  // the int8 tile as it arrives (8 KB)
  static constexpr int NCOL = NW * TN;                 // accumulator columns
  // epilogue warps per tensor-memory quarter: wide tiles leave each of them 64 columns (measured at 512 rows: 12.1 ->
  // 11.8 ms per prefill against two warps), narrow ones are over before more warps would pay (batch 32: 6.92k tok/s
  // with two, 6.84k with four)
  static constexpr int EPW = TN >= 128 ? 4 : 2;
  static constexpr int THREADS = tc_threads(EPW);
  static constexpr uint32_t A_BYTES = TC_BM * TC_BK * 2;  // 16 KB
  static constexpr uint32_t B_BYTES = TN * TC_BK * 2;
  static constexpr uint32_t STAGE_BYTES = NW * (A_BYTES + RAW_BYTES) + B_BYTES;  // [A0 | A1 | B | raw0 | raw1]
  // HALF: a ring of half the shared memory, so that two CTAs share an SM (few activation rows only)
  static constexpr int STAGES_FIT = ((HALF ? 110 : 225) * 1024) / STAGE_BYTES;
  static constexpr int STAGES = STAGES_FIT > 10 ? 10 : STAGES_FIT;
  // int8: every epilogue warp converts during the main loop, in CONV_SPLIT groups (EPW / NW: 1, 2 or 4) of four warps per
  // matrix (one thread per weight row); group g takes the k-blocks g, g + CONV_SPLIT, ..., so that many k-blocks are being
  // converted at once and a group's fixed costs (barrier wait, proxy fence, arrival) hide behind the other groups' work
  static constexpr int CONV_SPLIT = W8 ? (EPW / NW >= 1 ? EPW / NW : 1) : 1;
  static constexpr int CONV_WARPS = W8 ? 4 * NW * CONV_SPLIT : 0;
  // A wait by parity tells a phase from its neighbours only, so a group may be at most one use of a stage ahead of the
  // loads.  Where STAGES is a multiple of the groups, the group that converts a use of a stage converted the use before, and
  // is never further ahead.  In rings of 5 stages and 4 groups, or 3 and 2 (33 to 128 rows), that was another group: one whose
  // block landed early went through the wait for use u + 1 while use u was still on its way (its phase open, the one before
  // of the same parity), converted stale bytes and arrived for them, and the sums were wrong or the ring stopped.  There a
  // group first waits for the MMAs on the previous use, which come behind its conversion; the producer waits for the same
  // before it requests the tile, so this costs no time.
  static constexpr bool CONV_WAIT_EMPTY = W8 && STAGES % CONV_SPLIT != 0;
  static constexpr uint32_t TMEM_COLS = NCOL <= 32 ? 32 : (NCOL <= 64 ? 64 : (NCOL <= 128 ? 128 : (NCOL <= 256 ? 256 : 512)));
  static constexpr size_t SMEM = (size_t)STAGES * STAGE_BYTES + 1024;
  // split-K peers park their accumulators ([column][128 lanes] fp32 each) in rank 0's pipeline buffers
  static constexpr int MAX_KS = 1 + (int)(((size_t)STAGES * STAGE_BYTES) / ((size_t)NCOL * TC_BM * 4));
};

template <int TN, int EPI, bool W8 = false, bool HALF = false>
__global__ void __launch_bounds__(TcCfg<TN, EPI, W8, HALF>::THREADS, HALF ? 2 : 1) gemm_tc_kernel(const __grid_constant__ CUtensorMap tm_w0,
                                                             const __grid_constant__ CUtensorMap tm_w1,
                                                             const __grid_constant__ CUtensorMap tm_x, const TcArgs a) {
  using Cfg = TcCfg<TN, EPI, W8, HALF>;
  constexpr int NW = Cfg::NW, STAGES = Cfg::STAGES, NCOL = Cfg::NCOL;
  constexpr uint32_t A_BYTES = Cfg::A_BYTES, STAGE_BYTES = Cfg::STAGE_BYTES, TMEM_COLS = Cfg::TMEM_COLS;
  constexpr uint32_t RAW_BYTES = Cfg::RAW_BYTES, B_BYTES = Cfg::B_BYTES, RAW_OFF = NW * A_BYTES + B_BYTES;
  static_assert(!W8 || Cfg::CONV_WARPS <= 4 * Cfg::EPW, "the converting warps are epilogue warps");
  __shared__ __align__(8) uint64_t raw_full[W8 ? STAGES : 1], a_full[W8 ? STAGES : 1];
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_bar;
  __shared__ uint32_t s_tmem;
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int tok0 = blockIdx.x * TN, feat0 = blockIdx.y * TC_BM;
  const int ks = gridDim.z, rank = blockIdx.z;  // the cluster is (1,1,ks): the rank in it is blockIdx.z
  const int n_kb = a.K / TC_BK;
  const int kb0 = (int)((long long)rank * n_kb / ks), nk = (int)((long long)(rank + 1) * n_kb / ks) - kb0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    if (W8)
      for (int s = 0; s < STAGES; s++) { mbar_init(&raw_full[s], 1); mbar_init(&a_full[s], 4 * NW); }
    mbar_init(&acc_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {  // tensor memory for the accumulator(s): one warp allocates, the same warp frees
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = s_tmem;
  pdl_launch();  // only now: see tcgen05.cuh
  bool acc_ok = false;

  // All lanes run the loops of warps 0 and 1 (see elect_one) but in int8 tiles of 256 rows, where 16 converting warps want the issue
  // slots that 31 more polling lanes take: us, 8B shapes, loops of one lane / of all: 100 rows qkv 33.4 / 28.7, wo 17.2 / 15.5,
  // gate and up 61.0 / 58.6, down 36.4 / 31.1; 300 rows 33.2 / 37.2, 24.8 / 25.5, 169.1 / 170.6, 61.4 / 67.0
  constexpr bool ONE_LANE = W8 && TN > 128;
  auto wait = [](uint64_t* bar, uint32_t parity) { return ONE_LANE ? mbar_wait_lane(bar, parity) : mbar_wait(bar, parity); };
  auto leader = [] { return ONE_LANE || elect_one(); };
  if (warp == 0 && (!ONE_LANE || lane == 0)) {
    // ---- producer.  Weights do not depend on the preceding kernel: the first tiles are requested before the wait.
    const int pre = nk < STAGES ? nk : STAGES;
    if (a.w_late) pdl_wait();
    // fp16 weights land in the A tiles and complete full_bar together with the activations; int8 weights land in the
    // raw tiles and complete raw_full (the converting warps then fill the A tiles and complete a_full)
    auto load_w = [&](int i, int s) {
      unsigned char* st = tiles + (size_t)s * STAGE_BYTES;
      if (W8) {
        mbar_expect_tx(&raw_full[s], NW * RAW_BYTES);
        tma_load_2d(st + RAW_OFF, &tm_w0, (kb0 + i) * TC_BK, feat0, &raw_full[s]);
        if (NW == 2) tma_load_2d(st + RAW_OFF + RAW_BYTES, &tm_w1, (kb0 + i) * TC_BK, feat0, &raw_full[s]);
        mbar_expect_tx(&full_bar[s], B_BYTES);
      } else {
        mbar_expect_tx(&full_bar[s], STAGE_BYTES);
        tma_load_2d(st, &tm_w0, (kb0 + i) * TC_BK, feat0, &full_bar[s]);
        if (NW == 2) tma_load_2d(st + A_BYTES, &tm_w1, (kb0 + i) * TC_BK, feat0, &full_bar[s]);
      }
    };
    if (leader())
      for (int i = 0; i < pre; i++) load_w(i, i);
    pdl_wait();  // X comes from the previous kernel
    if (leader())
      for (int i = 0; i < pre; i++)
        tma_load_2d(tiles + (size_t)i * STAGE_BYTES + NW * A_BYTES, &tm_x, (kb0 + i) * TC_BK, tok0, &full_bar[i]);
    for (int i = pre; i < nk; i++) {
      const int s = i % STAGES;
      // the MMAs of the stage's previous use are done: its A and B tiles are free, and so is its raw tile (converted
      // before those MMAs could start)
      if (!wait(&empty_bar[s], ((i / STAGES) - 1) & 1)) { atomicCAS(a.err, 0, 1); break; }
      if (leader()) {
        load_w(i, s);
        tma_load_2d(tiles + (size_t)s * STAGE_BYTES + NW * A_BYTES, &tm_x, (kb0 + i) * TC_BK, tok0, &full_bar[s]);
      }
    }
  } else if (warp == 1 && (!ONE_LANE || lane == 0)) {
    // ---- MMA issuer: 4 x (128 x TN x 16) per stage and matrix, accumulating in tensor memory
    const uint32_t idesc = (1u << 4) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);  // f32 acc, f16 x f16, K-major both
    bool ok = true;
    // the poll budget of the waits below starts only once the predecessor is done: the producer cannot request the
    // activation tiles any earlier, so a slow predecessor must not use the budget up
    pdl_wait();
    for (int i = 0; i < nk; i++) {
      const int s = i % STAGES;
      if (!wait(&full_bar[s], (i / STAGES) & 1)) { atomicCAS(a.err, 0, 2); ok = false; break; }
      if (W8 && !wait(&a_full[s], (i / STAGES) & 1)) { atomicCAS(a.err, 0, 2); ok = false; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      unsigned char* st = tiles + (size_t)s * STAGE_BYTES;
      const uint64_t bdesc = umma_desc(st + NW * A_BYTES);
      if (leader()) {
#pragma unroll
        for (int w = 0; w < NW; w++) {
          const uint64_t adesc = umma_desc(st + w * A_BYTES);
#pragma unroll
          for (int k = 0; k < TC_BK / 16; k++)  // 16 halves = 32 bytes further along K inside the swizzle row: +2 (16-byte units)
            umma_f16(tmem_base + w * TN, adesc + 2 * k, bdesc + 2 * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(&empty_bar[s]);  // arrives when the MMAs above have finished reading the stage
      }
    }
    if (ok && leader()) umma_commit(&acc_bar);  // ... and when the whole accumulation is complete
  } else if (warp >= 2) {
    if (W8 && warp - 2 < Cfg::CONV_WARPS) {
      // ---- converter: this thread's weight row of every stage, int8 -> half(q) * scale -> swizzled fp16 tile
      constexpr int CS = Cfg::CONV_SPLIT;
      const int cw = warp - 2, w = cw / (4 * CS), idx = cw % (4 * CS), r = (idx & 3) * 32 + lane, group = idx >> 2;
      if (a.w_late) pdl_wait();
      const __half2 sc = __half2half2((w == 0 ? a.s0 : a.s1)[min(feat0 + r, a.N - 1)]);
      const uint32_t row_off = (uint32_t)(r >> 3) * 1024u + (uint32_t)(r & 7) * 128u;
      for (int i = group; i < nk; i += CS) {
        const int s = i % STAGES;
        if (Cfg::CONV_WAIT_EMPTY && i >= STAGES && !mbar_wait(&empty_bar[s], ((i / STAGES) - 1) & 1)) { atomicCAS(a.err, 0, 1); break; }
        if (!mbar_wait(&raw_full[s], (i / STAGES) & 1)) { atomicCAS(a.err, 0, 1); break; }
        unsigned char* st = tiles + (size_t)s * STAGE_BYTES;
        const uint4* src = reinterpret_cast<const uint4*>(st + RAW_OFF + w * RAW_BYTES + r * TC_BK);
        unsigned char* dst = st + w * A_BYTES + row_off;
#pragma unroll
        for (int j = 0; j < 4; j++) {  // 16 weights -> two 16-byte chunks (2j, 2j + 1) of the row
          uint32_t d[8];
          w8_to_half2(src[j], sc, d);
          *reinterpret_cast<uint4*>(dst + (((2 * j) ^ (r & 7)) << 4)) = make_uint4(d[0], d[1], d[2], d[3]);
          *reinterpret_cast<uint4*>(dst + (((2 * j + 1) ^ (r & 7)) << 4)) = make_uint4(d[4], d[5], d[6], d[7]);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy stores -> visible to the MMA's reads
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&a_full[s])) : "memory");
      }
    }
    pdl_wait();  // the residual is read and Y written only after the previous kernel is done with them
    acc_ok = mbar_wait(&acc_bar, 0);
    if (!acc_ok && lane == 0) atomicCAS(a.err, 0, 3);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }

  // warp (id % 4) may touch tensor-memory lanes [32 * (id % 4), +32); lane l of it is weight row feat0 + 32q + l
  const int q = warp & 3, row = q * 32 + lane;
  // the two warps of a quarter split the accumulator columns (activation rows) between them
  const int part = (warp - 2) >> 2;
  constexpr int TN_PER = (TN / Cfg::EPW) >= 16 ? (TN / Cfg::EPW) : 16;
  constexpr int NC_PER = (NCOL / Cfg::EPW) >= 16 ? (NCOL / Cfg::EPW) : 16;
  const int tn_lo = part * TN_PER, tn_hi = min(TN, tn_lo + TN_PER);
  const int nc_lo = part * NC_PER, nc_hi = min(NCOL, nc_lo + NC_PER);
  const uint32_t t_lane = tmem_base + ((uint32_t)(q * 32) << 16);
  float* red = reinterpret_cast<float*>(tiles);  // rank 0: [ks-1][NCOL][128] partial accumulators of the peers
  if (ks > 1) {
    cluster_barrier();  // rank 0's MMAs have consumed its pipeline buffers (its epilogue warps waited for them)
    if (rank > 0 && warp >= 2 && acc_ok) {
      const uint32_t dst0 = map_to_rank(smem_u32(red + ((size_t)(rank - 1) * NCOL) * TC_BM + row), 0);
#pragma unroll 1
      for (int c0 = nc_lo; c0 < nc_hi; c0 += 16) {
        float r0[16];
        tmem_ld16(t_lane + c0, r0);
#pragma unroll
        for (int j = 0; j < 16; j++) st_cluster_f32(dst0 + (uint32_t)((c0 + j) * TC_BM * 4), r0[j]);
      }
    }
    cluster_barrier();  // the peers' partial sums have landed in rank 0
  }
  if (rank == 0 && warp >= 2 && acc_ok) {
    const int feat = feat0 + row;
#pragma unroll 1
    for (int c0 = tn_lo; c0 < tn_hi; c0 += 16) {
      float r0[16], r1[16];
      tmem_ld16(t_lane + c0, r0);
      if (NW == 2) tmem_ld16(t_lane + TN + c0, r1);
      for (int p = 1; p < ks; p++) {  // rank order
        const float* pr = red + ((size_t)(p - 1) * NCOL) * TC_BM + row;
#pragma unroll
        for (int j = 0; j < 16; j++) {
          r0[j] = __fadd_rn(r0[j], pr[(size_t)(c0 + j) * TC_BM]);
          if (NW == 2) r1[j] = __fadd_rn(r1[j], pr[(size_t)(TN + c0 + j) * TC_BM]);
        }
      }
      if (feat < a.N) {
        __half res[16];
        if (EPI == TC_RESIDUAL) {  // all loads first: Y may alias the residual, which would serialise load / store pairs
#pragma unroll
          for (int j = 0; j < 16; j++)
            res[j] = (tok0 + c0 + j < a.M) ? a.residual[(size_t)(tok0 + c0 + j) * a.N + feat] : __float2half_rn(0.f);
        }
#pragma unroll
        for (int j = 0; j < 16; j++) {
          const int tok = tok0 + c0 + j;
          if (tok < a.M) {
            const size_t o = (size_t)tok * a.N + feat;
            if (EPI == TC_PARTIAL) { a.y32[o] = r0[j]; continue; }
            __half v = __float2half_rn(r0[j]);
            if (EPI == TC_RESIDUAL) v = hadd1(res[j], v);
            if (EPI == TC_SWIGLU) v = jg_silu_mul(v, __float2half_rn(r1[j]));
            a.y[o] = v;
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// ------------------------------------------------------------------------------------------------ many rows
// What the paired kernel (gemm_pair.cuh) does with an accumulator: the same roundings as above.
template <int EPI>
struct TcPairEpi {
  static constexpr bool GLU = EPI == TC_SWIGLU, BF16 = false, RESIDUAL = EPI == TC_RESIDUAL;
  struct Args {
    __half* y;
    float* y32;
    const __half* residual;
    int aligned;  // results (and residual) start on 16 bytes
  };
  static __device__ __forceinline__ bool wide(const Args& e, const PairPlan& a, int feat) { return e.aligned && feat + (GLU ? 16 : 32) <= a.N; }
  static __device__ __forceinline__ bool f32(const Args&) { return EPI == TC_PARTIAL; }
  static __device__ __forceinline__ float* out32(const Args& e, const PairPlan& a, int tok, int feat) { return e.y32 + (size_t)tok * a.N + feat; }
  static __device__ __forceinline__ __half* out(const Args& e, const PairPlan& a, int tok, int feat) { return e.y + (size_t)tok * a.N + feat; }
  static __device__ __forceinline__ const __half* residual(const Args& e, const PairPlan& a, int tok, int feat) { return e.residual + (size_t)tok * a.N + feat; }
  static __device__ __forceinline__ float value(const Args&, const PairPlan&, int, int, float r) { return r; }
  static __device__ __forceinline__ uint16_t round(float v) { return __half_as_ushort(__float2half_rn(v)); }
  static __device__ __forceinline__ uint32_t add(uint32_t v, uint32_t res) {
    const __half2 h = __hadd2_rn(*reinterpret_cast<const __half2*>(&res), *reinterpret_cast<const __half2*>(&v));
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  static __device__ __forceinline__ uint16_t glu(const Args&, int, float gate, float up) {
    return __half_as_ushort(jg_silu_mul(__float2half_rn(gate), __float2half_rn(up)));
  }
  static __device__ __forceinline__ void store(const Args& e, const PairPlan& a, int feat, int tok, float v) {
    if (EPI == TC_PARTIAL) { *out32(e, a, tok, feat) = v; return; }
    __half h = __float2half_rn(v);
    if (EPI == TC_RESIDUAL) h = hadd1(*residual(e, a, tok, feat), h);
    *out(e, a, tok, feat) = h;
  }
};

// ------------------------------------------------------------------------------------------------ host side
static int cached_map(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows, const char* what, int bytes = 2) {
  return jg_tensor_map(out, base, rows, cols, cols, box_rows, what, bytes);
}

template <int TN, int EPI, bool W8 = false, bool HALF = false>
static int launch_tc(jg_dev* dev, const void* x, const void* w0, const void* w1, TcArgs a) {
  using Cfg = TcCfg<TN, EPI, W8, HALF>;
  auto kern = gemm_tc_kernel<TN, EPI, W8, HALF>;
  static bool attr_set[8] = {false, false, false, false, false, false, false, false};
  const int slot = dev->ordinal & 7;
  if (!attr_set[slot]) {
    JG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM));
    attr_set[slot] = true;
  }
  CUtensorMap tw0, tw1, tx;
  int rc = cached_map(&tw0, w0, a.N, a.K, TC_BM, "weights", W8 ? 1 : 2);
  if (rc) return rc;
  rc = cached_map(&tw1, Cfg::NW == 2 ? w1 : w0, a.N, a.K, TC_BM, "weights (second matrix)", W8 ? 1 : 2);
  if (rc) return rc;
  rc = cached_map(&tx, x, a.M, a.K, TN, "activations");
  if (rc) return rc;
  // up to 128 rows (weight streaming): split K over a cluster until the launch has CTAs for about two thirds of the
  // SMs, keeping at least 8 k-blocks per CTA and the peers' partial sums within rank 0's pipeline buffers
  const int tiles = ((a.M + TN - 1) / TN) * (a.N / TC_BM), n_kb = a.K / TC_BK;
  static int ks_env = -1;
  if (ks_env < 0) { const char* e = getenv("JG_TC_SPLITK"); ks_env = e ? atoi(e) : 0; }
  int ks = 1;
  if (a.M > 128) {
    // compute-bound tiles: the launch runs in waves of one CTA per SM, each costing its k-blocks (0.28 us apiece at
    // the tensor peak) plus about 18 us of fill, epilogue and cluster reduction (measured cold at 512 and 1024 rows:
    // qkv 36.9 us unsplit against 53.3 split in two, which makes 192 CTAs = two waves; wo 38.9 against 34.8; the
    // down projection 96.3 against 69.7).  Take the split with the smallest estimate.
    float best = 0.f;
    for (int c = 1; c <= Cfg::MAX_KS && c <= 8 && n_kb / c >= 8; c++) {
      const int waves = (tiles * c + dev->sm_count - 1) / dev->sm_count;
      const float t = (float)waves * ((float)(n_kb / c) * 0.28f + 18.f);
      if (c == 1 || t < best) { best = t; ks = c; }
    }
  } else {
    // half-size rings (two CTAs per SM): CTAs for four thirds of the SMs, but no more than four to a tile — beyond
    // that the cluster reduction costs more than the shorter streams save (wo at 32 rows: 18.5 us split in 4, 20.5 in 7;
    // 1B down projection, 45 rows, full rings: 23 us split in 7)
    while (ks < (tiles > 8 ? 4 : 8) && ks < Cfg::MAX_KS && tiles * ks * 3 < dev->sm_count * 2 * (HALF ? 2 : 1) && n_kb / (ks + 1) >= 8) ks++;
  }
  if (ks_env >= 1 && ks_env <= 8 && ks_env <= Cfg::MAX_KS && n_kb / ks_env >= 1) ks = ks_env;
  dev->tc_pending = true;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((a.M + TN - 1) / TN, a.N / TC_BM, ks);  // activation tiles fastest: CTAs sharing weights run together
  cfg.blockDim = dim3(Cfg::THREADS);
  cfg.dynamicSmemBytes = Cfg::SMEM;
  cfg.stream = dev->stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (ks > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 1;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = ks;
    na++;
  }
  if (dev->pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    na++;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tw0, tw1, tx, a);
  if (e != cudaSuccess) return jg_cuda_fail(e, "gemm_tc", __FILE__, __LINE__);
  return jg_after_launch(dev, "gemm_tc");
}

template <int EPI>
static int launch_tc_rows(jg_dev* dev, const void* x, const void* w0, const void* w1, const TcArgs& a) {
  // more than 64 rows, gate and up more than 32 (see cta_per_tile): pairs of CTAs.  us per launch, weights from HBM, one tile per CTA /
  // pairs: 8B shapes, 100 rows qkv 26.2 / 17.1, wo 17.0 / 14.9, down 31.0 / 32.2; 300 rows 26.4 / 19.9, 24.0 / 19.0, 53.5 / 40.5; 512
  // rows 26.8 / 26.4, 24.4 / 21.5, 59.0 / 55.4, gate and up 119 / 105; 1B shapes, 100 rows 12.4 / 10.0, 13.3 / 10.0, 26.8 / 19.8,
  // 20.6 / 16.1; 512 rows 15.7 / 11.7, 18.4 / 11.4, 40.3 / 34.5, 33.6 / 23.1
  if (a.s0 == nullptr && a.M > (EPI == TC_SWIGLU ? 32 : 64) && !(EPI == TC_SWIGLU && cta_per_tile(dev, a.M, a.N)))
    return launch_pair<TcPairEpi<EPI>>(dev, "gemm_pair", x, a.K, w0, w1, a.K, a.M, a.N, a.K, false, a.w_late,
                                       {a.y, a.y32, a.residual, (uintptr_t)a.y % 16 == 0 && (uintptr_t)a.residual % 16 == 0});
  if (a.s0 != nullptr) {  // int8 weights: used from 20 rows on (fewer go to the mma.sync kernel)
    if (a.M <= 32) return launch_tc<32, EPI, true>(dev, x, w0, w1, a);
    if (a.M <= 128) return launch_tc<128, EPI, true>(dev, x, w0, w1, a);
    return launch_tc<256, EPI, true>(dev, x, w0, w1, a);
  }
  // Up to 32 rows the single-matrix projections run with half-size rings, two CTAs to an SM and twice the split-K:
  // a qkv or wo launch is a few hundred KB per CTA, mostly fixed cost (measured cold and alone at 32 rows on the 8B
  // shapes: qkv 29.2 -> 22.6 us, wo 19.4 -> 18.5 at split 4, down 36.9 -> 37.9; the batch-32 decode step 4.27 -> 4.16 ms,
  // batch 16 4.04 -> 3.93).  JG_TC_HALF=0 turns it off.  The gate / up pair keeps the full ring (three stages would
  // not cover its loads).
  static int half_env = -1;
  if (half_env < 0) { const char* e = getenv("JG_TC_HALF"); half_env = e ? atoi(e) : 1; }
  if (half_env && EPI != TC_SWIGLU && a.M <= 32) {
    if (a.M <= 16) return launch_tc<16, EPI, false, true>(dev, x, w0, w1, a);
    return launch_tc<32, EPI, false, true>(dev, x, w0, w1, a);
  }
  if (a.M <= 16) return launch_tc<16, EPI>(dev, x, w0, w1, a);
  if (a.M <= 32) return launch_tc<32, EPI>(dev, x, w0, w1, a);
  if (a.M <= 64) return launch_tc<64, EPI>(dev, x, w0, w1, a);
  if constexpr (EPI == TC_SWIGLU) return a.M <= 128 ? launch_tc<128, EPI>(dev, x, w0, w1, a) : launch_tc<256, EPI>(dev, x, w0, w1, a);
  return JG_ENOTSUP;  // taken above
}

// Whether jg_gemm_tc takes this shape: fp16 weights, whole 128-row weight tiles and 64-wide k-blocks.
bool jg_gemm_tc_fits(int N, int K) { return N % TC_BM == 0 && K % TC_BK == 0; }

// Entry used by gemv.cu's public functions (fp16 weights, N % 128 == 0, K % 64 == 0).
// s0 / s1: per-row scales of int8 weights (w0 / w1 then hold int8), or null for fp16 weights.
int jg_gemm_tc(jg_dev* dev, int epi, const void* x, const void* w0, const void* w1, void* y, const void* residual, int M, int N, int K,
               const void* s0, const void* s1) {
  if (!jg_gemm_tc_fits(N, K)) {
    jg_set_error("projection: M=%d rows need N %% 128 == 0 and K %% 64 == 0 (N=%d, K=%d); split the rows into chunks of 64", M, N, K);
    return JG_ENOTSUP;
  }
  JG_REQUIRE(((uintptr_t)x % 16) == 0 && ((uintptr_t)w0 % 16) == 0, "projection: operands must be 16-byte aligned for TMA");
  TcArgs a = {};
  a.y = (__half*)y; a.y32 = (float*)y; a.residual = (const __half*)residual; a.err = dev->err_word; a.M = M; a.N = N; a.K = K;
  a.w_late = jg_is_fresh(dev, w0) || jg_is_fresh(dev, w1) || jg_is_fresh(dev, s0) || jg_is_fresh(dev, s1);
  a.s0 = (const __half*)s0; a.s1 = (const __half*)(s1 ? s1 : s0);
  switch (epi) {
    case TC_STORE: return launch_tc_rows<TC_STORE>(dev, x, w0, w1, a);
    case TC_RESIDUAL: return launch_tc_rows<TC_RESIDUAL>(dev, x, w0, w1, a);
    case TC_SWIGLU: return launch_tc_rows<TC_SWIGLU>(dev, x, w0, w1, a);
    case TC_PARTIAL: return launch_tc_rows<TC_PARTIAL>(dev, x, w0, w1, a);
  }
  jg_set_error("projection: epilogue %d has no tensor-core variant for M=%d rows", epi, M);
  return JG_ENOTSUP;
}
