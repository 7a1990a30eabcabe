// Projection of many rows on pairs of CTAs (tcgen05.mma.cta_group::2), persistent: Y[m][n] = epilogue(sum_k X[m][k] W[n][k]).
//
// What bounds it.  The MMAs of a 64-wide k-block of 256 x 256 take 512 cycles, the loop around them 527 (measured); with many
// rows the GPU then runs into its power limit (2048 rows of the 8B's gate and up: 1.2 GHz, 1.3 PFLOP/s).  Around that loop:
// two CTAs share a tile of 256 weight rows x up to 256 activation rows, each fetching its own weight rows and half of the
// activations, and a pair walks a list of tiles while the accumulators alternate between the two halves of tensor memory,
// so that the epilogue of one tile runs under the MMAs of the next.
//
// Shares.  Where the tiles are few, each is cut along K into `split` shares, a pair's whole work.  The pair with the first
// k-blocks stores the tile; the other pairs' accumulators reach it through global memory (fp32, a slot per CTA and a flag per
// warp), added in order of k, so a result never depends on timing.  A pair waits only for pairs of lower block index, and
// the reader clears the flag.  Slots and flags are touched after the dependency wait, so the next launch finds them free.
//
// Gate and up projections (GLU) interleave 16 rows of either matrix in the A tile: lanes l and l + 16 of a quarter of
// tensor memory then hold gate and up of one feature, and one shuffle per two columns brings them together.
//
// Every wait is bounded (JG_ETIMEDOUT at the next synchronisation).  No TMA multicast.
#pragma once
#include <math.h>

#include "tcgen05.cuh"

constexpr int GP_BK = 64, GP_STAGES = 7;
constexpr int GP_EPI_WARPS = 16, GP_PARTS = GP_EPI_WARPS / 4, GP_X_WARP = 2 + GP_EPI_WARPS, GP_THREADS = 32 * (GP_X_WARP + 1);
constexpr uint32_t GP_A_BYTES = 128 * GP_BK * 2, GP_STAGE_BYTES = 2 * GP_A_BYTES;
constexpr size_t GP_SMEM = (size_t)GP_STAGES * GP_STAGE_BYTES + 1024;
constexpr size_t GP_SLOT = 256 * 128;  // floats of one CTA's accumulators

struct PairPlan {
  int M, N, n_kb;
  int tn, tok_tiles;     // activation rows per tile (a multiple of 32), and tiles of them
  int tiles, pairs;      // tiles, and pairs in the grid
  int split, head;       // shares of a tile, and k-blocks in its first
  int w_late;
  int glu_one, glu_swap;  // GLU: one map covers both matrices; ... with the up projection first
  float* slots;           // [pairs][2][GP_SLOT]
  uint32_t* flags;        // [pairs][2][GP_EPI_WARPS]
  int* err;
};

// Makes sure that the device has slots and flags; false: not to be had now (first use inside a capture, no memory).
bool jg_pair_workspace(jg_dev* dev);
// Map of two [rows][cols] matrices, rows % 16 == 0, whose boxes are 64 columns of 4 groups of 16 rows of either in turn; false
// where their distance is none that a map can step by (lo < hi, a multiple of 16 bytes below 2^40).
bool jg_tensor_map_two(CUtensorMap* out, const void* lo, const void* hi, uint64_t rows, uint64_t cols, uint64_t ld, bool bf16);

#ifdef __CUDACC__
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int c0, int c1, uint32_t bar_cluster_addr) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(bar_cluster_addr), "r"(c0), "r"(c1)
               : "memory");
}
// box of a (k, 16 rows, matrix, group of rows) map: rows `group` * 16 ... of both matrices, 16 by 16 in turn
__device__ __forceinline__ void tma_load_4d_pair(void* dst, const CUtensorMap* map, int k, int group, uint32_t bar_cluster_addr) {
  asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %4, %5}], [%2];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(bar_cluster_addr), "r"(k), "r"(0), "r"(group)
               : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on this barrier of both CTAs once the pair's MMAs issued so far have completed.
__device__ __forceinline__ void umma_commit_both(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}
// mbar_wait for arrivals of the other CTA's threads
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity) {
  for (uint32_t i = 0; i < TC_SPIN_LIMIT; i++) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (__all_sync(0xffffffffu, ok != 0)) return true;
  }
  return false;
}

// What one pair works on: a share of a tile, or whole tiles in turn.
struct PairWork {
  int next, tile, k0, k1;
  __device__ __forceinline__ PairWork(const PairPlan& a, int pair) {
    next = pair;
    if (a.split > 1) next = a.pairs - 1 - pair;
  }
  __device__ __forceinline__ bool step(const PairPlan& a) {
    if (a.split > 1) {
      if (next < 0) return false;
      tile = next / a.split;
      const int part = next - tile * a.split, rest = a.n_kb - a.head;
      k0 = part == 0 ? 0 : a.head + (part - 1) * rest / (a.split - 1);
      k1 = part == 0 ? a.head : a.head + part * rest / (a.split - 1);
      next = -1;
      return true;
    }
    if (next >= a.tiles) return false;
    tile = next;
    k0 = 0;
    k1 = a.n_kb;
    next += a.pairs;
    return true;
  }
};

// Between lanes = features and lanes = tokens, so that a lane stores 16 bytes of a row.  A lane has the values of its feature for
// 16 tokens (pairs of 16-bit values, or 32-bit ones) and ends up with those of 8 features (lane & ~7 ...) for tokens lane & 7 and
// 8 + (lane & 7); of 4 features for tokens 4 m + (lane & 3).  Stores of 2 bytes per lane took 7.5 cycles an instruction: 7600
// cycles for a 256 x 256 tile at the end of a launch.
__device__ __forceinline__ uint32_t swap_lanes(uint32_t send, int bit) { return __shfl_xor_sync(0xffffffffu, send, bit); }
template <int NP>  // NP packed pairs: 8 (16 tokens) or 4 (8 tokens)
__device__ __forceinline__ void transpose_16bit(const uint32_t (&p)[NP], uint32_t (&o)[NP / 4][4], int lane) {
  const bool b0 = lane & 1, b1 = lane & 2, b2 = lane & 4;
  uint32_t q[NP], m[NP / 2][2];
#pragma unroll
  for (int i = 0; i < NP; i += 2) {  // two features of token 2 i + (lane & 1)
    const uint32_t got = swap_lanes(b0 ? __byte_perm(p[i], p[i + 1], 0x5410) : __byte_perm(p[i], p[i + 1], 0x7632), 1);
    q[i] = b0 ? __byte_perm(got, p[i], 0x7610) : __byte_perm(p[i], got, 0x5410);
    q[i + 1] = b0 ? __byte_perm(got, p[i + 1], 0x7632) : __byte_perm(p[i + 1], got, 0x7610);
  }
#pragma unroll
  for (int i = 0; i < NP; i += 2) {  // four
    const uint32_t got = swap_lanes(b1 ? q[i] : q[i + 1], 2);
    m[i / 2][0] = b1 ? got : q[i];
    m[i / 2][1] = b1 ? q[i + 1] : got;
  }
#pragma unroll
  for (int i = 0; i < NP / 2; i += 2)  // eight
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const uint32_t got = swap_lanes(b2 ? m[i][k] : m[i + 1][k], 4);
      o[i / 2][k] = b2 ? got : m[i][k];
      o[i / 2][2 + k] = b2 ? m[i + 1][k] : got;
    }
}
__device__ __forceinline__ void transpose_32bit(const float (&r)[16], float4 (&o)[4], int lane) {
  const bool b0 = lane & 1, b1 = lane & 2;
  float q[8][2];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const float got = __shfl_xor_sync(0xffffffffu, b0 ? r[2 * i] : r[2 * i + 1], 1);
    q[i][0] = b0 ? got : r[2 * i];
    q[i][1] = b0 ? r[2 * i + 1] : got;
  }
#pragma unroll
  for (int m = 0; m < 4; m++) {
    float w[4];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const float got = __shfl_xor_sync(0xffffffffu, b1 ? q[2 * m][k] : q[2 * m + 1][k], 2);
      w[k] = b1 ? got : q[2 * m][k];
      w[2 + k] = b1 ? q[2 * m + 1][k] : got;
    }
    o[m] = make_float4(w[0], w[1], w[2], w[3]);
  }
}

// Epi: GLU (two interleaved matrices), BF16, RESIDUAL, Args, and
//   wide(args, plan, feat)                whether the 32 (GLU: 16) features from feat on are stored in 16-byte pieces of rows
//   f32(args)                             results in 32 bits
//   out32, out, residual(args, plan, tok, feat)   where they, 16-bit ones and what is added to these are
//   value(args, plan, feat, tok, r)       what a 32-bit accumulator becomes ahead of the last rounding
//   round(v) / add(x, residual)           its 16 bits / two of them plus two of the residual
//   glu(args, feat, gate, up)             the 16 bits of a result (GLU)
//   store(args, plan, feat, tok, v)       one value, where the features are not wide
template <class Epi>
__global__ void __launch_bounds__(GP_THREADS, 1) gemm_pair_kernel(const __grid_constant__ CUtensorMap tm_w0, const __grid_constant__ CUtensorMap tm_w1,
                                                                  const __grid_constant__ CUtensorMap tm_x, const PairPlan a, const typename Epi::Args ea) {
  constexpr int STAGES = GP_STAGES;
  constexpr int FEATS = Epi::GLU ? 64 : 128;  // features of a CTA's part of a tile
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t s_tmem;
  const int warp = uniform_warp(), lane = threadIdx.x & 31, pair = blockIdx.x >> 1;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int s = 0; s < 2; s++) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], 2 * GP_EPI_WARPS); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {  // warp 1 of both CTAs together: all columns of both CTAs' tensor memory
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_barrier();  // the peer's barriers exist before anything is signalled across
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = s_tmem;
  pdl_launch();  // only now: see tcgen05.cuh

  if (warp == 0 || warp == GP_X_WARP) {
    // ---- producers of this CTA's weights and activations, a warp each.  Completions go to rank 0's barrier, armed there for both CTAs (by the weights' producer;
    // bytes that arrive ahead of it are only counted).
    const uint32_t stage_tx = 2 * (GP_A_BYTES + (uint32_t)(a.tn / 2) * GP_BK * 2);
    const uint32_t full0 = map_to_rank(smem_u32(full_bar), 0);
    const bool is_w = warp == 0;
    auto load = [&](unsigned char* st, uint32_t bar, int k, int at) {
      if (!is_w) {
        tma_load_2d_pair(st + GP_A_BYTES, &tm_x, k, at, bar);
      } else if (!Epi::GLU) {
        tma_load_2d_pair(st, &tm_w0, k, at, bar);
      } else if (a.glu_one) {
        tma_load_4d_pair(st, &tm_w0, k, at / 16, bar);
      } else {
#pragma unroll
        for (int g = 0; g < 4; g++) {
          tma_load_2d_pair(st + g * 4096, &tm_w0, k, at + g * 16, bar);
          tma_load_2d_pair(st + g * 4096 + 2048, &tm_w1, k, at + g * 16, bar);
        }
      }
    };
    // weights do not depend on the preceding kernel: the ring's first ones are requested ahead of the dependency wait
    bool waited = !is_w || a.w_late;
    if (waited) pdl_wait();
    int s = 0, round = 0;
    bool ok = true;
    for (PairWork w(a, pair); ok && w.step(a);) {
      const int ft = w.tile / a.tok_tiles, at = is_w ? (ft * 2 + (int)rank) * FEATS : (w.tile - ft * a.tok_tiles) * a.tn + (int)rank * (a.tn / 2);
      for (int kb = w.k0; kb < w.k1; kb++) {
        if (round > 0) {
          if (!waited) { pdl_wait(); waited = true; }
          if (!mbar_wait(&empty_bar[s], (round - 1) & 1)) { atomicCAS(a.err, 0, 1); ok = false; break; }
        }
        if (elect_one()) {
          if (is_w && rank == 0) mbar_expect_tx(&full_bar[s], stage_tx);
          load(tiles + (size_t)s * GP_STAGE_BYTES, full0 + 8 * s, kb * GP_BK, at);
        }
        if (++s == STAGES) { s = 0; round++; }
      }
    }
  } else if (warp == 1 && rank == 0) {
    // ---- MMA issuer of the pair: 4 x (256 x tn x 16) per k-block
    const uint32_t idesc = (1u << 4) | (Epi::BF16 ? (1u << 7) | (1u << 10) : 0u) | ((uint32_t)(a.tn >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
    const uint64_t desc0 = umma_desc(tiles);
    pdl_wait();  // the poll budget starts once the predecessor is done
    int s = 0, round = 0, job = 0;
    bool ok = true;
    for (PairWork w(a, pair); ok && w.step(a); job++) {
      const int buf = job & 1;
      if (job >= 2 && !mbar_wait_cluster(&acc_empty[buf], ((job >> 1) - 1) & 1)) { atomicCAS(a.err, 0, 2); break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem_base + buf * 256;
      for (int kb = w.k0; kb < w.k1; kb++) {
        if (!mbar_wait(&full_bar[s], round & 1)) { atomicCAS(a.err, 0, 2); ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t adesc = desc0 + (uint64_t)(s * (GP_STAGE_BYTES / 16)), bdesc = adesc + GP_A_BYTES / 16;
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < GP_BK / 16; k++) umma_f16_pair(acc, adesc + 2 * k, bdesc + 2 * k, idesc, (kb > w.k0 || k > 0) ? 1u : 0u);
          umma_commit_both(&empty_bar[s]);  // the stage is free in both CTAs
        }
        if (++s == STAGES) { s = 0; round++; }
      }
      if (ok && elect_one()) umma_commit_both(&acc_full[buf]);
    }
  } else if (warp >= 2 && warp < GP_X_WARP) {
    // ---- epilogue: a warp has 32 lanes (its id modulo 4) and every GP_PARTS-th run of 16 columns
    pdl_wait();
    const int q = warp & 3, ew = warp - 2, part = ew >> 2, row = q * 32 + lane, share = a.pairs - 1 - pair;
    int job = 0;
    for (PairWork w(a, pair); w.step(a); job++) {
      const int buf = job & 1;
      if (!mbar_wait(&acc_full[buf], (job >> 1) & 1)) { if (lane == 0) atomicCAS(a.err, 0, 3); break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t t_lane = tmem_base + buf * 256 + ((uint32_t)(q * 32) << 16);
      int parts = 0;  // the tile's other shares, in the slots behind this pair's
      if (w.k1 < a.n_kb && w.k0 == 0) {
        parts = a.split - 1;
        const uint32_t* f = a.flags + ((size_t)(share + 1 + min(lane, parts - 1)) * 2 + rank) * GP_EPI_WARPS + ew;
        uint32_t v = 0;
        for (uint32_t i = 0; i < TC_SPIN_LIMIT && v == 0; i++) asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
        __syncwarp();  // each flag was acquired by one lane, and all lanes read what stands behind it (a vote orders no memory)
        if (__any_sync(0xffffffffu, v == 0)) { if (lane == 0) atomicCAS(a.err, 0, 3); break; }
      }
      const int feat0 = ((w.tile / a.tok_tiles) * 2 + (int)rank) * FEATS, tok0 = (w.tile % a.tok_tiles) * a.tn;
      float4* mine = reinterpret_cast<float4*>(a.slots + ((size_t)share * 2 + rank) * GP_SLOT);
      const float4* theirs = mine + 2 * GP_SLOT / 4;  // the next share's
      auto release = [&] {  // this warp's columns are read: the MMAs may have this half of tensor memory again
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(map_to_rank(smem_u32(&acc_empty[buf]), 0));
      };
      if (part * 16 >= a.tn) release();
      const int fw = feat0 + q * (Epi::GLU ? 16 : 32), feat = fw + (Epi::GLU ? lane & 15 : lane);  // the warp's features, the lane's
      const bool wide = Epi::wide(ea, a, fw);
#pragma unroll 1
      for (int c0 = part * 16; c0 < a.tn; c0 += GP_PARTS * 16) {
        const int tok = tok0 + c0, wt = tok + (lane & 7), wf = fw + (lane & 24);
        // what the columns are added to is on its way while the accumulators come from tensor memory
        uint4 res[2] = {};
        if (Epi::RESIDUAL && wide && w.k0 == 0) {
#pragma unroll
          for (int i = 0; i < 2; i++)
            if (wt + 8 * i < a.M) res[i] = *reinterpret_cast<const uint4*>(Epi::residual(ea, a, wt + 8 * i, wf));
        }
        float r[16];
        float4 v[2][4];
        const int at = c0 * 32 + row;  // [four columns][row] of a slot
#pragma unroll
        for (int p = 0; p < 2; p++)
          if (p < parts) {
#pragma unroll
            for (int j = 0; j < 4; j++) v[p][j] = __ldcg(theirs + (size_t)p * (2 * GP_SLOT / 4) + at + j * 128);
          }
        tmem_ld16(t_lane + c0, r);
        if (c0 + GP_PARTS * 16 >= a.tn) release();
        if (w.k0 > 0) {
#pragma unroll
          for (int j = 0; j < 4; j++) __stcg(mine + at + j * 128, make_float4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]));
          continue;
        }
        auto plus = [&](const float4 (&x)[4]) {
#pragma unroll
          for (int j = 0; j < 4; j++) { r[4 * j] += x[j].x; r[4 * j + 1] += x[j].y; r[4 * j + 2] += x[j].z; r[4 * j + 3] += x[j].w; }
        };
        if (parts > 0) plus(v[0]);  // in order of k
        if (parts > 1) plus(v[1]);
        for (int p = 2; p < parts; p++) {
#pragma unroll
          for (int j = 0; j < 4; j++) v[0][j] = __ldcg(theirs + (size_t)p * (2 * GP_SLOT / 4) + at + j * 128);
          plus(v[0]);
        }
        if (tok >= a.M) continue;
        if constexpr (Epi::GLU) {
          // lanes l and l + 16 have gate and up of a feature: the lower ones finish even columns, the upper ones odd ones
          uint16_t y[8];
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const float other = __shfl_xor_sync(0xffffffffu, lane < 16 ? r[2 * j + 1] : r[2 * j], 16);
            const float first = lane < 16 ? r[2 * j] : other, second = lane < 16 ? other : r[2 * j + 1];
            y[j] = Epi::glu(ea, min(feat, a.N - 1), a.glu_swap ? second : first, a.glu_swap ? first : second);
          }
          const int half = lane >> 4;
          if (wide) {
            uint32_t p[4], o[1][4];
#pragma unroll
            for (int j = 0; j < 4; j++) p[j] = (uint32_t)y[2 * j] | ((uint32_t)y[2 * j + 1] << 16);
            transpose_16bit<4>(p, o, lane);
            const int t = tok + 2 * (lane & 7) + half;
            if (t < a.M) *reinterpret_cast<uint4*>(Epi::out(ea, a, t, fw + (lane & 8))) = make_uint4(o[0][0], o[0][1], o[0][2], o[0][3]);
          } else {
#pragma unroll
            for (int j = 0; j < 8; j++)
              if (feat < a.N && tok + 2 * j + half < a.M) *reinterpret_cast<uint16_t*>(Epi::out(ea, a, tok + 2 * j + half, feat)) = y[j];
          }
        } else if (wide) {
#pragma unroll
          for (int j = 0; j < 16; j++) r[j] = Epi::value(ea, a, feat, tok + j, r[j]);
          if (Epi::f32(ea)) {
            float4 o[4];
            transpose_32bit(r, o, lane);
#pragma unroll
            for (int m = 0; m < 4; m++)
              if (tok + 4 * m + (lane & 3) < a.M) *reinterpret_cast<float4*>(Epi::out32(ea, a, tok + 4 * m + (lane & 3), fw + (lane & 28))) = o[m];
          } else {
            uint32_t p[8], o[2][4];
#pragma unroll
            for (int j = 0; j < 8; j++) p[j] = (uint32_t)Epi::round(r[2 * j]) | ((uint32_t)Epi::round(r[2 * j + 1]) << 16);
            transpose_16bit<8>(p, o, lane);
#pragma unroll
            for (int i = 0; i < 2; i++) {
              if (Epi::RESIDUAL) { o[i][0] = Epi::add(o[i][0], res[i].x); o[i][1] = Epi::add(o[i][1], res[i].y); o[i][2] = Epi::add(o[i][2], res[i].z); o[i][3] = Epi::add(o[i][3], res[i].w); }
              if (wt + 8 * i < a.M) *reinterpret_cast<uint4*>(Epi::out(ea, a, wt + 8 * i, wf)) = make_uint4(o[i][0], o[i][1], o[i][2], o[i][3]);
            }
          }
        } else if (feat < a.N) {
#pragma unroll
          for (int j = 0; j < 16; j++)
            if (tok + j < a.M) Epi::store(ea, a, feat, tok + j, Epi::value(ea, a, feat, tok + j, r[j]));
        }
      }
      if (w.k0 > 0) {
        __syncwarp();
        if (lane == 0) asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(a.flags + ((size_t)share * 2 + rank) * GP_EPI_WARPS + ew), "r"(1u) : "memory");
      }
      if (parts > 0) {
        __syncwarp();
        for (int p = 1 + lane; p <= parts; p += 32) a.flags[((size_t)(share + p) * 2 + rank) * GP_EPI_WARPS + ew] = 0;
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_barrier();  // neither CTA leaves, or gives its tensor memory back, while the other may still use either's
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// Gate and up of up to 256 rows where a CTA to a 128-feature tile gives most of the SMs one, once: the launch is a stream of weights, and
// pairs need a second, half empty round.  us, weights from HBM, a CTA per tile / pairs: 14336 features (112 tiles) of 4096, 33 rows
// 44.3 / 58.4, 100 rows 48.6 / 60.1, 200 rows 61.8 / 68.3, 256 rows 65.3 / 70.0; 11008 (86 tiles) 54.4 / 45.6, 62.5 / 47.0, 58.8 / 53.2, 60.1 / 54.7.
static inline bool cta_per_tile(const jg_dev* dev, int M, int N) {
  const int tiles = (N + 127) / 128;
  return M <= 256 && tiles * 3 > dev->sm_count * 2 && tiles <= dev->sm_count;
}

// Tiles and shares with the smallest estimate, in SM cycles.  Measured at 1B and 8B shapes, 45 to 2048 rows: a k-block takes 300
// (up to 96 rows to a tile), 330 (128), 410 (192) and 530 (256), or as long as its weights need from HBM (9.6 for each pair that
// fetches other weights); a launch and its last tile's stores 4000 + 60 per row; a second share 5000 + 16 per row, each further
// one 400 + 8 per row.  us, 8B shapes, 200 rows, the plans taken / whole 256-row tiles: qkv 17.7 / 26.0, wo 16.2 / 27.5, gate and
// up 56.8 / 59.7, down 35.7 / 82.0.  Cutting whole rounds and their remainder into equal shares gained nothing at 1024 rows and
// more, where the power limit decides (gate and up, 1024 rows: 174 us in whole tiles, 178 in equal shares).
static inline void pair_plan(PairPlan& a, int feat_tiles, int P, bool shares) {
  float best = 0.f;
  for (int tn = 256; tn >= 32; tn -= 32) {
    const int tok = (a.M + tn - 1) / tn, T = tok * feat_tiles, waves = (T + P - 1) / P;
    for (int s = 1; s == 1 || (shares && s <= 4 && s * T <= P && a.n_kb >= 8 * s); s++) {
      const int pairs = s == 1 ? (T < P ? T : P) : s * T;
      const float kb = fmaxf(fmaxf(130.f + 1.57f * (float)tn, 300.f), 9.6f * (float)pairs / (float)tok);
      // the others' accumulators are written while the first share is still at work
      const int ahead = (int)(8.f * (float)tn / kb), head = s == 1 ? a.n_kb : (a.n_kb + (s - 1) * ahead) / s;
      if (s > 1 && a.n_kb - head < 2 * (s - 1)) break;
      float t = (float)(waves * head) * kb + 4000.f + 60.f * (float)tn;
      if (s > 1) t += 5000.f + 16.f * (float)tn + (float)(s - 2) * (400.f + 8.f * (float)tn);
      if (best != 0.f && t >= best) continue;
      best = t;
      a.tn = tn; a.tok_tiles = tok; a.tiles = T; a.pairs = pairs; a.split = s; a.head = head;
    }
  }
}

template <class Epi>
static int launch_pair(jg_dev* dev, const char* name, const void* x, int ldx, const void* w0, const void* w1, int ldw, int M, int N, int K, bool bf16, int w_late,
                       const typename Epi::Args& ea) {
  auto kern = gemm_pair_kernel<Epi>;
  static int max_pairs[8] = {};
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(GP_THREADS);
  cfg.dynamicSmemBytes = GP_SMEM;
  cfg.stream = dev->stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const int slot = dev->ordinal & 7;
  if (max_pairs[slot] == 0) {
    JG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GP_SMEM));
    cfg.gridDim = dim3((unsigned)(dev->sm_count / 2 * 2));
    int n = 0;
    JG_CUDA(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
    max_pairs[slot] = n < 1 ? 1 : (n > dev->sm_count / 2 ? dev->sm_count / 2 : n);
  }
  const int P = max_pairs[slot];
  PairPlan a = {};
  a.M = M; a.N = N; a.n_kb = (K + GP_BK - 1) / GP_BK; a.w_late = w_late; a.err = dev->err_word;
  const bool shares = jg_pair_workspace(dev);
  if (shares) { a.slots = dev->pair_slots; a.flags = dev->pair_flags; }
  constexpr int TILE_FEATS = Epi::GLU ? 128 : 256;
  pair_plan(a, (N + TILE_FEATS - 1) / TILE_FEATS, P, shares);
  CUtensorMap tw0, tw1, tx;
  int rc = JG_OK;
  if (Epi::GLU && N % 16 == 0 && jg_tensor_map_two(&tw0, w0 < w1 ? w0 : w1, w0 < w1 ? w1 : w0, N, K, ldw, bf16)) {
    a.glu_one = 1;
    a.glu_swap = w1 < w0;
  } else {
    rc = jg_tensor_map(&tw0, w0, N, K, ldw, Epi::GLU ? 16 : 128, "weights", 2, bf16);
    if (rc) return rc;
  }
  rc = jg_tensor_map(&tw1, Epi::GLU ? w1 : w0, N, K, ldw, Epi::GLU ? 16 : 128, "weights (second matrix)", 2, bf16);
  if (rc) return rc;
  rc = jg_tensor_map(&tx, x, M, K, ldx, a.tn / 2, "activations (half tile)", 2, bf16);
  if (rc) return rc;
  dev->tc_pending = true;
  cfg.gridDim = dim3(2 * a.pairs);
  if (dev->pdl) {
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  }
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tw0, tw1, tx, a, ea);
  if (e != cudaSuccess) return jg_cuda_fail(e, name, __FILE__, __LINE__);
  return jg_after_launch(dev, name);
}
#endif
