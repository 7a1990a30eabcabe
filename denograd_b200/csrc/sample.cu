// Stochastic `sample` (jsgrad/models/llama.ts:131-185) as one kernel per call: alpha penalties, NaN masking, softmax of
// logits / temperature, k rounds of (max, lowest index of the max, remove it), the approximate top-p cut on those k,
// and the multinomial draw (jsgrad/tensor.ts:1164-1172) from a uniform sample the caller supplies.
//
// The integer result depends on float32 sums (the softmax normaliser, the mass outside the top k, the cumulative
// sums of the draw), and a float32 sum depends on the order of its additions.  The kernel therefore adds in exactly
// the order the reference's kernels do — ascending within a reduction, reductions of 32768 elements and more first
// split into the largest number of equal contiguous chunks between 8 and 256 (UOp.r, jsgrad/ops.ts:433-455), cumulative
// sums beyond 512 elements in blocks of 256 behind a front pad (Tensor._split_cumalu, jsgrad/tensor.ts:2629-2643) — so
// that the chosen token is the reference's bit for bit, not merely "within rounding".  The chunks / blocks are what
// runs in parallel: one thread per chunk.
//
// One thread-block cluster serves one row of logits: each CTA keeps a contiguous slice of the distribution in shared
// memory (float32) and the head of the next CTA's slice behind it, so that the chunk and the block that straddle the
// border are added up where they begin, from local memory; the cluster meets at hardware barriers; no global scratch.
//
// What bounds a call is the length of the chains of dependent additions (V / 256 for a sum, 256 per block of a cumulative
// sum, 256 and V / 256 for the totals), at one add per 4 cycles, and the cluster barriers.  The chains therefore run from
// local shared memory with the loads of several steps in flight, on every CTA of the cluster at once, and the slice is
// laid out with one word of padding per 256 (`slot`), which puts chains that start a block apart on different banks.
// 128256 logits, one row, k = 0: 320 us with the chains of CTA 0 reading the peers' slices element by element, 23 us
// now; k = 40: 274 and 78 us.
#include <math.h>

#include <cooperative_groups.h>

#include "common.cuh"
#include "transcendental.cuh"

namespace cg = cooperative_groups;

constexpr int SMP_THREADS = 1024;
constexpr int SMP_MAX_CLUSTER = 8;
constexpr int SMP_MAXK = 512;      // beyond 512 the reference's cumulative sum changes shape; nobody samples from more
constexpr int SMP_MAX_BLOCKS = 2048;  // 256-element blocks of the k = 0 draw: vocabularies up to 524288

__device__ __forceinline__ float logit_f32(__half v) { return __half2float(v); }
__device__ __forceinline__ float logit_f32(float v) { return v; }

struct SampleArgs {
  const void* logits;    // [B][V] fp16, widened to fp32 as Transformer.forward does (jsgrad/models/llama.ts:210), or fp32
  const float* u;        // [B] uniform samples in [0, 1)
  int32_t* counter;      // [B][V] alpha counters, or null
  int32_t* tokens;       // [B]
  int V, k, per, ext;    // per: elements of the distribution held by one CTA; ext: the same with the head of the next slice
  int div, len;          // reductions over V: `div` chunks of `len` (div = 0: one sequential pass)
  float inv_temp, thr, af, ap;
};

// Word of a slice that holds its element i: chains that start 256 elements apart begin on neighbouring banks.
__host__ __device__ __forceinline__ int smp_slot(int i) { return i + (i >> 8); }

// Part of a row's distribution as one CTA sees it: its own slice and `ext - per` elements of the next one in local memory,
// anything beyond through distributed shared memory.
struct SliceView {
  float* const* base;  // the CTAs' slices
  const float* local;
  int per, ext, j0;
  __device__ __forceinline__ float load(int j) const {
    const int i = j - j0;
    if (i >= 0 && i < ext) return local[smp_slot(i)];
    return base[j / per][smp_slot(j % per)];
  }
  // s + t(j) + t(j + 1) + ... + t(j + n - 1), added in that order; t(x) = x * scale rounded once (scale 1: x)
  __device__ __forceinline__ float add_up(float s, int j, int n, float scale) const {
    const int i = j - j0;
    return i >= 0 && i + n <= ext ? chain(s, n, scale, [&](int k) { return local[smp_slot(i + k)]; })  // no test per element
                                  : chain(s, n, scale, [&](int k) { return load(j + k); });
  }
  template <typename F>
  __device__ __forceinline__ static float chain(float s, int n, float scale, F at) {
    constexpr int U = 16;
    int k = 0;
#pragma unroll 1
    for (; k + U <= n; k += U) {
      float v[U];
#pragma unroll
      for (int q = 0; q < U; q++) v[q] = at(k + q);
#pragma unroll
      for (int q = 0; q < U; q++) s = __fadd_rn(s, __fmul_rn(v[q], scale));
    }
    for (; k < n; k++) s = __fadd_rn(s, __fmul_rn(at(k), scale));
    return s;
  }
};

// s + p[0] + ... + p[n - 1] in that order (p in local shared memory); `prefix`, where given, receives the sum before each entry
__device__ __forceinline__ float chain_sum(float s, const float* p, int n, float* prefix) {
  constexpr int U = 16;
  int k = 0;
  for (; k + U <= n; k += U) {
    float v[U];
#pragma unroll
    for (int q = 0; q < U; q++) v[q] = p[k + q];
#pragma unroll
    for (int q = 0; q < U; q++) {
      if (prefix) prefix[k + q] = s;
      s = __fadd_rn(s, v[q]);
    }
  }
  for (; k < n; k++) {
    if (prefix) prefix[k] = s;
    s = __fadd_rn(s, p[k]);
  }
  return s;
}

template <typename LT>
__global__ void __launch_bounds__(SMP_THREADS, 1) sample_kernel(const SampleArgs a) {
  extern __shared__ __align__(16) float tbuf[];  // this CTA's slice and the head of the next: y, then e, then (k > 0) t
  __shared__ float s_red[32];
  __shared__ unsigned long long s_red64[32];
  __shared__ float s_cmax[SMP_MAX_CLUSTER];
  __shared__ unsigned long long s_key[2][SMP_MAX_CLUSTER];
  __shared__ float s_bcast;
  __shared__ float s_part[2][256];
  __shared__ float s_out[SMP_MAXK];
  __shared__ int s_idx[SMP_MAXK];
  __shared__ float s_tot[SMP_MAX_BLOCKS], s_base[SMP_MAX_BLOCKS];
  __shared__ float s_blk[256];
  __shared__ int s_count;
  __shared__ float* s_slices[SMP_MAX_CLUSTER];
  cg::cluster_group cluster = cg::this_cluster();
  const int cr = (int)cluster.block_rank(), cs = (int)cluster.num_blocks();
  const int b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int V = a.V, per = a.per;
  const int j0 = cr * per, j1 = min(V, j0 + per), nloc = max(j1 - j0, 0);
  const int next = max(min(V, j0 + a.ext) - j0, 0);  // elements in local memory, the next slice's head included
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  pdl_launch();
  pdl_wait();
  if (tid < cs) s_slices[tid] = cluster.map_shared_rank(tbuf, tid);
  if (tid == 0) s_count = 0;
  const float log2e = 1.4426950408889634f;  // (float)(1 / Math.log(2))
  const SliceView row = {s_slices, tbuf, per, next, j0};

  // ---- y = (logit - penalty) * (1 / temperature), NaN -> -inf; maximum over the row
  float lmax = -INFINITY;
#pragma unroll 4
  for (int i = tid; i < next; i += SMP_THREADS) {
    float x = logit_f32(reinterpret_cast<const LT*>(a.logits)[(size_t)b * V + j0 + i]);
    if (a.counter != nullptr) {
      const int c = a.counter[(size_t)b * V + j0 + i];
      const float pen = __fadd_rn(__fmul_rn((float)c, a.af), __fmul_rn(c >= 0 ? 1.0f : 0.0f, a.ap));
      x = __fsub_rn(x, pen);
    }
    if (x != x) x = -INFINITY;
    x = __fmul_rn(x, a.inv_temp);
    tbuf[smp_slot(i)] = x;
    lmax = fmaxf(lmax, x);
  }
  lmax = warp_max(lmax);
  if (lane == 0) s_red[warp] = lmax;
  __syncthreads();
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");  // the peers run: their shared memory may be written
  if (warp == 0) {
    const float m = warp_max(s_red[lane]);
    if (lane < cs) *cluster.map_shared_rank(&s_cmax[cr], lane) = m;
  }
  cluster.sync();
  float M = s_cmax[0];
  for (int c = 1; c < cs; c++) M = fmaxf(M, s_cmax[c]);

  // ---- e = exp2((y - M) / ln 2) with the polynomial exp2 (Tensor.exp, jsgrad/tensor.ts:2872-2875)
#pragma unroll 4
  for (int i = tid; i < next; i += SMP_THREADS) tbuf[smp_slot(i)] = jg_xexp2_f32(__fmul_rn(__fsub_rn(tbuf[smp_slot(i)], M), log2e));
  __syncthreads();

  // Sum over the whole row in the reference's order.  Every CTA adds up the chunks that begin in its slice and hands the
  // sums to all CTAs, each of which adds them up.  All CTAs call it; `slot` 0 or 1.
  auto row_sum = [&](int slot) -> float {
    if (a.div == 0) {  // one chain: CTA 0 walks all slices
      cluster.sync();
      if (cr == 0 && tid == 0) {
        const float s = row.add_up(0.f, 0, V, 1.0f);
        for (int c = 0; c < cs; c++) *cluster.map_shared_rank(&s_part[slot][0], c) = s;
      }
      cluster.sync();
      return s_part[slot][0];
    }
    const int c0 = (j0 + a.len - 1) / a.len, c1 = min((j1 + a.len - 1) / a.len, a.div);
    if (a.len > a.ext - per) cluster.sync();  // a chunk may reach into the next slice's own memory
    if (tid < c1 - c0) {
      const float s = row.add_up(0.f, (c0 + tid) * a.len, a.len, 1.0f);
      for (int c = 0; c < cs; c++) *cluster.map_shared_rank(&s_part[slot][c0 + tid], c) = s;
    }
    cluster.sync();
    if (tid == 0) s_bcast = chain_sum(0.f, s_part[slot], a.div, nullptr);
    __syncthreads();
    return s_bcast;
  };

  const float rinv = __fdiv_rn(1.0f, row_sum(0));

  int token = 0;
  if (a.k > 0) {
    for (int i = tid; i < next; i += SMP_THREADS) tbuf[smp_slot(i)] = __fmul_rn(tbuf[smp_slot(i)], rinv);  // t = e * (1 / sum)
    __syncthreads();
    // ---- k rounds: the largest probability and, among equals, its lowest index (the reference's
    //      t.eq(max) * arange(n-1 .. 0) trick); the winner is zeroed.  Probabilities are >= +0, so their bit patterns
    //      order like the values: the key (bits << 32 | ~index) finds both with one unsigned maximum.  A thread keeps the
    //      best key of its elements and looks them over again only when it was its own that won.
    auto scan = [&]() {
      unsigned long long best = 0ull;
#pragma unroll 4
      for (int i = tid; i < nloc; i += SMP_THREADS) {
        const unsigned long long key = ((unsigned long long)__float_as_uint(tbuf[smp_slot(i)]) << 32) | (unsigned long long)(0xFFFFFFFFu - (uint32_t)(j0 + i));
        best = key > best ? key : best;
      }
      return best;
    };
    unsigned long long mine = scan();
    for (int it = 0; it < a.k; it++) {
      unsigned long long best = mine;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
        best = other > best ? other : best;
      }
      if (lane == 0) s_red64[warp] = best;
      __syncthreads();
      if (warp == 0) {
        best = s_red64[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
          best = other > best ? other : best;
        }
        if (lane < cs) *cluster.map_shared_rank(&s_key[it & 1][cr], lane) = best;
      }
      cluster.sync();
      unsigned long long win = s_key[it & 1][0];
      for (int c = 1; c < cs; c++) win = s_key[it & 1][c] > win ? s_key[it & 1][c] : win;
      const int idx = (int)(0xFFFFFFFFu - (uint32_t)(win & 0xFFFFFFFFull)), i = idx - j0;
      if (tid == 0) {
        s_out[it] = __uint_as_float((uint32_t)(win >> 32));
        s_idx[it] = idx;
      }
      if (i >= 0 && i < next && i % SMP_THREADS == tid) {
        tbuf[smp_slot(i)] = 0.f;
        mine = scan();
      }
    }
    __syncthreads();
    const float rest = row_sum(1);
    if (cr == 0 && tid == 0) {
      // approximate top-p: tail[i] = out[k-1] + ... + out[i] (added in that order) + rest; entry i survives while
      // tail[i] >= 1 - p.  Then the draw: cumulative sums of the survivors, scaled by 1 / total, counted against u.
      const int k = a.k;
      float run = 0.f;
      for (int i = k - 1; i >= 0; i--) {
        run = __fadd_rn(run, s_out[i]);
        const bool keep = __fadd_rn(run, rest) >= a.thr;
        if (!keep) { s_out[i] = 0.f; s_idx[i] = 0; }
      }
      float cw = 0.f;
      for (int i = 0; i < k; i++) cw = __fadd_rn(cw, s_out[i]);
      const float r = __fdiv_rn(1.0f, cw);
      const float u = a.u[b];
      int cnt = 0;
      float acc = 0.f;
      for (int i = 0; i < k; i++) {
        acc = __fadd_rn(acc, s_out[i]);
        cnt += (u >= __fmul_rn(acc, r)) ? 1 : 0;
      }
      token = cnt < k ? s_idx[cnt] : 0;  // an index past the end gathers nothing
    }
  } else {
    // ---- draw from the whole distribution: cumulative sums in blocks of 256 behind a front pad (one block up to 512
    //      elements), block totals added on top, everything scaled by 1 / last, entries not above u counted.  Rounded sums
    //      of terms >= 0 never decrease, and the value at a block's end is the base of the next, so the count is all blocks
    //      whose end is not above u and what the next block holds: only that one is walked entry by entry.  (Where an entry is NaN the
    //      normaliser is, and no comparison holds.)
    const bool blocked = V > 512;
    const int np = (V + 255) / 256 * 256, pad = blocked ? np - V : 0, size = blocked ? 256 : V, nb = blocked ? np / 256 : 1;
    const int b0 = cr == 0 ? 0 : (j0 + pad + size - 1) / size, b1 = min((j1 + pad + size - 1) / size, nb);
    if (size > a.ext - per) cluster.sync();
    for (int blk = b0 + tid; blk < b1; blk += SMP_THREADS) {
      const int first = max(blk * size - pad, 0), n = (blk + 1) * size - pad - first;
      *cluster.map_shared_rank(&s_tot[blk], 0) = row.add_up(0.f, first, n, rinv);  // t = e * (1 / sum)
    }
    cluster.sync();
    if (cr == 0) {
      if (tid == 0) s_bcast = chain_sum(0.f, s_tot, nb, s_base);
      __syncthreads();
      const float r = __fdiv_rn(1.0f, s_bcast), u = a.u[b];
      for (int blk = tid; blk < nb; blk += SMP_THREADS)
        if (u >= __fmul_rn(__fadd_rn(s_tot[blk], s_base[blk]), r)) atomicAdd(&s_count, 1);
      __syncthreads();
      const int full = s_count;
      if (full == nb) token = V;
      else {
        const int first = max(full * size - pad, 0), n = (full + 1) * size - pad - first;
        float s = 0.f;
        int cnt = 0;
        for (int k0 = 0; k0 < n; k0 += 256) {
          __syncthreads();
          if (tid < 256 && k0 + tid < n) s_blk[tid] = __fmul_rn(row.load(first + k0 + tid), rinv);
          __syncthreads();
          if (tid == 0) {
            const int m = min(256, n - k0);
#pragma unroll 16
            for (int k = 0; k < m; k++) {
              s = __fadd_rn(s, s_blk[k]);
              cnt += (u >= __fmul_rn(blocked ? __fadd_rn(s, s_base[full]) : s, r)) ? 1 : 0;
            }
          }
        }
        token = first + cnt;
      }
    }
  }
  if (cr == 0 && tid == 0) {
    a.tokens[b] = token;
    if (a.counter != nullptr && token >= 0 && token < V) a.counter[(size_t)b * V + token] += 1;
  }
  cluster.sync();  // nobody leaves while a peer may still read its shared memory
}

// Tokens for B rows of fp16 logits [B][V] (device): tokens_out int32 [B]; u float32 [B], one uniform sample in [0, 1)
// per row (what Tensor.rand hands to multinomial); alpha_counter int32 [B][V] or 0.  temp must be >= 1e-6 (below
// that `sample` is an argmax: jg_argmax).  The reference applies `sample` to one flattened row (jsgrad/models/llama.ts:
// 132,212); rows here are independent.
template <typename LT>
static int run_sample(jg_dev* dev, uint64_t tokens_out, uint64_t logits, uint64_t u, uint64_t alpha_counter, int32_t B,
                      int32_t V, float temp, int32_t k, float p, float af, float ap) {
  JG_ENTER(dev);
  JG_REQUIRE(B > 0 && B <= 65535 && V > 0, "sample: bad shape B=%d V=%d", B, V);
  JG_REQUIRE(p >= 0.f && p <= 1.f, "sample: p must be between 0 and 1");
  JG_REQUIRE(k >= 0 && k <= V, "sample: k must be between 0 and numel");
  JG_REQUIRE(k <= SMP_MAXK, "sample: k=%d above %d is not implemented", k, SMP_MAXK);
  JG_REQUIRE(temp >= 1e-6f, "sample: temperature below 1e-6 selects argmax (jg_argmax)");
  JG_REQUIRE(jg_aligned(tokens_out, 4) && jg_aligned(logits, sizeof(LT)) && jg_aligned(u, 4) && (alpha_counter == 0 || jg_aligned(alpha_counter, 4)),
             "sample: null or misaligned pointer");
  JG_REQUIRE((V + 255) / 256 <= SMP_MAX_BLOCKS, "sample: a vocabulary of %d exceeds %d", V, SMP_MAX_BLOCKS * 256);
  SampleArgs a = {};
  a.logits = (const void*)logits; a.u = (const float*)u; a.tokens = (int32_t*)tokens_out;
  a.counter = (af != 0.f || ap != 0.f) ? (int32_t*)alpha_counter : nullptr;
  JG_REQUIRE(!(af != 0.f || ap != 0.f) || alpha_counter != 0, "sample: alpha penalties need the counter buffer");
  a.V = V; a.k = k; a.af = af; a.ap = ap;
  a.inv_temp = (float)(1.0 / (double)temp);
  a.thr = (float)(1.0 - (double)p);
  if (V >= 32768)
    for (int c = 256; c >= 8; c--)
      if (V % c == 0) { a.div = c; a.len = V / c; break; }
  // cluster of 8 (fewer for small rows); every CTA's slice must fit next to the static tables
  int cs = SMP_MAX_CLUSTER;
  while (cs > 1 && V / cs < 2048) cs >>= 1;
  a.per = (V + cs - 1) / cs;
  // the head of the next slice is kept where a chunk is short enough for it (a vocabulary with a divisor near 256); longer
  // chunks, found with odd vocabularies, read the rest through distributed shared memory
  a.ext = cs > 1 ? a.per + (a.len > 256 && a.len <= 2048 ? a.len : 256) : a.per;
  // a slice takes as much as it ever did (its values, 40 KB left over); its padding and the neighbour's head come out of those 40 KB,
  // of which the static tables take 25
  const size_t optin = dev->prop.sharedMemPerBlockOptin, limit = optin - 28 * 1024, smem = (size_t)(smp_slot(a.ext) + 1) * sizeof(float);
  if ((size_t)a.per * sizeof(float) > optin - 40 * 1024 || smem > limit) {
    jg_set_error("sample: %d values per CTA need %zu B of shared memory (limit %zu)", a.per, smem, limit);
    return JG_ENOTSUP;
  }
  static size_t smem_set[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const int slot = dev->ordinal & 7;
  if (smem > 8 * 1024 && smem > smem_set[slot]) {
    JG_CUDA(cudaFuncSetAttribute(sample_kernel<LT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit));
    smem_set[slot] = limit;
  }
  return jg_launch_cluster(dev, "sample", sample_kernel<LT>, dim3((unsigned)cs, (unsigned)B), dim3(SMP_THREADS), smem, cs, a);
}

JG_API int jg_sample(jg_dev* dev, uint64_t tokens_out, uint64_t logits, uint64_t u, uint64_t alpha_counter, int32_t B,
                     int32_t V, float temp, int32_t k, float p, float af, float ap) {
  return run_sample<__half>(dev, tokens_out, logits, u, alpha_counter, B, V, temp, k, p, af, ap);
}
JG_API int jg_sample_f32(jg_dev* dev, uint64_t tokens_out, uint64_t logits, uint64_t u, uint64_t alpha_counter, int32_t B,
                         int32_t V, float temp, int32_t k, float p, float af, float ap) {
  return run_sample<float>(dev, tokens_out, logits, u, alpha_counter, B, V, temp, k, p, af, ap);
}
