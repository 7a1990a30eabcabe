// Prompt attention on the 5th-generation tensor cores, shared by the models: 128-row tiles of queries against 128-row tiles
// of keys and values, scores and outputs in tensor memory.
//
// The weights are rounded to 16 bits after normalisation, so the row maximum and sum come first: pass 1 walks the keys for
// them, pass 2 walks keys and values for p = round(2^(s - m) / l) and o = p.V.  (That also leaves no running maximum to
// rescale the outputs by.)
//
// A CTA runs two streams of 128 rows, each with four softmax warps (one thread per row) and a score tile of its own in
// tensor memory, so that one stream's exponentials overlap the other's products:
//   SPLIT = false   the streams are two tiles of queries that share every tile of keys and values;
//   SPLIT = true    the streams are the even and the odd key tiles of one tile of queries (launches too small to fill the
//                   machine with pairs): the maxima and sums of the two meet after pass 1, the outputs are added after pass 2.
// Warps 0-3 and 4-7 softmax, 8 producer (TMA, a lane per run of rows), 9 MMA issuer.  Score tile S = Q.K^T: both operands
// K-major in 128-byte swizzled shared memory, 64 columns per block.  P replaces S in tensor memory (16-bit pairs) and is
// the A operand of P.V, whose B operand is the value tile as it lies in memory (rows of keys: MN-major).  The tensor pipe runs a CTA's
// products in order, so the next S of a stream may be issued right behind the P.V that still reads its P.
//
// What bounds it: per 256 rows x 128 keys the exponentials of both passes (65536 at 16 per clock and SM: 2.1 us) against six
// products of 128 x 128 x 128 (2.2 us at the measured tensor peak); operands come from L2.
//
// Every mbarrier wait is bounded; a role that gives up sets the error word and the CTA winds down.
#pragma once
#include "tcgen05.cuh"

#ifdef __CUDACC__
constexpr int FT_ROWS = 128, FT_KV = 128, FT_THREADS = 320, FT_ST = 2;

__device__ __forceinline__ void ft_arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory"); }
__device__ __forceinline__ float ft_ex2(float x) {  // 2^x by the hardware's approximation (2^-22 relative), 0 for -inf
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
        "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]),
      "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
      "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
      : "memory");
}
// B operand tile [k rows][64 columns] per block of 128-byte swizzled rows, N along the columns (MN-major): blocks of 64
// columns `block_bytes` apart, groups of 8 rows 1024 bytes apart
__device__ __forceinline__ uint64_t umma_desc_mn(const void* tile, uint32_t block_bytes) {
  const uint32_t lo = ((smem_u32(tile) & 0x3FFFFu) >> 4) | ((block_bytes >> 4) << 16);
  const uint32_t hi = 64u | (1u << 14) | (2u << 29);
  return (uint64_t)lo | ((uint64_t)hi << 32);
}
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Shared memory of a CTA: query tiles, then the rings of key and value tiles, each 1024-byte aligned.
template <int DK, int DV, bool SPLIT>
struct FtCfg {
  static constexpr int NQ = SPLIT ? 1 : 2;
  static constexpr uint32_t Q_BYTES = FT_ROWS * DK * 2, K_BYTES = FT_KV * DK * 2, V_BYTES = FT_KV * DV * 2;
  static constexpr size_t SMEM = (size_t)NQ * Q_BYTES + FT_ST * (K_BYTES + V_BYTES) + 1024;
};

// P (a model's policy, one object per thread) supplies
//   DK, DV, BF16                    columns of a query / key row and of a value row (multiples of 64, DV 64 or 128)
//   bool begin()                    after the dependency wait: false if there is nothing to do; sets `tiles`
//   int tiles                       key tiles of the CTA
//   void q_row(stream, r, dst)      query row r as DK / 8 pieces of 16 bytes: dst(piece, uint4)
//   void rows(stream, r)            makes r this thread's row, for the three below
//   bool all(j) / bool none(j)      whether tile j is visible to the row entirely / not at all
//   bool sees(j, c)                 whether the row sees column c of tile j
//   float scale2, float extra2()    score scale times log2 e; score (in units of log2) of an entry without a value, or -inf
//   void load_k / load_v(j, dst, bar, lane)   issue the TMA loads of a tile (the whole warp calls them; bytes are expected by the caller)
//   int dead(j)                     rows from here on hold no key (0 .. 128): their values are zeroed
//   void store(stream, r, o, n, c)  columns c .. c + n - 1 of row r's result
template <class P, bool SPLIT>
__device__ __forceinline__ void flash_tc(P& p, int* err) {
  using Cfg = FtCfg<P::DK, P::DV, SPLIT>;
  constexpr int KB = P::DK / 64, VB = P::DV / 64;
  constexpr uint32_t K_BLOCK = FT_KV * 128, Q_BLOCK = FT_ROWS * 128;
  extern __shared__ __align__(1024) unsigned char ft_raw[];
  unsigned char* sQ = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ft_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* sK = sQ + (size_t)Cfg::NQ * Cfg::Q_BYTES;
  unsigned char* sV = sK + (size_t)FT_ST * Cfg::K_BYTES;
  __shared__ __align__(8) uint64_t k_full[FT_ST], k_empty[FT_ST], v_full[FT_ST], v_empty[FT_ST], s_full[2], s_used[2], o_full[2], q_full, v_part;
  __shared__ uint32_t s_tmem;
  __shared__ float s_m[2][FT_ROWS], s_l[2][FT_ROWS];
  const int tid = threadIdx.x, lane = tid & 31, warp = uniform_warp();
  if (tid == 0) {
    for (int i = 0; i < FT_ST; i++) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    for (int i = 0; i < 2; i++) { mbar_init(&s_full[i], 1); mbar_init(&s_used[i], 4); mbar_init(&o_full[i], 1); }
    mbar_init(&q_full, 4 * Cfg::NQ);
    mbar_init(&v_part, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;
  pdl_launch();  // only now: see tcgen05.cuh
  pdl_wait();
  const bool work = p.begin();  // the same for all threads
  const int n = work ? p.tiles : 0;
  auto count = [&](int q) { return SPLIT ? (n + 1 - q) / 2 : n; };  // tiles of a stream

  if (n == 0) {
  } else if (warp == 8) {
    // ---- producer: keys for pass 1, then keys and values
    bool ok = true;
    for (int i = 0; i < 2 * n && ok; i++) {
      const int s = i % FT_ST, j = i < n ? i : i - n;
      if (i >= FT_ST) ok = mbar_wait(&k_empty[s], ((i / FT_ST) - 1) & 1);
      if (!ok) break;
      if (lane == 0) mbar_expect_tx(&k_full[s], Cfg::K_BYTES);
      __syncwarp();
      p.load_k(j, sK + (size_t)s * Cfg::K_BYTES, &k_full[s], lane);
      if (i < n) continue;
      const int t = j % FT_ST, dead = p.dead(j);
      unsigned char* dst = sV + (size_t)t * Cfg::V_BYTES;
      if (j >= FT_ST) ok = mbar_wait(&v_empty[t], ((j / FT_ST) - 1) & 1);
      if (!ok) break;
      uint64_t* bar = dead < FT_KV ? &v_part : &v_full[t];
      if (lane == 0) mbar_expect_tx(bar, Cfg::V_BYTES);
      __syncwarp();
      p.load_v(j, dst, bar, lane);
      if (dead < FT_KV) {  // the last tile: rows nobody wrote may hold anything, and 0 * infinity is not 0
        ok = mbar_wait(&v_part, 0);
        if (!ok) break;
        for (int c = lane; c < (FT_KV - dead) * VB * 8; c += 32) {
          const int r = dead + c / (VB * 8), o = c % (VB * 8);
          *reinterpret_cast<uint4*>(dst + (o >> 3) * K_BLOCK + r * 128 + (o & 7) * 16) = make_uint4(0, 0, 0, 0);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) ft_arrive(&v_full[t]);
      }
    }
    if (!ok && lane == 0) atomicCAS(err, 0, 1);
  } else if (warp == 9) {
    // ---- MMA issuer
    constexpr uint32_t F = P::BF16 ? (1u << 7) | (1u << 10) : 0u;
    constexpr uint32_t id_s = (1u << 4) | F | ((uint32_t)(FT_KV >> 3) << 17) | ((uint32_t)(FT_ROWS >> 4) << 24);
    constexpr uint32_t id_o = (1u << 4) | F | (1u << 16) | ((uint32_t)(P::DV >> 3) << 17) | ((uint32_t)(FT_ROWS >> 4) << 24);
    int made[2] = {0, 0};  // score tiles issued per stream
    bool ok = mbar_wait(&q_full, 0);
    auto qk = [&](int q, int slot) {
      const uint64_t a = umma_desc(sQ + (SPLIT ? 0 : (size_t)q * Cfg::Q_BYTES)), b = umma_desc(sK + (size_t)slot * Cfg::K_BYTES);
      if (elect_one()) {
#pragma unroll
        for (int c = 0; c < KB; c++)
#pragma unroll
          for (int k = 0; k < 4; k++)
            umma_f16(tmem + q * 128, a + c * (Q_BLOCK >> 4) + 2 * k, b + c * (K_BLOCK >> 4) + 2 * k, id_s, (c > 0 || k > 0) ? 1u : 0u);
        umma_commit(&s_full[q]);
      }
      made[q]++;
    };
    auto commit = [&](uint64_t* bar) {
      if (elect_one()) umma_commit(bar);
    };
    auto used = [&](int q) {  // the last score tile of the stream has been read (pass 1) or replaced by weights (pass 2)
      const bool r = mbar_wait(&s_used[q], (made[q] - 1) & 1);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      return r;
    };
    auto keys = [&](int i) {
      const bool r = mbar_wait(&k_full[i % FT_ST], (i / FT_ST) & 1);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      return r;
    };
    for (int j = 0; j < n && ok; j++) {  // pass 1
      ok = keys(j);
      for (int q = SPLIT ? j & 1 : 0; q < (SPLIT ? (j & 1) + 1 : 2) && ok; q++) {
        if (made[q] > 0) ok = used(q);
        if (ok) qk(q, j % FT_ST);
      }
      if (ok) commit(&k_empty[j % FT_ST]);
    }
    auto pv = [&](int q, int slot, bool first) {
      const uint64_t b = umma_desc_mn(sV + (size_t)slot * Cfg::V_BYTES, K_BLOCK);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < FT_KV / 16; k++)  // 16 rows of values = 2048 bytes further
          umma_f16_ts(tmem + 256 + q * 128, tmem + q * 128 + k * 8, b + k * 128, id_o, (!first || k > 0) ? 1u : 0u);
      }
    };
    const int ahead = SPLIT ? 2 : 1;  // tiles whose scores are made before the first product with values
    for (int j = 0; j < ahead && j < n && ok; j++) {
      ok = keys(n + j);
      for (int q = SPLIT ? j : 0; q < (SPLIT ? j + 1 : 2) && ok; q++) {
        ok = made[q] == 0 || used(q);
        if (ok) qk(q, (n + j) % FT_ST);
      }
      if (ok) commit(&k_empty[(n + j) % FT_ST]);
    }
    for (int j = 0; j < n && ok; j++) {  // pass 2
      ok = mbar_wait(&v_full[j % FT_ST], (j / FT_ST) & 1);
      const bool more = j + ahead < n;
      bool have = false;
      for (int q = SPLIT ? j & 1 : 0; q < (SPLIT ? (j & 1) + 1 : 2) && ok; q++) {
        ok = used(q);
        if (!ok) break;
        pv(q, j % FT_ST, SPLIT ? j < 2 : j == 0);
        if (j + ahead >= n) commit(&o_full[q]);
        if (more) {
          if (!have) { ok = keys(n + j + ahead); have = true; }
          if (ok) qk(q, (n + j + ahead) % FT_ST);
        }
      }
      if (!ok) break;
      commit(&v_empty[j % FT_ST]);
      if (more) commit(&k_empty[(n + j + ahead) % FT_ST]);
    }
    if (!ok && lane == 0) atomicCAS(err, 0, 2);
  } else {
    // ---- softmax: thread = row
    const int q = warp >> 2, r = tid & 127, mine = count(q);
    const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16), S = lanes + q * 128, O = lanes + 256 + q * 128;
    bool ok = true;
    if (!SPLIT || q == 0) {
      unsigned char* row = sQ + (SPLIT ? 0 : (size_t)q * Cfg::Q_BYTES) + (r >> 3) * 1024 + (r & 7) * 128;
      p.q_row(q, r, [&](int c, const uint4& v) { *reinterpret_cast<uint4*>(row + (size_t)(c >> 3) * Q_BLOCK + (((c & 7) ^ (r & 7)) << 4)) = v; });
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) ft_arrive(&q_full);
    }
    p.rows(SPLIT ? 0 : q, r);
    float v[FT_KV];
    auto scores = [&](int i) {  // the stream's i-th score tile into registers
      ok = mbar_wait(&s_full[q], i & 1);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c = 0; c < FT_KV; c += 32) tmem_ld32(S + c, v + c);
      tmem_ld_wait();
    };
    auto release = [&]() {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) ft_arrive(&s_used[q]);
    };
    auto hide = [&](int j) {  // scores of keys the row does not see
      if (__all_sync(0xffffffffu, p.all(j))) return;
#pragma unroll
      for (int c = 0; c < FT_KV; c++) v[c] = p.sees(j, c) ? v[c] : -INFINITY;
    };
    const float sc = p.scale2;
    float m = -INFINITY, l = 0.f;  // largest score; sum of 2^((s - m) sc)
    for (int i = 0; i < mine; i++) {
      const int j = SPLIT ? 2 * i + q : i;
      scores(i);
      if (!ok) break;
      release();
      hide(j);
      float t0 = m, t1 = m, t2 = m, t3 = m;
#pragma unroll
      for (int c = 0; c < FT_KV; c += 4) { t0 = fmaxf(t0, v[c]); t1 = fmaxf(t1, v[c + 1]); t2 = fmaxf(t2, v[c + 2]); t3 = fmaxf(t3, v[c + 3]); }
      const float top = fmaxf(fmaxf(t0, t1), fmaxf(t2, t3)), base = top == -INFINITY ? 0.f : top * sc;
      l *= ft_ex2(m == -INFINITY ? -INFINITY : m * sc - base);
      m = top;
      float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
      for (int c = 0; c < FT_KV; c += 4) {
        a0 += ft_ex2(fmaf(v[c], sc, -base));
        a1 += ft_ex2(fmaf(v[c + 1], sc, -base));
        a2 += ft_ex2(fmaf(v[c + 2], sc, -base));
        a3 += ft_ex2(fmaf(v[c + 3], sc, -base));
      }
      l += (a0 + a1) + (a2 + a3);
    }
    float base = m == -INFINITY ? -INFINITY : m * sc;
    if (SPLIT) {
      s_m[q][r] = base;
      s_l[q][r] = l;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      const float other = s_m[q ^ 1][r], both = fmaxf(base, other), zero = both == -INFINITY ? 0.f : both;
      l = l * ft_ex2(base - zero) + s_l[q ^ 1][r] * ft_ex2(other - zero);
      base = both;
    }
    const float ex = p.extra2();
    if (ex != -INFINITY) {  // an entry that takes weight and has no value
      const float both = fmaxf(base, ex);
      l = l * ft_ex2(base - both) + ft_ex2(ex - both);
      base = both;
    }
    if (base == -INFINITY) base = 0.f;
    const float rl = __fdiv_rn(1.0f, l);
    for (int i = 0; i < mine && ok; i++) {
      const int j = SPLIT ? 2 * i + q : i;
      scores(mine + i);
      if (!ok) break;
      hide(j);
#pragma unroll
      for (int c = 0; c < FT_KV; c += 64) {
        uint32_t w[32];
#pragma unroll
        for (int k = 0; k < 32; k++) {
          const float x = ft_ex2(fmaf(v[c + 2 * k], sc, -base)) * rl, y = ft_ex2(fmaf(v[c + 2 * k + 1], sc, -base)) * rl;
          if (P::BF16) asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w[k]) : "f"(y), "f"(x));
          else asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(w[k]) : "f"(y), "f"(x));
        }
        tmem_st32(S + c / 2, w);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      release();
    }
    if (ok && mine > 0) {
      ok = mbar_wait(&o_full[q], 0);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    if (!ok && lane == 0) atomicCAS(err, 0, 3);
    if (SPLIT) {
      // the odd tiles' outputs meet the even ones' through shared memory (all products are done: the rings are free)
      float* red = reinterpret_cast<float*>(sK);
      const bool two = n > 1;
      if (q == 1 && ok && two) {
#pragma unroll
        for (int c = 0; c < P::DV; c += 32) {
          tmem_ld32(O + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 32; k++) red[(c + k) * FT_ROWS + r] = v[k];
        }
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (q == 0 && ok) {
#pragma unroll 1
        for (int c = 0; c < P::DV; c += 32) {
          tmem_ld32(O + c, v);
          tmem_ld_wait();
          if (two)
#pragma unroll
            for (int k = 0; k < 32; k++) v[k] += red[(c + k) * FT_ROWS + r];
          p.store(0, r, v, c);
        }
      }
    } else if (ok) {
#pragma unroll 1
      for (int c = 0; c < P::DV; c += 32) {
        tmem_ld32(O + c, v);
        tmem_ld_wait();
        p.store(q, r, v, c);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 9) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}
#endif
