// Projection of a few activation rows: y = epilogue(x W^T), the weights read once from HBM.
//
// Bound by the weight stream and, for small matrices, by a launch's fixed latencies, so the kernel is built around the stream.  One
// CTA per SM has an equal run of outputs (whole weight rows, N / SMs of them, not rounded to a tile) and walks K once for all of them:
// a producer warp keeps a ring of stages in flight, each a TMA box of the run's rows x a few 128-byte runs of K (one instruction per
// matrix; a bulk copy per row piece moved 512 bytes in 75 cycles and no more) with the same k of the activations beside it.  Up to 16
// warps share a stage: warp (tile, k) has one 128-byte run of one or two 16-row tiles, whose 16-byte chunks in shared memory *are* A
// fragments of mma.sync.m16n8k16 (the k order inside a run may be permuted as long as the activations' is, too).  int8 has the sums of
// gemm_small.cu to the bit: a warp has one of its K slices, and a stage's box one or two runs of each slice.  The warps run free
// of each other through the ring (an mbarrier per stage in each direction) and meet once, at the end, to add the sums of the warps
// that share a tile, in a fixed order.  The first stages' weights are requested before the dependency wait: up to 28 MB in all, most
// small matrices whole.  Activations travel with each stage.
//
// us per launch, weights from HBM, back to back, the kernels used before / this one: 8B int8, 8 rows qkv 9.4 / 7.9, wo 7.6 / 6.7, gate
// and up 24.8 / 26.3 (between its neighbours in a step it gains, see skinny.cu), down 19.8 / 13.9, logits 97.8 / 90.4; 16 rows 14.4 /
// 9.7, 11.5 / 7.7, -, 30.1 / 18.5; 8B NF4, one row 8.9 / 9.0, 5.9 / 7.1, 28.3 / 24.6, 14.5 / 13.7 (in a step all four gain: 2.56 / 2.42
// ms a token); 1B fp16, 8 rows 6.2 / 5.5, 5.4 / 5.1, 15.2 / 13.6, 11.2 / 8.4; 8B fp16 logits, 8 rows 163.9 / 155.9 (6.7 TB/s).  The
// stream alone would take 21 us for the 8B int8 gate and up: what is left there is unpacking, at 40 % of the issue slots, and requests
// of 128 bytes a row where slices lie apart (24.3 us with whole rows of a stage); a launch costs about 4 us beyond its stream.
//
// Weights: fp16, bf16, int8 (half(q) * scale of the row, one rounding) or NF4 (half(code * scale of the block) out of a table of byte
// -> two codes, one copy of it per lane and so per bank).  Products are exact, sums fp32.
//
// Every mbarrier wait is bounded: a warp whose wait gives up records it and goes on without waiting (the results are void, the host
// reports JG_ETIMEDOUT at the next synchronisation); the producer stops requesting and lets the copies in flight land.
#pragma once
#include "nf4.cuh"
#include "quant.cuh"
#include "skinny_plan.h"
#include "tcgen05.cuh"

struct SkArgs {
  const __half *s0, *s1;  // int8: a scale per row
  int* err;
  int M, N;
  int tr, sp;             // outputs of a pass; NF4: bytes of a row's scales in a stage
  int tiles, ks, units;   // 16-row tiles of a pass, warps that share one along K, runs of a warp in a stage
  int runs, pieces, slice;  // runs of a stage, stages of a pass; W8: runs of a slice
  int stages, stage_bytes, block_shift;
  int w_late;             // the weights were written by a launch that may still be running
};

constexpr int SK_THREADS = 32 * (SK_WARPS + 1);
// NT tiles of 8 activation rows x TP tiles of 16 weight rows to a warp
template <int TYPE, int NT, int TP> struct SkCfg {
  static constexpr int CPL = sk_runs_x(TYPE);
  static constexpr int LUT = TYPE == SK_NF4 ? SK_TABLE : 0;
  static constexpr int PERW = TP * NT * 4;  // sums of a lane
  static constexpr int PART = sk_part(NT, TP);
  static constexpr int EPT = 4 * NT;        // sums a thread finishes at most
};

#ifdef __CUDACC__
template <bool BF>
__device__ __forceinline__ void sk_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if (BF)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 sk_lds(uint32_t p) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(p) : "memory");
  return v;
}
__device__ __forceinline__ __half sk_lds_half(uint32_t p) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(p) : "memory");
  return __ushort_as_half(v);
}

// What this CTA alone will read, asked into L2.
__device__ __forceinline__ void prefetch_run(const void* p, int bytes) {
  for (int i = threadIdx.x * 128; i < bytes + 127; i += SK_WARPS * 32 * 128) prefetch_l2((const char*)p + min(i, bytes - 1));
}

// E: what happens to a finished sum.  E::Pre is what it needs from global memory.
template <int TYPE, int NT, int TP, bool GLU, class E>
__global__ void __launch_bounds__(SK_THREADS, 1)
    skinny_kernel(const __grid_constant__ CUtensorMap tm_w0, const __grid_constant__ CUtensorMap tm_w1, const __grid_constant__ CUtensorMap tm_x,
                  const __grid_constant__ CUtensorMap tm_s0, const __grid_constant__ CUtensorMap tm_s1, const SkArgs a, const typename E::Args e) {
  using C = SkCfg<TYPE, NT, TP>;
  constexpr int CPL = C::CPL, NW = GLU ? 2 : 1, PERW = C::PERW, EPT = C::EPT;
  constexpr bool W8 = TYPE == SK_W8;
  extern __shared__ __align__(1024) unsigned char sk_raw[];
  // [sums | table | ring]
  const uint32_t raw = smem_u32(sk_raw), lut = C::LUT ? (raw + C::PART + C::LUT - 1) & ~(uint32_t)(C::LUT - 1) : 0;
  float* part = reinterpret_cast<float*>(sk_raw);
  unsigned char* ring = sk_raw + ((C::LUT ? lut + C::LUT : (raw + C::PART + 1023) & ~1023u) - raw);
  __shared__ __align__(8) uint64_t full[SK_MAX_STAGES], empty[SK_MAX_STAGES];
  const int warp = uniform_warp(), lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int S = a.stages, M = a.M, tr = a.tr, KS = a.ks, U = a.units, RUNS = a.runs;
  const int n0 = (int)((long long)blockIdx.x * a.N / gridDim.x), cnt = (int)((long long)(blockIdx.x + 1) * a.N / gridDim.x) - n0;
  const int passes = (cnt + tr - 1) / tr, np = a.pieces, total = passes * np;
  const int w_al = sk_align(RUNS * tr * 128, 1024), x_al = sk_align(RUNS * CPL * M * 128, 1024), s_al = sk_align(tr * a.sp, 128);
  pdl_launch();

  if (warp == SK_WARPS) {
    // ---- producer
    if (lane == 0) {
      for (int s = 0; s < S; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], (a.tiles + TP - 1) / TP * KS); }
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    // W8: a stage has the next U runs of every slice: run of the slice, first slice
    auto slice_at = [&](int piece) {
      const int per = a.slice / U;
      return make_int2(piece % per * U, piece / per * KS);
    };
    auto load_w = [&](int i) {
      const int pass = i / np, piece = i - pass * np, s = i % S, row = n0 + pass * tr;
      unsigned char* st = ring + s * a.stage_bytes;
      mbar_expect_tx(&full[s], NW * tr * (RUNS * 128 + a.sp) + M * CPL * RUNS * 128);
      if (W8) {
        const int2 at = slice_at(piece);
        tma_load_4d(st, &tm_w0, 0, row, at.x, at.y, &full[s]);
        if (GLU) tma_load_4d(st + w_al, &tm_w1, 0, row, at.x, at.y, &full[s]);
        return;
      }
      tma_load_3d(st, &tm_w0, 0, row, piece * RUNS, &full[s]);
      if (GLU) tma_load_3d(st + w_al, &tm_w1, 0, row, piece * RUNS, &full[s]);
      if (TYPE == SK_NF4) {
        tma_load_2d(st + NW * w_al + x_al, &tm_s0, piece * (a.sp / 2), row, &full[s]);
        if (GLU) tma_load_2d(st + NW * w_al + x_al + s_al, &tm_s1, piece * (a.sp / 2), row, &full[s]);
      }
    };
    auto load_x = [&](int i) {
      unsigned char* st = ring + (i % S) * a.stage_bytes + NW * w_al;
      if (W8) {
        const int2 at = slice_at(i % np);
        tma_load_4d(st, &tm_x, 0, 0, at.x * CPL, at.y, &full[i % S]);
      } else {
        tma_load_3d(st, &tm_x, 0, 0, i % np * (RUNS * CPL), &full[i % S]);
      }
    };
    const int pre = min(S, total);
    if (a.w_late) pdl_wait();
    if (elect_one())
      for (int i = 0; i < pre; i++) load_w(i);
    __syncthreads();  // the barriers, and NF4's table
    pdl_wait();       // the rows come from the launch before
    if (elect_one())
      for (int i = 0; i < pre; i++) load_x(i);
    bool ok = true;
    int done = pre;
    for (int i = pre; i < total && ok; i++) {
      ok = mbar_wait(&empty[i % S], ((i / S) - 1) & 1);
      if (!ok) break;
      if (elect_one()) { load_w(i); load_x(i); }
      done++;
    }
    // copies in flight land before the CTA may go (the other warps have waited for them unless one gave up)
    for (int i = max(done - S, 0); i < done; i++) ok = mbar_wait(&full[i % S], (i / S) & 1) && ok;
    if (!ok && lane == 0) atomicCAS(a.err, 0, 1);
    return;
  }

  if constexpr (TYPE == SK_NF4) {  // [byte][lane]: half2(code of the high nibble, of the low one)
    uint32_t* table = reinterpret_cast<uint32_t*>(sk_raw + (lut - raw));
    const float lane_code = nf4_code(lane & 15);
    for (int b = warp; b < 256; b += SK_WARPS) {
      const __half2 h = nf4_pair(lane_code, b);
      table[b * 32 + lane] = *reinterpret_cast<const uint32_t*>(&h);
    }
  }
  const uint32_t lut_lane = lut + lane * 4;
  if (W8 && !a.w_late) {  // the run's scales
    prefetch_run(a.s0 + n0, cnt * 2);
    if (GLU) prefetch_run(a.s1 + n0, cnt * 2);
  }
  __syncthreads();
  pdl_wait();
  // This warp's run of a stage and its row tile, and where their fragments lie: rows g and g + 8 of the tile (of a gated pair row g of
  // both matrices), 16-byte chunk c of row r at c ^ (r % 8).
  const int my_tile = warp / KS * TP, my_k = warp % KS;
  const bool active = my_tile < a.tiles;
  // Offsets into a stage, worked out once: a run of a stage lies where it lay in the last one.
  constexpr int UMAX = sk_units(TYPE, NT);
  uint32_t wo[UMAX][2], xo[UMAX][2][NT], so[UMAX][2];
  int xs[UMAX][2][NT];
#pragma unroll
  for (int u = 0; u < UMAX; u++)
#pragma unroll
    for (int h = 0; h < 2; h++) {  // blocks of 64 bytes of a weight row
      const int run = W8 ? my_k * U + u : u * KS + my_k, wr = run * tr + (GLU ? my_tile * 8 : my_tile * 16) + g;
      wo[u][h] = wr * 128 + (((t + 4 * h) ^ (wr & 7)) << 4);
      so[u][h] = NW * w_al + x_al + ((GLU ? my_tile * 8 : my_tile * 16) + g) * a.sp + ((run * 256 + h * 128 + 32 * t) >> a.block_shift) * 2;
#pragma unroll
      for (int n = 0; n < NT; n++) {
        // the k of these weights: half a run of the activations, a run, or two (lanes 0 and 1 in the first)
        const int xr = (TYPE == SK_NF4 ? 4 * run + 2 * h + (t >> 1) : W8 ? 2 * run + h : run) * M + min(n * 8 + g, M - 1);
        xs[u][h][n] = xr & 7;
        xo[u][h][n] = NW * w_al + xr * 128;
      }
    }
  const uint32_t second = GLU ? w_al : 8 * 128, ring0 = smem_u32(ring);
  // the sums this thread finishes: sum j is (weight row 16 tile + g + 8 (i / 2), activation row 8 nt + 2 t + i % 2), j = (tile NT + nt) 4 + i
  const int m_out = (warp / 4 % NT) * 8 + 2 * t + (warp & 1), per = a.tiles * NT * 4;
  auto out_of = [&](int j) { const int tile = j / (4 * NT); return GLU ? tile * 8 + g : tile * 16 + g + 8 * ((j >> 1) & 1); };
  const bool finishes = m_out < M && !(GLU && (warp & 2));
  unsigned long long best = 0ull;
  bool dead = false;
  int slot = 0;
  uint32_t parity = 0;
  for (int pass = 0; pass < passes; pass++) {
    const int nr = min(tr, cnt - pass * tr), base = n0 + pass * tr;
    typename E::Pre pre;
    if (finishes && warp < per && out_of(warp) < nr) pre = E::fetch(e, base + out_of(warp), m_out);
    __half2 s2[TP][2];
    if (W8) {
#pragma unroll
      for (int p = 0; p < TP; p++)
#pragma unroll
        for (int h = 0; h < 2; h++)
          s2[p][h] = __half2half2((GLU && h ? a.s1 : a.s0)[min(base + (GLU ? (my_tile + p) * 8 + g : (my_tile + p) * 16 + g + 8 * h), a.N - 1)]);
    }
    float acc[TP][NT][4];
#pragma unroll
    for (int p = 0; p < TP; p++)
#pragma unroll
      for (int n = 0; n < NT; n++) acc[p][n][0] = acc[p][n][1] = acc[p][n][2] = acc[p][n][3] = 0.f;
    for (int piece = 0; piece < np && active; piece++) {
      if (!dead && !mbar_wait(&full[slot], parity)) { dead = true; if (lane == 0) atomicCAS(a.err, 0, 2); }
      const uint32_t st = ring0 + slot * a.stage_bytes;
#pragma unroll
      for (int u = 0; u < UMAX; u++) {
        if (u >= U) break;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          // everything out of shared memory first: the loads of one tile must not wait for the products of another
          uint4 va[TP], vb[TP];
          __half hs[TP][2];
          uint32_t xw[NT][4 * CPL];
#pragma unroll
          for (int p = 0; p < TP; p++) {
            constexpr int step = GLU ? 8 : 16;  // rows of a tile in the first matrix
            va[p] = sk_lds(st + wo[u][h] + p * step * 128);
            vb[p] = sk_lds(st + wo[u][h] + p * step * 128 + second);
            if (TYPE == SK_NF4) { hs[p][0] = sk_lds_half(st + so[u][h] + p * step * a.sp); hs[p][1] = sk_lds_half(st + so[u][h] + p * step * a.sp + (GLU ? s_al : 8 * a.sp)); }
          }
#pragma unroll
          for (int n = 0; n < NT; n++)
#pragma unroll
            for (int c = 0; c < CPL; c++) {
              const int xc = TYPE == SK_NF4 ? 4 * (t & 1) + c : W8 ? 2 * t + c : t + 4 * h;
              const uint4 v = sk_lds(st + xo[u][h][n] + ((xc ^ xs[u][h][n]) << 4));
              xw[n][4 * c] = v.x; xw[n][4 * c + 1] = v.y; xw[n][4 * c + 2] = v.z; xw[n][4 * c + 3] = v.w;
            }
#pragma unroll
          for (int p = 0; p < TP; p++) {
            if (TYPE == SK_F16 || TYPE == SK_BF16) {
#pragma unroll
              for (int n = 0; n < NT; n++) {
                sk_mma<TYPE == SK_BF16>(acc[p][n], va[p].x, vb[p].x, va[p].y, vb[p].y, xw[n][0], xw[n][1]);
                sk_mma<TYPE == SK_BF16>(acc[p][n], va[p].z, vb[p].z, va[p].w, vb[p].w, xw[n][2], xw[n][3]);
              }
            } else if (W8) {
              uint32_t da[8], db[8];
              w8_to_half2(va[p], s2[p][0], da);
              w8_to_half2(vb[p], s2[p][1], db);
#pragma unroll
              for (int n = 0; n < NT; n++)
#pragma unroll
                for (int i = 0; i < 4; i++) sk_mma<false>(acc[p][n], da[2 * i], db[2 * i], da[2 * i + 1], db[2 * i + 1], xw[n][(2 * i) % (4 * CPL)], xw[n][(2 * i + 1) % (4 * CPL)]);
            } else {
              const __half2 sa = __half2half2(hs[p][0]), sb = __half2half2(hs[p][1]);
              const uint32_t wa[4] = {va[p].x, va[p].y, va[p].z, va[p].w}, wb[4] = {vb[p].x, vb[p].y, vb[p].z, vb[p].w};
              auto pair = [&](uint32_t off, __half2 s) {
                uint32_t c;
                asm("ld.shared.u32 %0, [%1];" : "=r"(c) : "r"((off & 0x7F80u) | lut_lane));
                const __half2 v = __hmul2_rn(*reinterpret_cast<const __half2*>(&c), s);
                return *reinterpret_cast<const uint32_t*>(&v);
              };
#pragma unroll
              for (int i = 0; i < 4; i++) {  // a word holds 8 weights of a row: two instructions
                const uint32_t p0 = pair(wa[i] << 7, sa), p1 = pair(wb[i] << 7, sb), p2 = pair(wa[i] >> 1, sa), p3 = pair(wb[i] >> 1, sb);
                const uint32_t p4 = pair(wa[i] >> 9, sa), p5 = pair(wb[i] >> 9, sb), p6 = pair(wa[i] >> 17, sa), p7 = pair(wb[i] >> 17, sb);
#pragma unroll
                for (int n = 0; n < NT; n++) {
                  sk_mma<false>(acc[p][n], p0, p1, p2, p3, xw[n][(4 * i) % (4 * CPL)], xw[n][(4 * i + 1) % (4 * CPL)]);
                  sk_mma<false>(acc[p][n], p4, p5, p6, p7, xw[n][(4 * i + 2) % (4 * CPL)], xw[n][(4 * i + 3) % (4 * CPL)]);
                }
              }
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&empty[slot])) : "memory");
      if (++slot == S) { slot = 0; parity ^= 1u; }
    }
    // ---- the pass is complete: the sums of the warps that share a tile meet
    if (pass > 0) asm volatile("bar.sync 1, %0;" ::"n"(32 * SK_WARPS) : "memory");  // the last pass's have been read
#pragma unroll
    for (int j = 0; j < PERW; j++) part[(warp * PERW + j) * 32 + lane] = acc[j / (4 * NT)][j / 4 % NT][j & 3];
    asm volatile("bar.sync 1, %0;" ::"n"(32 * SK_WARPS) : "memory");
#pragma unroll
    for (int k = 0; k < EPT; k++) {
      const int j = warp + k * SK_WARPS, o = out_of(j);
      if (finishes && j < per && o < nr) {
        const float* p = part + (j / (4 * NT * TP) * KS * PERW + j % (4 * NT * TP)) * 32 + lane;
        float s = 0.f, u = 0.f;
        for (int q = 0; q < KS; q++) s += p[q * PERW * 32];
        if (GLU)
          for (int q = 0; q < KS; q++) u += p[(q * PERW + 2) * 32];
        E::store(e, base + o, m_out, s, u, k == 0 ? pre : E::fetch(e, base + o, m_out), best);
      }
    }
  }
  if (E::keys(e)) {  // lanes with the same t hold the same activation rows
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
      best = other > best ? other : best;
    }
    if (g == 0 && best != 0ull) atomicMax(E::keys(e) + m_out, best);
  }
}

// ------------------------------------------------------------------------------------------------ host side
struct SkOperands {
  const void *x, *w0, *w1;
  int K, ldx, ldw;  // elements (NF4: ldw = K)
};
template <int TYPE, int NT, int TP, bool GLU, class E>
static int launch_skinny_tp(jg_dev* dev, const char* name, const SkOperands& o, const SkPlan& p, SkArgs a, const typename E::Args& e) {
  a.tr = p.tr; a.tiles = p.tiles; a.ks = p.ks; a.units = p.units; a.runs = p.runs; a.sp = p.sp; a.slice = p.slice; a.pieces = p.pieces;
  a.stages = p.stages; a.stage_bytes = p.stage_bytes;
  const size_t smem = (size_t)p.smem;
  static size_t set[8] = {};
  if (smem > set[dev->ordinal & 7]) {
    JG_CUDA(cudaFuncSetAttribute(skinny_kernel<TYPE, NT, TP, GLU, E>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    set[dev->ordinal & 7] = smem;
  }
  CUtensorMap w0, w1, x, s0, s1;
  const int wb = TYPE == SK_F16 || TYPE == SK_BF16 ? 2 : 1, div = TYPE == SK_NF4 ? 2 : 1, cpl = sk_runs_x(TYPE), slices = TYPE == SK_W8 ? p.ks : 1;
  const bool bf = TYPE == SK_BF16;
  int rc = jg_tensor_map(&w0, o.w0, a.N, o.K / div, o.ldw / div, a.tr, "weights", wb, bf, p.runs, p.slice, slices);
  if (!rc) rc = jg_tensor_map(&w1, GLU ? o.w1 : o.w0, a.N, o.K / div, o.ldw / div, a.tr, "weights (second matrix)", wb, bf, p.runs, p.slice, slices);
  if (!rc) rc = jg_tensor_map(&x, o.x, a.M, o.K, o.ldx, a.M, "activations", 2, bf, p.runs * cpl, p.slice * cpl, slices);
  if (rc) return rc;
  s0 = s1 = x;
  if (TYPE == SK_NF4) {
    rc = jg_tensor_map(&s0, a.s0, a.N, o.K >> a.block_shift, o.K >> a.block_shift, a.tr, "scales", 2, false, -a.sp / 2);
    if (!rc) rc = jg_tensor_map(&s1, GLU ? a.s1 : a.s0, a.N, o.K >> a.block_shift, o.K >> a.block_shift, a.tr, "scales (second matrix)", 2, false, -a.sp / 2);
    if (rc) return rc;
  }
  dev->tc_pending = true;
  return jg_launch(dev, name, skinny_kernel<TYPE, NT, TP, GLU, E>, dim3((unsigned)p.grid), dim3(SK_THREADS), smem, w0, w1, x, s0, s1, a, e);
}
template <int TYPE, int NT, bool GLU, class E>
static int launch_skinny_as(jg_dev* dev, const char* name, const SkOperands& o, const SkArgs& a, const typename E::Args& e) {
  const SkPlan p = sk_plan(TYPE, GLU, a.M, a.N, o.K, a.block_shift, dev->sm_count);
  JG_REQUIRE(p.ok, "%s: no plan for %d rows, N=%d K=%d", name, a.M, a.N, o.K);
  return p.tp == 1 ? launch_skinny_tp<TYPE, NT, 1, GLU, E>(dev, name, o, p, a, e) : launch_skinny_tp<TYPE, NT, 2, GLU, E>(dev, name, o, p, a, e);
}
#endif
