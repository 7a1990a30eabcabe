// Projections straight from NF4 weights for up to 8 activation rows (NF4Linear, jsgrad/models/llama3.ts:79-94):
// y[m][n] = half( sum_k float( x[m][k] * half(CODE[code] * scale) ) ), fp32 accumulation, one fp16 scale per `block`
// consecutive elements of the flattened matrix.
//
// The kernel here takes the shapes that skinny.cuh does not (n4_skinny).
//
// The matrix crosses HBM once, packed.  (Writing an fp16 copy first and projecting from that moves 9 bytes per pair of
// weights instead of 1: 10.0 ms per token for the 8B shapes, 2.8 with this kernel.)  At that rate the unpacking is what
// counts: a byte holds two codes, and the pair's fp16 values come out of a 256-entry table in shared memory, one word of
// it per lane and byte in the lane's own bank (32 KB; a table shared by the lanes would meet 3-4 conflicts per access),
// so a pair of weights takes a shift, a mask, a load and a half2 product with the block's scale (one rounding, as the
// dequantised matrix has).  The products run on mma.sync.m16n8k16 with 16 weight rows as A: a lane's 16-byte load of row
// g (and of row g + 8) at k-offset 32 t of a 128-wide k block is its A fragment of eight instructions, the k order inside
// a block being the same permutation for the activations, which come from L1 (columns past the last row repeat it).
//
// A warp walks its (tile, k block) pairs with U loads of each row in flight, refilled across the ends of tiles; KS warps
// share a tile and add their sums in a fixed order at a barrier of their own, two copies of the sums taking turns.
// Epilogues: STORE, RESIDUAL (fp16 add), SWIGLU (two matrices).
#include "skinny.cuh"
#include "transcendental.cuh"

enum { N4_STORE = 0, N4_RESIDUAL = 1, N4_SWIGLU = 2 };

struct Nf4Args {
  const __half* x;  // [M][K]
  const uint8_t *w0, *w1;
  const __half *s0, *s1;
  __half* y;
  const __half* residual;
  int M, N, K, block_shift, late;
};

constexpr int N4_THREADS = 256, N4_WARPS = 8;

__device__ __forceinline__ void n4_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int EPI, int KS>
__global__ void __launch_bounds__(N4_THREADS, 2) jg_matvec_nf4_kernel(const Nf4Args a) {
  constexpr int NW = EPI == N4_SWIGLU ? 2 : 1, U = EPI == N4_SWIGLU ? 2 : 4, GROUPS = N4_WARPS / KS;
  __shared__ uint32_t lut[256 * 32];                      // [byte][lane]: half2(code of the high nibble, of the low one)
  __shared__ float part[2][N4_WARPS][NW][4][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int group = warp / KS, sub = warp % KS;
  const int K = a.K, N = a.N, n_it = K / 128, per = (n_it + KS - 1) / KS;  // k blocks of a row, and of a warp per tile
  const int n_tiles = (N + 15) / 16;
  const long long gg = (long long)blockIdx.x * GROUPS + group, n_groups = (long long)gridDim.x * GROUPS;
  const int tile0 = (int)(gg * n_tiles / n_groups), tile1 = (int)((gg + 1) * n_tiles / n_groups);
  const int total = (tile1 - tile0) * per;
  const size_t row_bytes = (size_t)K / 2, row_blocks = (size_t)(K >> a.block_shift);
  pdl_launch();
  const float lane_code = nf4_code(lane & 15);
  for (int b = warp; b < 256; b += N4_WARPS) {
    const __half2 h = nf4_pair(lane_code, b);
    lut[b * 32 + lane] = *reinterpret_cast<const uint32_t*>(&h);
  }
  if (a.late) pdl_wait();  // the weights were written by a launch that may still be running

  // ---- the stream of weights: register set u holds the pair (tile, k block) that is next in it
  uint4 wv[NW][2][U];
  __half sv[NW][2][U];
  int l_tile = tile0, l_k = 0;  // what is to be loaded next
  auto load = [&](int u) {
    const int it = sub + KS * l_k;
    const bool ok = l_tile < tile1 && it < n_it;
    const int at = it * 128 + t * 32;
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const size_t row = (size_t)min(l_tile * 16 + g + 8 * r, N - 1);  // a repeated row is never stored
#pragma unroll
      for (int w = 0; w < NW; w++) {
        wv[w][r][u] = ok ? ld_stream_128((w ? a.w1 : a.w0) + row * row_bytes + at / 2) : make_uint4(0, 0, 0, 0);
        sv[w][r][u] = ok ? (w ? a.s1 : a.s0)[row * row_blocks + (at >> a.block_shift)] : __float2half_rn(0.f);
      }
    }
    if (++l_k == per) { l_k = 0; l_tile++; }
  };
#pragma unroll
  for (int u = 0; u < U; u++) load(u);
  __syncthreads();  // the table
  if (!a.late) pdl_wait();
  const __half* xr = a.x + (size_t)min(g, a.M - 1) * K + t * 32;
  const unsigned char* mine = reinterpret_cast<const unsigned char*>(lut) + lane * 4;

  float acc[NW][4];
  int c_tile = tile0, c_k = 0;
  for (int j0 = 0; j0 < total; j0 += U) {
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (j0 + u >= total) break;
      if (c_k == 0) {
#pragma unroll
        for (int w = 0; w < NW; w++) acc[w][0] = acc[w][1] = acc[w][2] = acc[w][3] = 0.f;
      }
      uint4 cw[NW][2];
      __half2 cs[NW][2];
#pragma unroll
      for (int w = 0; w < NW; w++)
#pragma unroll
        for (int r = 0; r < 2; r++) { cw[w][r] = wv[w][r][u]; cs[w][r] = __half2half2(sv[w][r][u]); }
      load(u);
      const int it = sub + KS * c_k;
      uint4 xv[4];
#pragma unroll
      for (int i = 0; i < 4; i++) xv[i] = it < n_it ? ld_128(xr + it * 128 + i * 8) : make_uint4(0, 0, 0, 0);
      const uint32_t* xw = reinterpret_cast<const uint32_t*>(xv);
#pragma unroll
      for (int w = 0; w < NW; w++) {
        const uint32_t* wa = reinterpret_cast<const uint32_t*>(&cw[w][0]);
        const uint32_t* wb = reinterpret_cast<const uint32_t*>(&cw[w][1]);
        auto pair = [&](uint32_t off, __half2 s) {
          const __half2 v = __hmul2_rn(*reinterpret_cast<const __half2*>(mine + (off & 0x7F80u)), s);
          return *reinterpret_cast<const uint32_t*>(&v);
        };
#pragma unroll
        for (int i = 0; i < 4; i++) {  // one word = 8 weights of each row = two instructions
          n4_mma(acc[w], pair(wa[i] << 7, cs[w][0]), pair(wb[i] << 7, cs[w][1]), pair(wa[i] >> 1, cs[w][0]), pair(wb[i] >> 1, cs[w][1]), xw[4 * i], xw[4 * i + 1]);
          n4_mma(acc[w], pair(wa[i] >> 9, cs[w][0]), pair(wb[i] >> 9, cs[w][1]), pair(wa[i] >> 17, cs[w][0]), pair(wb[i] >> 17, cs[w][1]), xw[4 * i + 2], xw[4 * i + 3]);
        }
      }
      if (++c_k < per) continue;
      // ---- a tile is complete: the warps of the group add their sums, in turn
      const int buf = (c_tile - tile0) & 1;
#pragma unroll
      for (int w = 0; w < NW; w++)
#pragma unroll
        for (int i = 0; i < 4; i++) part[buf][warp][w][i][lane] = acc[w][i];
      if (KS == N4_WARPS) __syncthreads();
      else if (KS > 1) asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(KS * 32) : "memory");
      else __syncwarp();
      if (sub == (c_tile - tile0) % KS) {
#pragma unroll
        for (int i = 0; i < 4; i++) {  // sum i of a lane: weight row g + 8 (i / 2), activation row 2 t + i % 2
          const int n = c_tile * 16 + g + 8 * (i >> 1), m = 2 * t + (i & 1);
          if (n < N && m < a.M) {
            float s[NW];
#pragma unroll
            for (int w = 0; w < NW; w++) {
              s[w] = 0.f;
#pragma unroll
              for (int q = 0; q < KS; q++) s[w] += part[buf][group * KS + q][w][i][lane];
            }
            const size_t o = (size_t)m * N + n;
            __half v = __float2half_rn(s[0]);
            if (EPI == N4_RESIDUAL) v = hadd1(a.residual[o], v);
            if (EPI == N4_SWIGLU) v = jg_silu_mul(v, __float2half_rn(s[NW - 1]));
            a.y[o] = v;
          }
        }
      }
      c_k = 0;
      c_tile++;
    }
  }
}

template <int EPI, int KS>
static int launch_n4(jg_dev* dev, const Nf4Args& a, const char* name) {
  const long long n_tiles = (a.N + 15) / 16, groups = N4_WARPS / KS;
  long long blocks = 2LL * dev->sm_count;
  if (blocks * groups > n_tiles) blocks = (n_tiles + groups - 1) / groups;
  return jg_launch(dev, name, jg_matvec_nf4_kernel<EPI, KS>, dim3((unsigned)blocks), dim3(N4_THREADS), 0, a);
}

// K over 1, 2, 4 or 8 warps: the one whose warps have the fewest k blocks to walk, and among equals the fewest warps per
// tile (fewer barriers).
template <int EPI>
static int launch_n4_ks(jg_dev* dev, const Nf4Args& a, const char* name) {
  const long long n_tiles = (a.N + 15) / 16, n_it = a.K / 128, warps = 2LL * dev->sm_count * N4_WARPS;
  int best = 1;
  long long best_walk = 0;
  for (int ks = 1; ks <= N4_WARPS; ks <<= 1) {
    const long long groups = warps / ks, walk = (n_tiles + groups - 1) / groups * ((n_it + ks - 1) / ks);
    if (ks == 1 || walk < best_walk) { best = ks; best_walk = walk; }
  }
  switch (best) {
    case 1: return launch_n4<EPI, 1>(dev, a, name);
    case 2: return launch_n4<EPI, 2>(dev, a, name);
    case 4: return launch_n4<EPI, 4>(dev, a, name);
  }
  return launch_n4<EPI, 8>(dev, a, name);
}

// What skinny.cuh does with a sum: the roundings above.
struct SkNf4 {
  struct Args {
    __half* y;
    const __half* residual;
    int N, glu;
  };
  typedef __half Pre;
  static __device__ __forceinline__ unsigned long long* keys(const Args&) { return nullptr; }
  static __device__ __forceinline__ __half fetch(const Args& e, int n, int m) { return e.residual ? e.residual[(size_t)m * e.N + n] : __float2half_rn(0.f); }
  static __device__ __forceinline__ void store(const Args& e, int n, int m, float s, float u, __half pre, unsigned long long&) {
    __half v = __float2half_rn(s);
    if (e.residual) v = hadd1(pre, v);
    if (e.glu) v = jg_silu_mul(v, __float2half_rn(u));
    e.y[(size_t)m * e.N + n] = v;
  }
};
// Rows of whole 128-byte runs and blocks whose scales come in 16-byte pieces: the kernel around the weight stream (skinny.cuh), where it
// has a plan.
static bool n4_skinny(const jg_dev* dev, const Nf4Args& a, bool glu) {
  return a.block_shift >= 5 && a.block_shift <= 8 && a.K % (8 << a.block_shift) == 0 && a.K % 256 == 0 && (uintptr_t)a.s0 % 16 == 0 &&
         (uintptr_t)a.s1 % 16 == 0 && sk_plan(SK_NF4, glu, a.M, a.N, a.K, a.block_shift, dev->sm_count).ok;
}
template <bool GLU>
static int launch_n4_skinny(jg_dev* dev, const Nf4Args& n, const char* name) {
  SkArgs a = {};
  a.s0 = n.s0; a.s1 = n.s1; a.err = dev->err_word; a.M = n.M; a.N = n.N; a.block_shift = n.block_shift; a.w_late = n.late;
  const SkOperands o = {n.x, n.w0, n.w1, n.K, n.K, n.K};
  const SkNf4::Args e = {n.y, n.residual, n.N, GLU};
  return launch_skinny_as<SK_NF4, 1, GLU, SkNf4>(dev, name, o, a, e);
}

// Rows a call takes.  One n-tile of the MMA: up to 8 rows cost what one does.  Beyond, a dequantised copy and the
// tensor-core projection are used (jg_dequant_nf4_f16, jg_linear).
constexpr int N4_MAX_ROWS = 8;

static int nf4_check(const char* name, uint64_t y, uint64_t x, uint64_t w, uint64_t scale, int M, int N, int K, int block, Nf4Args* a) {
  JG_REQUIRE(M > 0 && N > 0 && K > 0 && block > 0, "%s: bad shape M=%d N=%d K=%d block=%d", name, M, N, K, block);
  JG_REQUIRE(jg_aligned(y, 2) && jg_aligned(x, 16) && jg_aligned(w, 16) && jg_aligned(scale, 2), "%s: null or misaligned pointer", name);
  if (M > N4_MAX_ROWS || K % 128 != 0 || block < 32 || (block & (block - 1)) != 0 || K % block != 0) {
    jg_set_error("%s: M=%d K=%d block=%d: up to %d rows, K a multiple of 128 and of a power-of-two block of 32 or more", name, M, K, block, N4_MAX_ROWS);
    return JG_ENOTSUP;
  }
  a->x = (const __half*)x; a->y = (__half*)y; a->w0 = (const uint8_t*)w; a->s0 = (const __half*)scale;
  a->M = M; a->N = N; a->K = K; a->block_shift = 31 - __builtin_clz((unsigned)block);
  return JG_OK;
}

JG_API int jg_linear_nf4(jg_dev* dev, uint64_t y, uint64_t x, uint64_t w, uint64_t scale, uint64_t residual, int32_t M, int32_t N, int32_t K,
                         int32_t block) {
  JG_ENTER(dev);
  Nf4Args a = {};
  int rc = nf4_check("linear_nf4", y, x, w, scale, M, N, K, block, &a);
  if (rc) return rc;
  a.late = jg_is_fresh(dev, a.w0) || jg_is_fresh(dev, a.s0);
  jg_mark_fresh(dev, y, (uint64_t)M * N * 2);
  JG_REQUIRE(residual == 0 || jg_aligned(residual, 2), "linear_nf4: misaligned residual pointer");
  a.residual = (const __half*)residual;
  if (n4_skinny(dev, a, false)) return launch_n4_skinny<false>(dev, a, "linear_nf4");
  if (!residual) return launch_n4_ks<N4_STORE>(dev, a, "linear_nf4");
  return launch_n4_ks<N4_RESIDUAL>(dev, a, "linear_nf4");
}

JG_API int jg_swiglu_nf4(jg_dev* dev, uint64_t y, uint64_t x, uint64_t w_gate, uint64_t s_gate, uint64_t w_up, uint64_t s_up, int32_t M, int32_t N,
                         int32_t K, int32_t block) {
  JG_ENTER(dev);
  Nf4Args a = {};
  int rc = nf4_check("swiglu_nf4", y, x, w_gate, s_gate, M, N, K, block, &a);
  if (rc) return rc;
  JG_REQUIRE(jg_aligned(w_up, 16) && jg_aligned(s_up, 2), "swiglu_nf4: null or misaligned up-projection weight");
  a.w1 = (const uint8_t*)w_up; a.s1 = (const __half*)s_up;
  a.late = jg_is_fresh(dev, a.w0) || jg_is_fresh(dev, a.s0) || jg_is_fresh(dev, a.w1) || jg_is_fresh(dev, a.s1);
  jg_mark_fresh(dev, y, (uint64_t)M * N * 2);
  if (n4_skinny(dev, a, true)) return launch_n4_skinny<true>(dev, a, "swiglu_nf4");
  return launch_n4_ks<N4_SWIGLU>(dev, a, "swiglu_nf4");
}
