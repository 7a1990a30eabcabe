// Projections of the Llama with few activation rows (skinny.cuh): fp16 and int8 weights, the roundings and epilogues of gemm_small.cu.
#include "skinny.cuh"
#include "transcendental.cuh"

enum { SKE_STORE = 0, SKE_RESIDUAL = 1, SKE_SWIGLU = 2, SKE_LOGITS = 3, SKE_PARTIAL = 4 };

struct SkLlama {
  struct Args {
    __half* y;   // [M][N]
    float* y32;  // PARTIAL
    const __half* residual;
    unsigned long long* key;  // LOGITS: [M] (value, lowest index)
    int kind, N, row_offset;
  };
  typedef __half Pre;
  static __device__ __forceinline__ unsigned long long* keys(const Args& e) { return e.key; }
  static __device__ __forceinline__ __half fetch(const Args& e, int n, int m) {
    return e.kind == SKE_RESIDUAL ? e.residual[(size_t)m * e.N + n] : __float2half_rn(0.f);
  }
  static __device__ __forceinline__ void store(const Args& e, int n, int m, float s, float u, __half pre, unsigned long long& best) {
    const size_t o = (size_t)m * e.N + n;
    if (e.kind == SKE_PARTIAL) { e.y32[o] = s; return; }
    __half v = __float2half_rn(s);
    if (e.kind == SKE_RESIDUAL) v = hadd1(pre, v);
    if (e.kind == SKE_SWIGLU) v = jg_silu_mul(v, __float2half_rn(u));
    e.y[o] = v;
    if (e.kind == SKE_LOGITS) {
      const unsigned long long k = argmax_key(v, (uint32_t)(n + e.row_offset));
      best = k > best ? k : best;
    }
  }
};

// Which calls come here.
//
// int8: of those that would go to gemm_small.cu up to 8 rows the single matrices and logits, gate and up from 5 rows on where they are not
// small, 9 to 16 rows the single matrices with an fp16 result.  Their sums are gemm_small.cu's to the bit (skinny_plan.h): a token drawn
// from the flat tail of a quantised model's distribution moves with the last bit of a logit.  ms a step with gate and up there / here: 1B 2
// rows 0.631 / 0.667, 8 rows 0.673 / 0.679; 3B 4 rows 1.500 / 1.604, 5 to 8 rows 1.637 / 1.607 on average; 8B 3 rows 2.26 / 2.30, 4 rows
// 2.29 / 2.29, 8 rows 2.39 / 2.28; with the single matrices there / here 1B 0.80 / 0.67, 3B 1.90 / 1.60, 8B 2.66 / 2.30 (4 rows).  At 16
// rows, us: gate and up of the 8B 32.8 / 34.1, logits 130.3 / 126.7 (9 rows 115.6 / 122.4).
//
// fp16: 3 to 8 rows, logits to 16 (8B: 171.9 / 186.7), but for gate and up where gemm_tc.cu's 128-row tiles keep two thirds of the SMs busy
// (8B: 40.4 / 39.0); at 9 to 16 rows that kernel's MMAs cost no more while these read twice the activations (8B step, 16 rows: 3.90 /
// 3.74 ms with all projections here / there).
bool jg_skinny_fits(const jg_dev* dev, int type, int epi, int M, int N, int K) {
  const bool glu = epi == SKE_SWIGLU;
  if (type == SK_W8) {
    if (glu ? M < 5 || M > 8 || (long long)N * K < 20ll << 20 : M > (epi == SKE_LOGITS ? 8 : 16)) return false;
  } else {
    if (M < 3 || M > (epi == SKE_LOGITS ? 16 : 8) || (glu && N % 128 == 0 && N / 128 * 3 >= dev->sm_count * 2)) return false;
  }
  return sk_plan(type, glu, M, N, K, 0, dev->sm_count).ok;
}

template <int TYPE>
static int launch_skinny(jg_dev* dev, int epi, const SkOperands& o, const SkArgs& a, const SkLlama::Args& e) {
  if (epi == SKE_SWIGLU) return launch_skinny_as<TYPE, 1, true, SkLlama>(dev, "skinny_glu", o, a, e);
  return a.M <= 8 ? launch_skinny_as<TYPE, 1, false, SkLlama>(dev, "skinny", o, a, e) : launch_skinny_as<TYPE, 2, false, SkLlama>(dev, "skinny", o, a, e);
}

// Entry used by gemv.cu's public functions, which ask jg_skinny_fits first; s0, s1: the scales of int8 weights.
int jg_skinny(jg_dev* dev, int type, int epi, const void* x, const void* w0, const void* w1, const void* s0, const void* s1, void* y, const void* residual,
              void* key, int M, int N, int K, int row_offset) {
  const SkOperands o = {x, w0, w1, K, K, K};
  SkArgs a = {};
  a.s0 = (const __half*)s0; a.s1 = (const __half*)s1; a.err = dev->err_word; a.M = M; a.N = N;
  a.w_late = jg_is_fresh(dev, w0) || jg_is_fresh(dev, w1) || jg_is_fresh(dev, s0) || jg_is_fresh(dev, s1);
  SkLlama::Args e = {};
  e.y = (__half*)y; e.y32 = (float*)y; e.residual = (const __half*)residual; e.key = epi == SKE_LOGITS ? (unsigned long long*)key : nullptr;
  e.kind = epi; e.N = N; e.row_offset = row_offset;
  return type == SK_W8 ? launch_skinny<SK_W8>(dev, epi, o, a, e) : launch_skinny<SK_F16>(dev, epi, o, a, e);
}
