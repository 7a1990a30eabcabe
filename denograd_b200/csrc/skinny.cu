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

// Which calls come here.  int8: up to 8 rows all, 9 to 16 the single matrices with an fp16 result (gate and up of the 8B at 16 rows, us
// here / in gemm_small.cu: 34.1 / 32.8, logits 126.7 / 130.3 at 16 and 122.4 / 115.6 at 9 rows; the others as in skinny.cuh).  fp16: 3 to
// 8 rows, logits to 16 (8B: 171.9 / 186.7), but for gate and up where gemm_tc.cu's 128-row tiles keep two thirds of the SMs busy
// (8B: 40.4 / 39.0); at 9 to 16 rows that kernel's MMAs cost no more while these read twice the activations (8B step, 16 rows: 3.90 /
// 3.74 ms with all projections here / there).
bool jg_skinny_fits(const jg_dev* dev, bool w8, int epi, int M, int N, int K) {
  if (w8) return K % 128 == 0 && (M <= 8 || (M <= 16 && epi != SKE_SWIGLU && epi != SKE_LOGITS));
  if (K % 64 != 0 || M < 3) return false;
  if (epi == SKE_LOGITS) return M <= 16;
  return M <= 8 && !(epi == SKE_SWIGLU && N % 128 == 0 && N / 128 * 3 >= dev->sm_count * 2);
}

template <int TYPE>
static int launch_skinny(jg_dev* dev, int epi, const SkOperands& o, const SkArgs& a, const SkLlama::Args& e) {
  if (epi == SKE_SWIGLU) return launch_skinny_as<TYPE, 1, true, SkLlama>(dev, "skinny_glu", o, a, e);
  return a.M <= 8 ? launch_skinny_as<TYPE, 1, false, SkLlama>(dev, "skinny", o, a, e) : launch_skinny_as<TYPE, 2, false, SkLlama>(dev, "skinny", o, a, e);
}

// Entry used by gemv.cu's public functions; s0 / s1 non-null = int8 weights with per-row scales.
int jg_skinny(jg_dev* dev, int epi, const void* x, const void* w0, const void* w1, const void* s0, const void* s1, void* y, const void* residual,
              void* key, int M, int N, int K, int row_offset) {
  const SkOperands o = {x, w0, w1, K, K, K};
  SkArgs a = {};
  a.s0 = (const __half*)s0; a.s1 = (const __half*)s1; a.err = dev->err_word; a.M = M; a.N = N;
  a.w_late = jg_is_fresh(dev, w0) || jg_is_fresh(dev, w1) || jg_is_fresh(dev, s0) || jg_is_fresh(dev, s1);
  SkLlama::Args e = {};
  e.y = (__half*)y; e.y32 = (float*)y; e.residual = (const __half*)residual; e.key = epi == SKE_LOGITS ? (unsigned long long*)key : nullptr;
  e.kind = epi; e.N = N; e.row_offset = row_offset;
  return s0 ? launch_skinny<SK_W8>(dev, epi, o, a, e) : launch_skinny<SK_F16>(dev, epi, o, a, e);
}
