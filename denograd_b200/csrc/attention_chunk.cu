// Attention for a multi-position chunk (prompt processing): Sc consecutive positions of each of B sequences attend
// causally to the paged KV cache, which already holds the chunk's own K and V (jg_rope_kvwrite_rows ran before).
//
// Arithmetic is Tensor.scaled_dot_product_attention with the additive causal mask of Transformer.forward
// (jsgrad/tensor.ts:3920-3934, softmax :2186-2214, mask jsgrad/models/llama.ts:208): fp32 scores (q.k) * 1/sqrt(hd),
// masked above the diagonal; e = exp2((s - max) * 1/ln2) with the polynomial exp2; p = half(e * (1/sum e));
// out = half(sum_t p_t * v_t) accumulated in fp32.  p is rounded to fp16 *after* normalisation, so the row maximum and
// sum must be known before the first p.v product: the context is walked twice (max and sum together, then p.v),
// recomputing the cheap q.k^T on the tensor cores instead of keeping a [rows][context] score matrix.  (exp2 is the
// hardware's, 2^-22 relative, where the reference's polynomial is good to 2^-23: both far below the 2^-11 of p.)
//
// The work runs in flash_tc.cuh: a tile of 128 query rows is 128 / n_rep consecutive positions times the n_rep heads that
// share one kv head (repeat_kv, jsgrad/models/llama.ts:34-39), so a tile of keys serves them all; pages of the cache are
// the boxes of the TMA loads.  8B shapes, us per launch with a cold cache, against mma.sync on tiles of 16 positions: 512
// positions 24.6 (63.0), 1024 55 (143), 2048 114 (471), 512 after 1536 52 (222), 45 16.4 (15.9).
#include <stdlib.h>

#include "common.cuh"
#include "flash_tc.cuh"
#include "kvcache.cuh"

struct ChunkArgs {
  const __half* qkv;  // [R][qkv_stride], row = s * B + b, q heads first, already rotated
  const __half* k_layer;
  const __half* v_layer;
  const int32_t* block_table;
  const int32_t* pos;  // [R]; pos[s * B + b] = pos[b] + s
  const int32_t* seq;  // [R] row -> block-table row, or null (row b of the chunk is sequence b)
  __half* out;         // [R][H * hd]
  int qkv_stride, H, G, B, Sc, page, page_shift, max_pages_per_seq, max_ctx;
  int n_seq;  // rows of the block table: a sequence whose seq[] entry lies outside [0, n_seq) is skipped
  float scale;
  int* err;
};

template <int HD, int NREP, bool SPLIT>
struct ChunkPolicy {
  static constexpr int DK = HD, DV = HD, PT = FT_ROWS / NREP;  // positions of a 128-row tile
  static constexpr bool BF16 = false;
  const ChunkArgs& a;
  const CUtensorMap *mk, *mv;
  int tiles, b, g, s0, p_lo, written, lim;
  bool valid;
  const int32_t* bt_row;
  float scale2;
  __device__ ChunkPolicy(const ChunkArgs& a_, const CUtensorMap* k, const CUtensorMap* v) : a(a_), mk(k), mv(v) {}
  __device__ __forceinline__ bool begin() {
    constexpr int POS = PT * (SPLIT ? 1 : 2);
    const int qt = (int)gridDim.x - 1 - (int)blockIdx.x;  // long rows first
    g = blockIdx.y;
    b = blockIdx.z;
    const int sq = a.seq ? a.seq[b] : b;
    if ((unsigned)sq >= (unsigned)a.n_seq) return false;
    const int pos0 = a.pos[b];
    if (pos0 < 0) return false;
    written = min(pos0 + a.Sc, a.max_ctx);  // the cache holds positions [0, written) of this sequence
    s0 = qt * POS;
    p_lo = pos0 + s0;
    tiles = (min(p_lo + min(POS, a.Sc - s0), written) + FT_KV - 1) / FT_KV;
    bt_row = a.block_table + (size_t)sq * a.max_pages_per_seq;
    scale2 = a.scale * 1.4426950408889634f;
    return tiles > 0;
  }
  __device__ __forceinline__ int position(int stream, int r) const { return s0 + stream * PT + r / NREP; }  // within the chunk
  template <typename F>
  __device__ __forceinline__ void q_row(int stream, int r, F dst) const {
    const int s = min(position(stream, r), a.Sc - 1);  // rows past the end repeat the last position
    const __half* q = a.qkv + ((size_t)s * a.B + b) * a.qkv_stride + (size_t)(g * NREP + r % NREP) * HD;
#pragma unroll
    for (int c = 0; c < HD / 8; c++) dst(c, ld_128(q + c * 8));
  }
  __device__ __forceinline__ void rows(int stream, int r) {
    const int s = position(stream, r);
    valid = r < PT * NREP && s < a.Sc;
    lim = min(p_lo - s0 + min(s, a.Sc - 1), written - 1);
  }
  __device__ __forceinline__ bool all(int j) const { return j * FT_KV + FT_KV - 1 <= lim; }
  __device__ __forceinline__ bool sees(int j, int c) const { return j * FT_KV + c <= lim; }
  __device__ __forceinline__ float extra2() const { return -INFINITY; }
  __device__ __forceinline__ int dead(int j) const { return min(FT_KV, written - j * FT_KV); }
  __device__ __forceinline__ void load(const CUtensorMap* m, int j, unsigned char* dst, uint64_t* bar, int lane) const {
    constexpr int KB = HD / 64;
    const int run = lane / KB, block = lane % KB;
    if (run * a.page >= FT_KV) return;
    const int pg = bt_row[min(((j * FT_KV) >> a.page_shift) + run, (written - 1) >> a.page_shift)];  // past the end: some page, masked
    tma_load_2d(dst + block * (FT_KV * 128) + run * a.page * 128, m, block * 64, (pg * a.G + g) * a.page, bar);
  }
  __device__ __forceinline__ void load_k(int j, unsigned char* dst, uint64_t* bar, int lane) const { load(mk, j, dst, bar, lane); }
  __device__ __forceinline__ void load_v(int j, unsigned char* dst, uint64_t* bar, int lane) const { load(mv, j, dst, bar, lane); }
  __device__ __forceinline__ void store(int stream, int r, const float* o, int c) const {
    if (!valid) return;
    __half* out = a.out + ((size_t)position(stream, r) * a.B + b) * ((size_t)a.H * HD) + (size_t)(g * NREP + r % NREP) * HD + c;
#pragma unroll
    for (int k = 0; k < 32; k += 8) {
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const __half2 h = __floats2half2_rn(o[k + 2 * i], o[k + 2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t*>(&h);
      }
      *reinterpret_cast<uint4*>(out + k) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
};

template <int HD, int NREP, bool SPLIT>
__global__ void __launch_bounds__(FT_THREADS, 1) attn_chunk_kernel(const __grid_constant__ CUtensorMap mk, const __grid_constant__ CUtensorMap mv,
                                                                   const ChunkArgs a) {
  ChunkPolicy<HD, NREP, SPLIT> p(a, &mk, &mv);
  flash_tc<ChunkPolicy<HD, NREP, SPLIT>, SPLIT>(p, a.err);
}

template <int HD, int NREP, bool SPLIT>
static int launch_chunk(jg_dev* dev, const ChunkArgs& a, const CUtensorMap& mk, const CUtensorMap& mv) {
  auto kern = attn_chunk_kernel<HD, NREP, SPLIT>;
  const size_t smem = FtCfg<HD, HD, SPLIT>::SMEM;
  static bool attr_set[8] = {false, false, false, false, false, false, false, false};
  const int slot = dev->ordinal & 7;
  if (!attr_set[slot]) {
    JG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_set[slot] = true;
  }
  constexpr int POS = FT_ROWS / NREP * (SPLIT ? 1 : 2);
  dim3 grid((a.Sc + POS - 1) / POS, a.G, a.B);
  dev->tc_pending = true;
  return jg_launch(dev, "attn_chunk", kern, grid, dim3(FT_THREADS), smem, mk, mv, a);
}

// Pairs of query tiles where they give every SM a CTA; below that the key tiles of single ones are split between the streams.
template <int HD, int NREP>
static int launch_chunk_rows(jg_dev* dev, const ChunkArgs& a, const CUtensorMap& mk, const CUtensorMap& mv) {
  constexpr int POS = FT_ROWS / NREP * 2;
  const long long pairs = (long long)((a.Sc + POS - 1) / POS) * a.G * a.B;
  return pairs >= dev->sm_count ? launch_chunk<HD, NREP, false>(dev, a, mk, mv) : launch_chunk<HD, NREP, true>(dev, a, mk, mv);
}

JG_API int jg_attn_chunk(jg_dev* dev, jg_kvcache* kv, int32_t layer, uint64_t out, uint64_t qkv, uint64_t pos, uint64_t seq,
                         int32_t B, int32_t Sc, int32_t H) {
  JG_ENTER(dev);
  JG_REQUIRE(kv != nullptr && kv->dev == dev, "attn_chunk: cache belongs to another device");
  JG_REQUIRE(layer >= 0 && layer < kv->d.n_layers, "attn_chunk: layer %d out of range", layer);
  JG_REQUIRE(B > 0 && B <= 65535 && (seq != 0 || B <= kv->d.max_batch) && Sc > 0 && Sc <= kv->max_ctx && H == kv->d.n_heads,
             "attn_chunk: B=%d Sc=%d H=%d do not match the cache (max_batch %d, context %d, n_heads %d)", B, Sc, H,
             kv->d.max_batch, kv->max_ctx, kv->d.n_heads);
  JG_REQUIRE(jg_aligned(out, 16) && jg_aligned(qkv, 16) && jg_aligned(pos, 4) && (seq == 0 || jg_aligned(seq, 4)),
             "attn_chunk: null or misaligned pointer");
  const int G = kv->d.n_kv_heads, hd = kv->d.head_dim, n_rep = H / G;
  ChunkArgs a = {};
  a.qkv = (const __half*)qkv;
  a.k_layer = kv->k_pool + kv->layer_elems * layer;
  a.v_layer = kv->v_pool + kv->layer_elems * layer;
  a.block_table = kv->block_table;
  a.pos = (const int32_t*)pos; a.seq = (const int32_t*)seq; a.out = (__half*)out;
  a.qkv_stride = (H + 2 * G) * hd; a.H = H; a.G = G; a.B = B; a.Sc = Sc;
  a.page = kv->d.page_size; a.page_shift = ilog2(kv->d.page_size);
  a.max_pages_per_seq = kv->d.max_pages_per_seq; a.max_ctx = kv->max_ctx; a.n_seq = kv->d.max_batch;
  a.scale = (float)(1.0 / (double)(float)sqrt((double)hd));  // as the reference folds it (jsgrad/tensor.ts:3923)
  CUtensorMap mk, mv;
  const uint64_t rows = (uint64_t)kv->d.n_pages * G * kv->d.page_size;
  int rc = jg_tensor_map(&mk, a.k_layer, rows, hd, hd, a.page, "cached keys");
  if (!rc) rc = jg_tensor_map(&mv, a.v_layer, rows, hd, hd, a.page, "cached values");
  if (rc) return rc;
  a.err = dev->err_word;
#define JG_CH_CASE(HD_, NR_) if (hd == HD_ && n_rep == NR_) return launch_chunk_rows<HD_, NR_>(dev, a, mk, mv);
  JG_CH_CASE(64, 1) JG_CH_CASE(64, 2) JG_CH_CASE(64, 3) JG_CH_CASE(64, 4) JG_CH_CASE(64, 8)
  JG_CH_CASE(128, 1) JG_CH_CASE(128, 2) JG_CH_CASE(128, 3) JG_CH_CASE(128, 4) JG_CH_CASE(128, 8)
#undef JG_CH_CASE
  jg_set_error("attn_chunk: head_dim %d with %d query heads per kv head not supported", hd, n_rep);
  return JG_ENOTSUP;
}
