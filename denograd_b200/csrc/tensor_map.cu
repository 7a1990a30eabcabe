// Encoded TMA tensor maps of the tensor-core projections, kept per operand (declared in tcgen05.cuh).
#include <mutex>

#include "gemm_pair.cuh"

typedef CUresult (*encode_tiled_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                    const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static encode_tiled_fn g_encode = nullptr;

static int find_encoder() {
  if (!g_encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres);
    if (e != cudaSuccess || fn == nullptr) {
      jg_set_error("cuTensorMapEncodeTiled is not available from this driver");
      return JG_ENOTSUP;
    }
    g_encode = (encode_tiled_fn)fn;
  }
  return JG_OK;
}
// `bytes` = element size: 2 for fp16 operands (128-byte swizzle, the layout the MMA descriptors name), 1 for int8
// weight tiles, which land unswizzled (64-byte rows) for the converting warps
static int make_map(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows, const char* what, int bytes, bool bf16, int groups,
                    int slice, int slices) {
  const int rc = find_encoder();
  if (rc) return rc;
  const cuuint32_t run = 128 / bytes;
  const cuuint64_t dims[4] = {groups > 0 ? run : cols, rows, slice > 0 ? slice : cols / run, slice > 0 ? cols / run / slice : 1};  // innermost first
  const cuuint64_t strides[3] = {ld * (cuuint64_t)bytes, 128, 128ull * slice};  // bytes between rows, between runs, between slices
  const cuuint32_t box[4] = {groups > 0 ? run : groups < 0 ? (cuuint32_t)-groups : 64, box_rows, (cuuint32_t)(groups / slices), (cuuint32_t)slices};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUtensorMapDataType type = bytes == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : (bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16);
  CUresult r = g_encode(m, type, slice > 0 ? 4 : groups > 0 ? 3 : 2, const_cast<void*>(base), dims,
                        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        groups > 0 || (bytes == 2 && groups == 0) ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    jg_set_error("tensor map for %s (%llu x %llu) rejected: CUresult %d", what, (unsigned long long)rows, (unsigned long long)cols, (int)r);
    return JG_EINVAL;
  }
  return JG_OK;
}

// Encoded maps are kept per (base, rows, cols, box rows): a model's weights and workspaces keep their addresses, so a
// step after the first finds all of its maps here instead of encoding three per launch.
struct MapKey { const void* base; uint64_t rows, cols, ld; uint32_t box_rows; int bytes; bool bf16; int groups, slice, slices; };
struct MapSlot { MapKey k; CUtensorMap m; bool used; };
constexpr int MAP_SLOTS = 8192;
static MapSlot g_maps[MAP_SLOTS];

int jg_tensor_map(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows, const char* what,
                  int bytes, bool bf16, int groups, int slice, int slices) {
  uint64_t h = (uint64_t)(uintptr_t)base * 0x9E3779B97F4A7C15ull ^ (rows * 0xBF58476D1CE4E5B9ull) ^ (cols << 20) ^ (ld << 4) ^ box_rows ^ ((uint64_t)bytes << 40) ^ ((uint64_t)bf16 << 43) ^ ((uint64_t)(uint32_t)groups << 44) ^
               ((uint64_t)slice << 48) ^ ((uint64_t)slices << 58);
  h ^= h >> 29;
  for (int probe = 0; probe < 8; probe++) {
    MapSlot& s = g_maps[(h + probe) % MAP_SLOTS];
    if (s.used && s.k.base == base && s.k.rows == rows && s.k.cols == cols && s.k.ld == ld && s.k.box_rows == box_rows && s.k.bytes == bytes &&
        s.k.bf16 == bf16 && s.k.groups == groups && s.k.slice == slice && s.k.slices == slices) { *out = s.m; return JG_OK; }
    if (!s.used) {
      int rc = make_map(&s.m, base, rows, cols, ld, box_rows, what, bytes, bf16, groups, slice, slices);
      if (rc) return rc;
      s.k = MapKey{base, rows, cols, ld, box_rows, bytes, bf16, groups, slice, slices};
      s.used = true;
      *out = s.m;
      return JG_OK;
    }
  }
  MapSlot& s = g_maps[h % MAP_SLOTS];  // neighbourhood full: replace
  int rc = make_map(&s.m, base, rows, cols, ld, box_rows, what, bytes, bf16, groups, slice, slices);
  if (rc) { s.used = false; return rc; }
  s.k = MapKey{base, rows, cols, ld, box_rows, bytes, bf16, groups, slice, slices};
  s.used = true;
  *out = s.m;
  return JG_OK;
}

bool jg_tensor_map_two(CUtensorMap* out, const void* lo, const void* hi, uint64_t rows, uint64_t cols, uint64_t ld, bool bf16) {
  const uint64_t apart = (uint64_t)(uintptr_t)hi - (uint64_t)(uintptr_t)lo;
  if (lo >= hi || apart % 16 != 0 || apart >= (1ull << 40) || rows % 16 != 0 || find_encoder() != JG_OK) return false;
  const cuuint64_t dims[4] = {cols, 16, 2, rows / 16}, strides[3] = {2 * ld, apart, 32 * ld};
  const cuuint32_t box[4] = {64, 16, 2, 4}, estr[4] = {1, 1, 1, 1};
  return g_encode(out, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void*>(lo), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static size_t pair_flag_bytes(const jg_dev* dev) { return (size_t)(dev->sm_count / 2) * 2 * GP_EPI_WARPS * sizeof(uint32_t); }
bool jg_pair_workspace(jg_dev* dev) {
  static std::mutex m;
  std::lock_guard<std::mutex> lock(m);
  if (dev->pair_slots != nullptr) return true;
  if (dev->capturing) return false;
  const size_t slots = (size_t)(dev->sm_count / 2) * 2 * GP_SLOT * sizeof(float);
  void* p = nullptr;
  if (cudaMalloc(&p, slots + pair_flag_bytes(dev)) != cudaSuccess) { cudaGetLastError(); return false; }
  if (cudaMemsetAsync((char*)p + slots, 0, pair_flag_bytes(dev), dev->stream) != cudaSuccess) { cudaGetLastError(); cudaFree(p); return false; }
  dev->pair_flags = (uint32_t*)((char*)p + slots);
  dev->pair_slots = (float*)p;
  return true;
}
void jg_pair_reset(jg_dev* dev) {
  if (dev->pair_flags != nullptr) cudaMemsetAsync(dev->pair_flags, 0, pair_flag_bytes(dev), dev->stream);
}
