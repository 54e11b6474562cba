// Host side of the tensor maps: cuTensorMapEncodeTiled, looked up through the runtime (no link to libcuda).
#include "tensor_map.cuh"

#include <numeric>

namespace ha {

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                             const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeFn encode_fn() {
  static const EncodeFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult qr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &qr) != cudaSuccess) f = nullptr;
    return (EncodeFn)f;
  }();
  return fn;
}

static CUtensorMapDataType map_type(int dtype) {
  return dtype == HA_FP32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : dtype == HA_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
}

static bool encode(CUtensorMap* map, int dtype, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box,
                   CUtensorMapL2promotion promo) {
  const EncodeFn fn = encode_fn();
  if (!fn || (uintptr_t)base % 16 != 0) return false;
  for (int i = 0; i < rank - 1; ++i)
    if (strides[i] == 0 || strides[i] % 16 != 0 || strides[i] >= (1ull << 40)) return false;
  for (int i = 0; i < rank; ++i)
    if (dims[i] == 0 || dims[i] > 0x7fffffffull) return false;
  const cuuint32_t ones[4] = {1, 1, 1, 1};
  return fn(map, map_type(dtype), (cuuint32_t)rank, const_cast<void*>(base), dims,
            strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, promo,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool encode_tile_map(CUtensorMap* map, int dtype, const void* base, int width, long long rows, int H, int B, int64_t sn, int64_t sh, int64_t sb,
                     int box_rows) {
  // a dimension of extent 1 is never stepped through: its stride is only a number the encoder checks
  if (H == 1) sh = sn;
  if (B == 1) sb = sn;
  if (sn < width || sh < 0 || sb < 0) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)width, (cuuint64_t)rows, (cuuint64_t)H, (cuuint64_t)B};
  const cuuint64_t strides[3] = {(cuuint64_t)sn * 2, (cuuint64_t)sh * 2, (cuuint64_t)sb * 2};
  const cuuint32_t box[4] = {64, (cuuint32_t)box_rows, 1, 1};
  return encode(map, dtype, base, 4, dims, strides, box, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
}

bool encode_acc_map(CUtensorMap* map, float* base, int width, long long rows, long long heads) {
  const cuuint64_t dims[3] = {(cuuint64_t)width, (cuuint64_t)rows, (cuuint64_t)heads};
  const cuuint64_t strides[2] = {(cuuint64_t)width * 4, (cuuint64_t)width * 4 * (cuuint64_t)rows};
  const cuuint32_t box[3] = {32, TILE, 1};
  return encode(map, HA_FP32, base, 3, dims, strides, box, CU_TENSOR_MAP_L2_PROMOTION_NONE);
}

bool encode_row_map(CUtensorMap* map, int dtype, const void* base, int width, long long rows, int H, int B, int64_t sn, int64_t sh, int64_t sb,
                    int64_t* pitch) {
  if (sn <= 0 || sh < 0 || sb < 0) return false;
  int64_t g = sn;
  if (H > 1) g = std::gcd(g, sh);
  if (B > 1) g = std::gcd(g, sb);
  if (g < width) return false;
  const long long last = ((B > 1 ? (B - 1) * sb : 0) + (H > 1 ? (H - 1) * sh : 0) + (rows - 1) * sn) / g;
  const cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)(last + 1)};
  const cuuint64_t strides[1] = {(cuuint64_t)g * 2};
  const cuuint32_t box[2] = {64, 1};
  *pitch = g;
  // single rows in no order: nothing beyond the row itself is worth fetching
  return encode(map, dtype, base, 2, dims, strides, box, width <= 64 ? CU_TENSOR_MAP_L2_PROMOTION_L2_128B : CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
}

}  // namespace ha
