// SPDX-License-Identifier: Apache-2.0
// The cache of TMA tensor maps, with an encoder that only notes what it was asked for: no GPU and no driver.
#include "kernels/tensor_map.h"

#include <cstring>
#include <vector>

#include "cs_test.h"

namespace {
int g_encoded = 0;

// The values a map was made from, kept in its opaque words.
CUresult encode(CUtensorMap *out, CUtensorMapDataType type, cuuint32_t, void *ptr, const cuuint64_t *dims, const cuuint64_t *strides,
                const cuuint32_t *box, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                CUtensorMapFloatOOBfill) {
  ++g_encoded;
  std::memset(out, 0, sizeof(*out));
  const cuuint64_t words[7] = {reinterpret_cast<cuuint64_t>(ptr), dims[0], dims[1], strides[0], box[0], box[1],
                               type == CU_TENSOR_MAP_DATA_TYPE_FLOAT32 ? 4u : 2u};
  std::memcpy(out->opaque, words, sizeof(words));
  return CUDA_SUCCESS;
}
bool holds(const CUtensorMap &map, const cs::kernels::TensorMapKey &k) {
  const cuuint64_t words[7] = {reinterpret_cast<cuuint64_t>(k.ptr), k.inner, k.outer, k.stride_bytes, k.box_inner, k.box_outer,
                               static_cast<cuuint64_t>(k.elem_bytes)};
  return std::memcmp(map.opaque, words, sizeof(words)) == 0;
}
cs::kernels::TensorMapKey rows_of(uint64_t address, uint64_t cols, uint64_t rows, uint32_t box_rows) {
  return {reinterpret_cast<const void *>(address), cols, rows, cols * 2, 64, box_rows, 2};
}
}  // namespace

// qkv [rows, 3 * width] and a gradient [rows, width] whose addresses differ in just the bits that an exclusive-or of the
// address with the shifted column count cancels: 2 GiB for 16 heads of 64, 1 GiB for 8, 512 MiB for 4.
CS_TEST(TensorMap, TensorsAtRelatedAddressesKeepTheirOwnMaps) {
  for (const uint64_t heads : {4, 8, 12, 16, 20}) {
    for (const uint32_t box_rows : {64u, 128u}) {
      cs::kernels::TensorMapCache cache;
      const uint64_t width = heads * 64, rows = 16384, qkv = 0x7f5a00000000ULL;
      const uint64_t grad = qkv ^ ((3 * width ^ width) << 20);
      std::vector<cs::kernels::TensorMapKey> keys{rows_of(qkv, 3 * width, rows, box_rows), rows_of(grad, width, rows, box_rows)};
      for (const auto &key : keys) {
        CUtensorMap map;
        EXPECT_TRUE(cache.get(encode, key, &map));
        EXPECT_TRUE(holds(map, key));
      }
    }
  }
}

CS_TEST(TensorMap, EveryFieldCountsAndAnEntryIsEncodedOnce) {
  cs::kernels::TensorMapCache cache;
  const cs::kernels::TensorMapKey base{reinterpret_cast<const void *>(0x1000), 768, 128, 1536, 64, 128, 2};
  std::vector<cs::kernels::TensorMapKey> keys(8, base);
  keys[1].ptr = reinterpret_cast<const void *>(0x2000);
  keys[2].inner = 760;
  keys[3].outer = 256;
  keys[4].stride_bytes = 4608;
  keys[5].box_inner = 32;
  keys[6].box_outer = 64;
  keys[7].elem_bytes = 4;
  g_encoded = 0;
  for (int pass = 0; pass < 2; ++pass) {
    for (const auto &key : keys) {
      CUtensorMap map;
      EXPECT_TRUE(cache.get(encode, key, &map));
      EXPECT_TRUE(holds(map, key));
    }
    EXPECT_TRUE(g_encoded == static_cast<int>(keys.size()));
  }
  CUtensorMap map;
  EXPECT_TRUE(!cs::kernels::TensorMapCache{}.get(nullptr, base, &map));  // no driver
}

int main(int argc, char **argv) { return cs_test::run_all(argc, argv); }
