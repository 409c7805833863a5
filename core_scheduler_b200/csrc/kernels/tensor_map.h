// SPDX-License-Identifier: Apache-2.0
// Host side of TMA: 2-D tensor maps with the 128-byte swizzle, encoded once per (address, shape, stride, box) and kept.
// A map holds nothing but these values, so an entry stays right for whatever memory comes to lie at its address later.
#pragma once

#include <cuda.h>

#include <cstddef>
#include <cstdint>
#include <mutex>
#include <unordered_map>

namespace cs::kernels {
using TensorMapEncodeFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                       const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                       CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// `inner` contiguous elements per row, `outer` rows; the copied box is box_inner x box_outer.
struct TensorMapKey {
  const void *ptr;
  uint64_t inner, outer, stride_bytes;
  uint32_t box_inner, box_outer;
  int elem_bytes;  // 4: fp32, else bf16
  bool operator==(const TensorMapKey &o) const {
    return ptr == o.ptr && inner == o.inner && outer == o.outer && stride_bytes == o.stride_bytes &&
           box_inner == o.box_inner && box_outer == o.box_outer && elem_bytes == o.elem_bytes;
  }
};
struct TensorMapKeyHash {
  size_t operator()(const TensorMapKey &k) const {
    size_t h = reinterpret_cast<size_t>(k.ptr);
    auto mix = [&h](uint64_t v) { h ^= v + 0x9e3779b97f4a7c15ULL + (h << 6) + (h >> 2); };
    mix(k.inner);
    mix(k.outer);
    mix(k.stride_bytes);
    mix((static_cast<uint64_t>(k.box_inner) << 32) | k.box_outer);
    return h;
  }
};

// Two entries are the same only if every field is (equal hashes are not enough: a map with another tensor's base, stride or
// extent would read that tensor's data, or past its end).
class TensorMapCache {
 public:
  // `encode` may be null (no driver): every lookup then fails. False when the encoder refuses the values.
  bool get(TensorMapEncodeFn encode, const TensorMapKey &key, CUtensorMap *out) {
    std::lock_guard<std::mutex> lock{mu_};
    auto it = maps_.find(key);
    if (it != maps_.end()) {
      *out = it->second;
      return true;
    }
    if (!encode) return false;
    const cuuint64_t dims[2] = {key.inner, key.outer};
    const cuuint64_t strides[1] = {key.stride_bytes};
    const cuuint32_t box[2] = {key.box_inner, key.box_outer};
    const cuuint32_t elem_strides[2] = {1, 1};
    CUtensorMap map;
    if (encode(&map, key.elem_bytes == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
               const_cast<void *>(key.ptr), dims, strides, box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return false;
    if (maps_.size() > 8192) maps_.clear();
    maps_.emplace(key, map);
    *out = map;
    return true;
  }

 private:
  std::mutex mu_;
  std::unordered_map<TensorMapKey, CUtensorMap, TensorMapKeyHash> maps_;
};

// The process's cache and the driver's encoder. Row stride in elements; box_inner elements are 128 bytes.
bool get_tensor_map(const void *ptr, uint64_t inner, uint64_t outer, uint64_t stride_elems, uint32_t box_inner,
                    uint32_t box_outer, CUtensorMap *out, int elem_bytes = 2);
}  // namespace cs::kernels
