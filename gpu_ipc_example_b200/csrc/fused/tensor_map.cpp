// Tensor maps of the GEMM kernels' operands.
#include "tensor_map.h"

#include <deque>
#include <map>
#include <mutex>
#include <tuple>

#include "../common/check.h"
#include "../common/cu_driver.h"

namespace b200ipc {
namespace {

// Tensor maps depend only on (pointer, extents, box, type): weights and activation buffers are
// reused call after call, so encoding is done once per distinct operand.  The cache is bounded: when
// it is full the oldest entry makes room (never a wholesale clear in the middle of serving).
using MapKey = std::tuple<const void*, uint64_t, uint64_t, uint32_t, int>;
constexpr size_t kMaxCachedMaps = 4096;
std::mutex g_enc_mu;
std::map<MapKey, CUtensorMap> g_maps;
std::deque<MapKey> g_map_order;
}  // namespace

void encode_tile_map(CUtensorMap* map, DType t, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows) {
  const MapKey key(base, rows, cols, box_rows, int(t));
  {
    std::lock_guard<std::mutex> lk(g_enc_mu);
    auto it = g_maps.find(key);
    if (it != g_maps.end()) {
      *map = it->second;
      return;
    }
  }
  B200_REQUIRE((reinterpret_cast<uintptr_t>(base) & 15) == 0, "GEMM operands must be 16-byte aligned");
  B200_REQUIRE((cols * 2) % 16 == 0, "the K extent must be a multiple of 8 elements");
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {cols * 2};
  cuuint32_t box[2] = {uint32_t(kTileMapCols), box_rows};
  cuuint32_t estr[2] = {1, 1};
  B200_CU_CHECK(cu().TensorMapEncodeTiled(map, t == DType::F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                                          2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
  std::lock_guard<std::mutex> lk(g_enc_mu);
  if (g_maps.emplace(key, *map).second) {
    g_map_order.push_back(key);
    if (g_map_order.size() > kMaxCachedMaps) {
      g_maps.erase(g_map_order.front());
      g_map_order.pop_front();
    }
  }
}

}  // namespace b200ipc
