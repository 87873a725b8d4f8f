// Publication of the call's expert ids: int16 in this rank's routing buffer, behind a header that holds T.
#pragma once
#include "common.cuh"
#include "../../include/dist_moe_b200.h"

namespace dm {

struct IdPublish {
  const void* ids = nullptr;  // null: nothing to publish
  uint8_t* routing = nullptr;
  int64_t n_ids = 0;
  int ids_are_int64 = 0, T = 0, E = 0, validate = 0;
  int* status = nullptr;
};

__device__ __forceinline__ void publish_ids(const IdPublish& p) {
  if (p.ids == nullptr) return;
  const int64_t tid = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  if (tid == 0) *reinterpret_cast<int32_t*>(p.routing) = p.T;
  int16_t* out = reinterpret_cast<int16_t*>(p.routing + DM_ROUTING_HEADER_BYTES);
  for (int64_t i = tid; i < p.n_ids; i += stride) {
    const int64_t v = p.ids_are_int64 ? static_cast<const int64_t*>(p.ids)[i] : static_cast<const int32_t*>(p.ids)[i];
    if (p.validate && (v < -1 || v >= p.E)) set_status(p.status, kInvalidExpertId, static_cast<int>(i), static_cast<int>(v));
    out[i] = static_cast<int16_t>(v);
  }
}

}  // namespace dm
