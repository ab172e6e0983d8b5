// Tensor maps (TMA descriptors) of 2-byte element tensors, encoded once and kept.
#pragma once

#include "aps_common.cuh"

#include <cuda.h>

namespace aps {

// A tiled tensor map with 128-byte swizzle over fp16 / bf16 data.  dims / box: innermost
// first; strides_bytes[i] = byte stride of dimension i + 1.  rank 2 or 3.
struct TensorMapSpec {
  const void* base;
  int dtype;                  // APS_F16 / APS_BF16
  int rank;
  uint64_t dims[3];
  uint64_t strides_bytes[2];
  uint32_t box[3];
};

// A tensor map is a pure function of its spec: the last encoded maps are kept in a small per-thread table (the library
// has one calling thread).  A layer called again and again finds its up to eight maps there; the layers of a model
// called in turn have more than the table holds and encode theirs every time, beside the GPU's work: 40 OPT-13B
// layers of one request each in turn 57 us a layer, one layer 58; 24 OPT-1.3B layers of eight requests 43 and 43.
int cached_tensor_map(CUtensorMap* out, const TensorMapSpec& spec, const char* what);

}  // namespace aps
