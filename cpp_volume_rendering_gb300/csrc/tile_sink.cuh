// tile_sink.cuh — the network's input tile as a sink of sur_features.
#pragma once

#include "mlp_tile.cuh"

namespace cvr {

// Packs features pairwise to BF16 and stores each 8-feature chunk of this
// thread's row of the input tile as soon as it is complete.
struct TileSink {
  uint8_t* tile;
  int row;
  uint32_t w[4];
  float lo;
  __device__ __forceinline__ void operator()(int k, float v) {
    if (k & 1) {
      w[(k >> 1) & 3] = pack_bf16(lo, v);
      if ((k & 7) == 7) store_chunk(tile, row, k >> 3, w[0], w[1], w[2], w[3]);
    } else {
      lo = v;
    }
  }
};

}  // namespace cvr
