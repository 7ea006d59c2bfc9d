// core_rows.cuh -- walking the bitmaps over core-local ids (CoreRows in stages.h).
#pragma once
#include "device_util.cuh"
#include "stages.h"

using cds::CoreBand;
using cds::CoreRows;

__device__ __forceinline__ CoreBand band_of(const CoreRows &r, uint32_t v) {
  return r.band[r.of_vertex ? r.of_vertex[v] : 0u];
}

// Words of the rows dealt to warps, `per` of them (up to 32) at a time, and every
// word that is not empty handed to its warp as f(a, band, word of the row, bits).
template <class F>
__device__ __forceinline__ void each_word(const CoreRows &r, uint32_t ncore, const uint32_t *core_vertex,
                                          const uint32_t *bits, F &&f) {
  const uint64_t total = (uint64_t)ncore * r.words, warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  const uint32_t per = (uint32_t)(total / warps >= 32 ? 32 : total / warps ? total / warps : 1);
  for (uint64_t x0 = ((uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * per; x0 < total;
       x0 += warps * per) {
    uint32_t m = 0;
    const uint64_t x = x0 + lane_id();
    if (lane_id() < per && x < total) {
      const uint32_t a = (uint32_t)(x / r.words), w = (uint32_t)(x % r.words);
      const CoreBand bd = band_of(r, core_vertex[a]);
      if (w < bd.width && w >= ((a - bd.lid) >> 5)) m = bits[bd.word + (a - bd.lid) * bd.width + w];
    }
    for (uint32_t on = __ballot_sync(CDS_FULL, m != 0); on; on &= on - 1) {
      const uint32_t l = __ffs(on) - 1;
      const uint32_t a = (uint32_t)((x0 + l) / r.words), w = (uint32_t)((x0 + l) % r.words);
      f(a, band_of(r, core_vertex[a]), w, __shfl_sync(CDS_FULL, m, l));
    }
  }
}

