// Light buffer and direction buffer construction (light_buffer.cu): per point
// light, the spheres that can block a shadow ray in each direction cell
// around the light; per sphere, the spheres a ray leaving it can hit in each
// direction cell.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "wavefront.h"

namespace atx {

// Device bytes cells_build needs for the light buffer of nl lights, and for
// the direction buffer of n spheres, at res cells along a face's edge and
// line_words 16-bit words per cell (kLbLine, or kBvhLine for LBVH scenes).
uint64_t lb_bytes(uint32_t nl, uint32_t res, uint32_t line_words = kLbLine);
uint64_t db_bytes(uint32_t n, uint32_t res, uint32_t line_words = kLbLine);

// Builds, on stream, for the n spheres sph (cx, cy, cz, r*r) with radii
// radius[], at res cells along a face's edge (kCellResMin..kBvhLightRes):
//   the light buffer of the nl lights (1 <= nl <= kLbMaxLights, n <=
//   kLbMaxSpheres) into lbuf (lb_bytes() of device memory; null: none), *lv
//   its view;
//   the direction buffer (n <= kDbMaxBvhSpheres) into dbuf (db_bytes(); null:
//   none), *dv its view: the cells of spheres db_first.. db_first + db_count - 1
//   of it, so that a large one can be built over several calls.
cudaError_t cells_build(const float4* sph, const float* radius, uint32_t n, const DevLight* lights, uint32_t nl,
                        uint32_t res, uint32_t line_words, void* lbuf, uint64_t lbytes, LightBufferView* lv,
                        void* dbuf, uint64_t dbytes, DirBufferView* dv, cudaStream_t stream, uint32_t db_first = 0,
                        uint32_t db_count = ~0u);

}  // namespace atx
