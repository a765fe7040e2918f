// Whether a default form's smaller tiles, which hand over more edges than the nominal
// tiling's, would crowd out the angular flux and the expanded source (`fluxes` bytes at
// most): more than half of what the device can give the handle.  That is the memory
// free now and what the handle holds of these buffers already, so the answer is the
// same before and after its first sweep.
#pragma once

#include <cstddef>

namespace ouranos {

inline bool edges_crowd(size_t edges, size_t nominal_edges, size_t fluxes, size_t free_now, size_t held) {
  return edges > nominal_edges && edges + fluxes > (free_now + held) / 2;
}

}  // namespace ouranos
