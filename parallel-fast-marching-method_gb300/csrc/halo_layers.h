// halo_layers.h -- which layer of a halo column a step of the main sweep reads.
#pragma once

#include "stencil.cuh"

namespace fm3dt {

// Step t reads a halo column's layer t - late, counted from the bottom; false
// where the grid has no such layer (before the column's first step, and in the
// sweep's last steps, when only layers read before are still in use): a copy
// there would leave the event's field.
FM_HD bool halo_layer_in(int t, int late, int nnr) { return (unsigned)(t - late) < (unsigned)nnr; }

}  // namespace fm3dt
