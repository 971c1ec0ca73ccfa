// Clearance map of a geometry (see clearance.cu): built on the device when the
// geometry is set, used by the transport to skip the octree walk of steps that
// cannot meet a triangle.
#pragma once

#include <cuda_runtime.h>

#include "dev_types.h"

namespace nbx {

struct ClearanceMap {
    dev::Clearance map{};   // what the kernels take; map.top == nullptr: no map
    void* memory = nullptr;   // the device allocation behind it
    size_t bytes = 0;         // its size
};

// Builds the map of `n_tri` triangles (three float4 each, device memory) over
// the octree's root box.  Without memory for it the call succeeds with an empty
// map (the transport then walks every step); every other error is returned.
cudaError_t build_clearance(const float4* tri, int n_tri, const float center[3], const float half[3], int sms,
                            cudaStream_t s, ClearanceMap* out);
void free_clearance(ClearanceMap* m);

}  // namespace nbx
