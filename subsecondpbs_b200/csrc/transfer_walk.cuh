// How the transfer kernels (BEV -> dose, its transpose, and the influence columns) walk a
// box of dose voxels.
//
// A warp takes a patch of voxels of one z chunk. Where the beam runs along y or z the
// patch is 32 voxels along x, whose BEV samples lie side by side in one plane. Where it
// runs along x those 32 voxels would sample 32 planes, a 128-byte line each for every one
// of the eight texels; a patch of 4 x 8 samples 4 planes in rows of 8, and still reads and
// writes the dose in whole 32-byte sectors. Beams along x: 256 x 256 x 160 voxels
// 27 -> 17 us, 512 x 512 x 200 515 -> 187 us (this change alone).
#pragma once

#include "pbs_types.h"

namespace pbs {

// BEV planes per voxel in x above which the patch is 4 x 8.
constexpr float kAcrossPlanes = 0.25f;

// Calls f(x, y, chunk) for the voxel columns [lo, lo + n) in x and y and the z chunks
// [0, chunks), each by one lane. The blocks of the grid's x dimension share the box.
template <typename F>
__device__ __forceinline__ void walk_box(const TransferParams& t, int lox, int loy, int nx, int ny, int chunks, F f) {
    const bool across = fabsf(t.coefIdxI.z) > kAcrossPlanes;
    const int shift = across ? 2 : 5;
    const int lane = threadIdx.x & 31;
    const int px = (nx + (1 << shift) - 1) >> shift, py = (ny + (32 >> shift) - 1) >> (5 - shift);
    // Patches that share BEV lines follow one another: along y for the 4 x 8 patch.
    const int inner = across ? py : px, outer = across ? px : py;
    const long long patches = static_cast<long long>(px) * py * chunks;
    const int warps = static_cast<int>(gridDim.x * blockDim.x) >> 5;
    for (long long w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < patches; w += warps) {
        const int i = static_cast<int>(w % inner);
        const long long r = w / inner;
        const int o = static_cast<int>(r % outer);
        const int x = ((across ? o : i) << shift) + (lane & ((1 << shift) - 1));
        const int y = ((across ? i : o) << (5 - shift)) + (lane >> shift);
        if (x < nx && y < ny) f(lox + x, loy + y, static_cast<int>(r / outer));
    }
}

}  // namespace pbs
