// Small device helpers shared by several kernels.
#pragma once

#include <cuda_runtime.h>

namespace pbs {

// Programmatic dependent launch: a kernel launched with launch_pdl calls pdl_wait()
// first (its predecessor on the stream has completed and its writes are visible); a
// kernel that may precede one calls pdl_trigger() to let it be scheduled early.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// tex1D with linear filtering, clamp addressing and unnormalised coordinates
// (texel i centred at i + 0.5), evaluated with full-precision weights. The texel
// coordinate is clamped to [0, n - 1] before the split into index and weight: below
// the table and past its end the filter returns the edge texel either way (the two
// taps coincide or the weight is 0), and a NaN coordinate gives texel 0.
__device__ __forceinline__ float lut_linear_clamp(const float* __restrict__ t, int n, float x) {
    const float xb = fminf(fmaxf(x - 0.5f, 0.0f), float(n - 1));
    const float fl = floorf(xb);
    const int i0 = int(fl);
    const int i1 = min(i0 + 1, n - 1);
    const float a = xb - fl;
    const float v0 = __ldg(t + i0), v1 = __ldg(t + i1);
    return v0 + (v1 - v0) * a;
}

// Unsigned key with the order of the float values (negative floats reversed).
__device__ __forceinline__ unsigned float_order_key(float v) {
    const unsigned b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float float_from_order_key(unsigned k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// A tile's range of rSigma as one word: the upper bound in the high half, the lower one
// in the low half, each the top 16 bits of the positive float below its sign (2^-8
// relative, rounded outwards); 0 is no depositing source.
__device__ __forceinline__ unsigned range_word(int loBits, int hiBits) {
    const unsigned hi = min(static_cast<unsigned>(hiBits) + 0x7fffu, 0x7fffffffu);  // (NaN: 0xffff)
    return max(__byte_perm(static_cast<unsigned>(max(loBits, 0)) << 1, hi << 1, 0x7632), 0x10000u);
}
__device__ __forceinline__ unsigned merge_range(unsigned a, unsigned b) {
    if (!a || !b) return a | b;
    return max(a >> 16, b >> 16) << 16 | min(a & 0xffffu, b & 0xffffu);
}

// Same lookup on a table staged in shared memory.
__device__ __forceinline__ float lut_linear_clamp_smem(const float* t, int n, float x) {
    const float xb = fminf(fmaxf(x - 0.5f, 0.0f), float(n - 1));
    const float fl = floorf(xb);
    const int i0 = int(fl);
    const int i1 = min(i0 + 1, n - 1);
    const float a = xb - fl;
    const float v0 = t[i0], v1 = t[i1];
    return v0 + (v1 - v0) * a;
}

// The same on a table in shared memory whose last entry is stored twice.
__device__ __forceinline__ float lut_linear_clamp_padded(const float* t, int n, float x) {
    const float xb = fminf(fmaxf(x - 0.5f, 0.0f), float(n - 1));
    const float fl = floorf(xb);
    const int i = int(fl);
    const float a = xb - fl;
    const float v0 = t[i], v1 = t[i + 1];
    return v0 + (v1 - v0) * a;
}

// Radius bucket of a tile from its minimum rSigmaEff (complete_superposition.cu:242):
// min(int(3 / (sqrt(2) * min) + 0.5), 33), with IEEE division.
__device__ __forceinline__ int tile_radius_bucket(float minRSigma) {
    const float q = __fadd_rn(__fdiv_rn(3.0f, __fmul_rn(1.41421354f, minRSigma)), 0.5f);
    if (!(q < 34.0f)) return (q != q) ? 0 : 33;
    return min(int(q), 33);
}

// Calls f(x, y, z) for the cells of a box of w x rows x planes: a warp takes a row at a
// time, so that a cell costs no division (with one 64-bit division per axis and cell,
// clearing 64 influence columns took 64 us in place of 34 us).
template <typename F>
__device__ __forceinline__ void walk_rows(int w, int rows, int planes, F f) {
    const unsigned warps = gridDim.x * blockDim.x >> 5, n = static_cast<unsigned>(rows) * planes;
    const int lane = threadIdx.x & 31;
    for (unsigned r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n; r += warps) {
        const int z = static_cast<int>(r / rows), y = static_cast<int>(r - static_cast<unsigned>(z) * rows);
        for (int x = lane; x < w; x += 32) f(x, y, z);
    }
}

}  // namespace pbs
