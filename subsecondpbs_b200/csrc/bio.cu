// Biological maps on top of the physical dose. CarbonPBS accumulates, per voxel,
// the dose-weighted linear-quadratic parameters of its point-kernel dose
// (cuCalFinalDoseAndRBEKernel, carbonPBS/deviceCalDose.cu:587-736, alpha and
// sqrt(beta) weighted by dose, LET by dose) and turns them into RBE maps
// (LQRBEKernel :738-772, mkmRBEMapKernel :1060-1126). Here the factors ride on the
// pencil-beam pipeline: bio_channel_kernel scales every step's IDD by the step's
// factor (alpha, sqrt(beta), z1D or LET at the step's water-equivalent depth),
// the scaled IDD is superposed with the dose's own radii and work list and
// transferred like the dose, and bio_map_kernel evaluates the maps per voxel.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "kernels.h"
#include "../../include/subsecondpbs.h"

namespace pbs {

namespace {

// Value of a [n] table at fractional index x, clamped to the table.
__device__ __forceinline__ float table_at(const float* __restrict__ t, int n, float x) {
    x = fminf(fmaxf(x, 0.0f), float(n - 1));
    const float f = floorf(x);
    const int i0 = int(f), i1 = min(i0 + 1, n - 1);
    const float a = __ldg(t + i0), b = __ldg(t + i1);
    return a + (b - a) * (x - f);
}

// LET of a step: dose-averaged over the depth samples of the layer's row. `row(i)` is the
// row's value at depth sample i; depths are in samples of the table.
template <typename Row>
__device__ __forceinline__ float step_let(const BioDev& m, float weq, float spacing, float perDepth, Row row) {
    const float last = float(m.letDepths - 1), half = 0.5f * float(m.letSamples - 1);
    float s1 = 0.0f, s2 = 0.0f;
#pragma unroll 2
    for (int j = 0; j < m.letSamples; ++j) {
        const float depth = weq + m.rangeShifter + (float(j) - half) * spacing;
        const float x = fminf(fmaxf((depth - m.letDepth0) * perDepth, 0.0f), last);
        const float f = floorf(x);
        const int i0 = int(f);
        const float a = row(i0), b = row(min(i0 + 1, m.letDepths - 1));
        const float t = a + (b - a) * (x - f);
        s1 += t;
        s2 += t * t;
    }
    return s1 > 0.0f ? s2 / s1 : 0.0f;
}

// Longest LET row that a block keeps in shared memory.
constexpr int kMaxSharedDepths = 48 * 1024 / 4;

// One chunk of layers: out = (idd * factor of `channel`, rSigma) for the sources of the
// live tiles, the only ones the superposition reads (channel 0: alpha (LQ) or z1D (MKM), 1:
// sqrt(beta) (LQ), 2: LET). A block takes one layer (blockIdx.y), whose LET row, between
// two of the table's, it works out first; one warp per (step, tile), lane = column. Bound
// by the instructions of the LET samples. Over every source of every step, live or not,
// with the table's two rows read for each sample, it took 185 us in place of 86 us
// (12 layers, 96 x 96 rays, 128 steps, 5 samples). A row too long for shared memory is
// interpolated where it is read.
template <bool SharedRow>
__global__ void __launch_bounds__(256)
bio_channel_kernel(BeamGeomDev g, BioDev m, int layer0, const float2* __restrict__ sources,
                   const uint8_t* __restrict__ codes, const float* __restrict__ wepl,
                   const LayerStateDev* __restrict__ ls, const BeamStateDev* __restrict__ beam,
                   const float* __restrict__ layerRow, int channel, float2* __restrict__ out) {
    extern __shared__ float sRow[];
    const int lane = threadIdx.x & 31;
    const int l = layer0 + blockIdx.y;
    const float at = fminf(fmaxf(layerRow[l], 0.0f), float(m.letRows - 1));
    const int r0 = int(floorf(at));
    const float ar = at - float(r0);
    const float* t0 = m.letTable + static_cast<size_t>(r0) * m.letDepths;
    const float* t1 = m.letTable + static_cast<size_t>(min(r0 + 1, m.letRows - 1)) * m.letDepths;
    const auto table = [&](int i) {
        const float a = __ldg(t0 + i);
        return a + (__ldg(t1 + i) - a) * ar;
    };
    if (SharedRow) {
        for (int i = threadIdx.x; i < m.letDepths; i += blockDim.x) sRow[i] = table(i);
        __syncthreads();
    }
    const auto row = [&](int i) { return SharedRow ? sRow[i] : table(i); };
    const float spacing = m.estDimension / float(m.letSamples), perDepth = 1.0f / m.letDepthStep;

    const int tiles = g.tilesX * g.tilesY;
    const int rayPlane = g.rayX * g.rayY;
    const int first = beam->firstInside;
    const int perLayer = min(g.steps, ls[l].afterLast - first) * tiles;
    const size_t base = static_cast<size_t>(blockIdx.y) * g.steps * tiles;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < perLayer; i += int(gridDim.x * blockDim.x) >> 5) {
        if (!(codes[base + i] & 0x80)) continue;
        const int zr = i / tiles, tile = i - zr * tiles;
        const int x = tile % g.tilesX * kTileX + lane, y0 = tile / g.tilesX * kTileY;
        const float* weq = wepl + static_cast<size_t>(first + zr) * rayPlane + y0 * g.rayX + x;
        const size_t s0 = (base + i) * kTileSources + lane;
#pragma unroll 4
        for (int r = 0; r < kTileY; ++r) {
            float2 v = make_float2(0.0f, 0.0f);
            if (x < g.rayX && y0 + r < g.rayY) {
                v = sources[s0 + r * kTileX];
                const float d = v.x;
                v.x = 0.0f;
                if (d > 0.0f) {
                    const float let = step_let(m, weq[r * g.rayX], spacing, perDepth, row);
                    float f = let;
                    if (channel < 2) {
                        const float li = let > 0.0f ? (log10f(let) - m.lqLog0) / m.lqLogStep : 0.0f;
                        if (m.model == PBS_BIO_MKM)
                            f = table_at(m.z1d, m.nLq, li);
                        else
                            f = channel == 0 ? table_at(m.alpha, m.nLq, li)
                                             : sqrtf(fmaxf(table_at(m.beta, m.nLq, li), 0.0f));
                    }
                    v.x = d * f;
                }
            }
            out[s0 + r * kTileX] = v;
        }
    }
}

// Maps from the FP64 accumulators (dose, dose * channel 0, 1, 2).
__global__ void bio_map_kernel(const double* __restrict__ dose, const double* __restrict__ c0,
                               const double* __restrict__ c1, const double* __restrict__ c2, size_t n, BioDev m,
                               int map, float* __restrict__ out) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
        const double d = dose[i];
        double v = 0.0;
        if (map == PBS_BIO_MAP_DOSE) {
            v = d;
        } else if (map == PBS_BIO_MAP_LETD) {
            v = d > 0.0 ? c2[i] / d : 0.0;
        } else if (map == PBS_BIO_MAP_ALPHA) {
            v = d > 0.0 ? c0[i] / d : 0.0;
        } else if (map == PBS_BIO_MAP_BETA) {
            const double sb = d > 0.0 ? c1[i] / d : 0.0;
            v = sb * sb;
        } else if (map == PBS_BIO_MAP_Z1D) {
            const double z = d > 0.0 ? c0[i] / d : 0.0;
            v = 0.172 + double(m.beta0) * z;
        } else {  // RBE or RBE x dose
            double rbe = 1.0;
            if (m.model == PBS_BIO_MKM) {
                // mkmRBEMapKernel (deviceCalDose.cu:1060-1126): the photon dose of equal
                // effect over the ion dose, 1 at or below 1e-3 Gy.
                const double z = d > 0.0 ? c0[i] / d : 0.0;
                const double a = 0.172 + double(m.beta0) * z;
                const double b0 = double(m.beta0), t2 = double(m.alpha0) / 2.0 / b0;
                const double dx = -t2 + sqrt(t2 * t2 + (a * d + b0 * d * d) / b0);
                rbe = d > 1e-3 ? dx / d : 1.0;
            } else {
                // LQRBEKernel (deviceCalDose.cu:738-772): 3.988565 Gy over the ion dose of
                // 10 % survival, 1 where the dose, alpha or beta vanishes.
                if (d != 0.0 && c0[i] != 0.0 && c1[i] != 0.0) {
                    const double a = c0[i] / d;
                    const double sb = c1[i] / d, b = sb * sb;
                    const double d10 = (-a + sqrt(a * a - 4.0 * -2.302585 * b)) / b * 0.5;
                    rbe = 3.988565 / d10;
                }
            }
            v = map == PBS_BIO_MAP_RBE ? rbe : rbe * d;
        }
        out[i] = float(v);
    }
}

}  // namespace

cudaError_t launch_bio_channel(const BeamGeomDev& g, const BioDev& m, int layer0, int nLayers, const float2* sources,
                               const uint8_t* codes, const float* wepl, const LayerStateDev* ls,
                               const BeamStateDev* beam, const float* layerRow, int channel, float2* out,
                               cudaStream_t s) {
    // Layers in the grid's y dimension, at most 65535 of them; about 16 blocks per SM.
    const int perLayer = (g.steps * g.tilesX * g.tilesY + 7) / 8;
    const dim3 grid(std::max(1, std::min(perLayer, (148 * 16 + nLayers - 1) / nLayers)), nLayers);
    const bool fits = m.letDepths <= kMaxSharedDepths;
    const auto kernel = fits ? bio_channel_kernel<true> : bio_channel_kernel<false>;
    kernel<<<grid, 256, fits ? m.letDepths * sizeof(float) : 0, s>>>(g, m, layer0, sources, codes, wepl, ls, beam,
                                                                     layerRow, channel, out);
    return cudaGetLastError();
}

cudaError_t launch_bio_map(const double* dose, const double* c0, const double* c1, const double* c2, size_t n,
                           const BioDev& m, int map, float* out, cudaStream_t s) {
    const int blocks = int(std::min<size_t>((n + 255) / 256, 148 * 16));
    bio_map_kernel<<<blocks, 256, 0, s>>>(dose, c0, c1, c2, n, m, map, out);
    return cudaGetLastError();
}

__global__ void reset_work_claims_kernel(BeamStateDev* beam) {
    beam->workNext = 0;
    beam->workNextSmall = 0;
    beam->workNextTiny = 0;
}

cudaError_t launch_reset_work_claims(BeamStateDev* beam, cudaStream_t s) {
    reset_work_claims_kernel<<<1, 1, 0, s>>>(beam);
    return cudaGetLastError();
}

}  // namespace pbs
