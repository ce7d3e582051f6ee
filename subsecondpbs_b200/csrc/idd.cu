// Per-layer integrated depth dose and effective sigma along every ray, fused with the
// per-tile radius reduction and the per-layer radius histogram, followed by the
// device-side batching (one small CTA) and the radius-sorted work-list scatter.
#include <float.h>
#include <limits.h>

#include <algorithm>

#include "device_util.cuh"
#include "kernels.h"
#include "launch_util.h"

namespace pbs {

namespace {

constexpr float kPInv = 0.5649718f;   // 1/p, p = 1.77 (raytracedicom_integration.h:22)
constexpr float kECoef = 8.639415f;   // (10 alpha)^(-1/p) (raytracedicom_integration.h:23)
constexpr float kSqrt2 = 1.41421356f;
constexpr int kMaxChunkLayers = 64;

// Divisions in the per-step walk use the approximate reciprocal (within 2 ulp): the IEEE
// quotient's range check and slow path cost more ALU and branch issue than the rest of
// a step's arithmetic. The forms here leave out the scaling of subnormal operands, which
// would cost the kernel 2 %: energies and widths are none, and a dose of less than
// 2^-126 per unit mass, flushed to 0, is at the end of the superposition's fixed point (2^-120).
// The tile radius bucket keeps its IEEE division (tile_radius_bucket).
__device__ __forceinline__ float div_normal(float a, float b) {
    float q;
    asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(q) : "f"(a), "f"(b));
    return q;
}
__device__ __forceinline__ float pow_normal(float x, float y) {
    float l, r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y * l));
    return r;
}

// One CTA = one 32x8 tile of rays for one layer. Each thread walks its ray from the
// beam's first-inside step to the layer's cut-off step (fillIddAndSigmaKernel,
// idd_sigma.cu:46-259). After every step each warp reduces min(rSigmaEff) and
// the largest rSigmaEff with idd > 0 over its 32 rays into shared memory; once the walk is done the CTA
// turns the eight warp partials of every step into the tile's radius bucket
// (tileRadCalc, complete_superposition.cu:198-255), stores the code and, for a live
// tile, its range of rSigma (the superposition's interpolation range), and adds the
// tile's bucket counts to the layer histogram.
// Profile table value of channel c at a fractional depth and row index, both
// already clamped to the table: the linear filter of the reference's profile
// texture (wrapper.cu:2858-2860, unnormalised coordinates at texel centres) with
// exact weights.
__device__ __forceinline__ float profile_sample(const float* __restrict__ t, int depthN, int channels, int rows,
                                                int c, float depth, float row) {
    const float fd = floorf(depth), fr = floorf(row);
    const int d0 = int(fd), r0 = int(fr);
    const int d1 = min(d0 + 1, depthN - 1), r1 = min(r0 + 1, rows - 1);
    const float ad = depth - fd, ar = row - fr;
    auto at = [&](int r, int d) { return __ldg(t + (static_cast<size_t>(r) * depthN + d) * channels + c); };
    const float a0 = at(r0, d0), a1 = at(r0, d1), b0 = at(r1, d0), b1 = at(r1, d1);
    const float lo = a0 + (a1 - a0) * ad, hi = b0 + (b1 - b0) * ad;
    return lo + (hi - lo) * ar;
}

template <bool kNuclear, bool kProfile>
__global__ void __launch_bounds__(256)
idd_kernel(BeamGeomDev g, LutsDev luts, int layer0, const float2* __restrict__ material,
           const float* __restrict__ wepl, const int* __restrict__ firstInside, const int* __restrict__ firstOutside,
           const float* __restrict__ rayW, const LayerParamsDev* __restrict__ lp, LayerStateDev* __restrict__ ls,
           const BeamStateDev* __restrict__ beam, float2* __restrict__ sources, unsigned* __restrict__ tileRange,
           uint8_t* __restrict__ codes, int* __restrict__ firstPassiveOut, const int* __restrict__ rayToNuc,
           const float* __restrict__ lattice, float2* __restrict__ nucSources) {
    extern __shared__ float smem[];
    float* ciddRow = smem;                                    // [nS + 1], the last entry twice
    float* nucWRow = ciddRow + luts.nS + 1;                   // [nS] with the nuclear halo
    float* nucSRow = nucWRow + (kNuclear ? luts.nS : 0);      // [nS] with the nuclear halo
    // [steps] (0.5 (voxel width x + y), step volume)
    float2* stepGeo = reinterpret_cast<float2*>(ciddRow + (((kNuclear ? 3 : 1) * luts.nS + 2) & ~1));
    float* partMin = reinterpret_cast<float*>(stepGeo + g.steps);              // [steps][8]
    unsigned* partRange = reinterpret_cast<unsigned*>(partMin + g.steps * 8);  // [steps][8]
    __shared__ int shHist[kBuckets], shLive[kBuckets], shPassive[8], shEnd;

    // Longest walks first: the layers are dispatched from the end of the chunk whose
    // cut-off step is deeper, so that the long CTAs do not form the grid's tail.
    const int nl = int(gridDim.z);
    const bool deepLast = ls[layer0].afterLast < ls[layer0 + nl - 1].afterLast;
    const int lc = deepLast ? nl - 1 - int(blockIdx.z) : int(blockIdx.z);
    const int l = layer0 + lc;
    const int tx = blockIdx.x, ty = blockIdx.y;
    const int lane = threadIdx.x, warp = threadIdx.y;
    const int tid = warp * 32 + lane;
    const int x = tx * kTileX + lane, y = ty * kTileY + warp;
    const LayerParamsDev p = lp[l];
    const int first = beam->firstInside;
    const int afterLastL = ls[l].afterLast;

    const bool real = x < g.rayX && y < g.rayY;
    const size_t rayPlane = static_cast<size_t>(g.rayX) * g.rayY;
    const size_t padPlane = static_cast<size_t>(g.pitchX) * g.pitchY;
    const size_t layerStride = static_cast<size_t>(g.steps) * padPlane;
    // This thread's source of the tile (tile-major planes).
    float2* srcL = sources + lc * layerStride + static_cast<size_t>(ty * g.tilesX + tx) * kTileSources + tid;
    const size_t ridx = static_cast<size_t>(y) * g.rayX + x;

    int firstIn = 0;
    unsigned int afterLast = 0;
    float rayWeight = 0.0f;
    bool live = false;
    if (real) {
        firstIn = firstInside[ridx];
        afterLast = static_cast<unsigned int>(min(firstOutside[ridx], afterLastL));
        rayWeight = rayW[static_cast<size_t>(l) * rayPlane + ridx];
        live = true;
        if (rayWeight < 1e-6f || afterLast < static_cast<unsigned int>(first)) {
            live = false;
            afterLast = 0;
        }
    }
    // No live ray: every step's bucket is 0 and nothing reads the tile's sources.
    if (!__syncthreads_or(live) && !g.fillDeadTiles) {
        const int nSteps = max(afterLastL - first, 0);
        const size_t tiles = static_cast<size_t>(g.tilesX) * g.tilesY;
        uint8_t* code = codes + static_cast<size_t>(lc) * g.steps * tiles + static_cast<size_t>(ty) * g.tilesX + tx;
        for (int zr = tid; zr < nSteps; zr += 256) code[zr * tiles] = 0;
        if (real && firstPassiveOut) firstPassiveOut[static_cast<size_t>(lc) * rayPlane + ridx] = 0;
        if (tid == 0) {
            if (nSteps > 0) atomicAdd(&ls[l].histAll[0], nSteps);
            atomicMax(&ls[l].maxFirstPassive, 0);
        }
        return;
    }

    // CIDD row of this layer's energy: the bilinear CIDD texture lookup at a fixed
    // energy coordinate is a depth lerp of the energy-interpolated row.
    {
        float eb = p.energyIdx;  // (energyIdx + 0.5) - 0.5 texel offset
        eb = fminf(fmaxf(eb, -1.0f), float(luts.nE));
        const float fl = floorf(eb);
        const float b = eb - fl;
        const int e0 = min(max(int(fl), 0), luts.nE - 1);
        const int e1 = min(max(int(fl) + 1, 0), luts.nE - 1);
        const float* r0 = luts.cidd + static_cast<size_t>(e0) * luts.nS;
        const float* r1 = luts.cidd + static_cast<size_t>(e1) * luts.nS;
        for (int d = tid; d <= luts.nS; d += 256) {
            const int i = min(d, luts.nS - 1);
            const float a0 = __ldg(r0 + i), a1 = __ldg(r1 + i);
            ciddRow[d] = a0 + (a1 - a0) * b;
        }
        if (kNuclear) {
            // Nuclear weight and sigma^2 tables share the CIDD axes (energy_reader.cpp:135-182).
            const float* w0 = luts.nucWeight + static_cast<size_t>(e0) * luts.nS;
            const float* w1 = luts.nucWeight + static_cast<size_t>(e1) * luts.nS;
            const float* q0 = luts.nucSqSigma + static_cast<size_t>(e0) * luts.nS;
            const float* q1 = luts.nucSqSigma + static_cast<size_t>(e1) * luts.nS;
            for (int d = tid; d < luts.nS; d += 256) {
                const float a0 = __ldg(w0 + d), a1 = __ldg(w1 + d);
                nucWRow[d] = a0 + (a1 - a0) * b;
                const float c0 = __ldg(q0 + d), c1 = __ldg(q1 + d);
                nucSRow[d] = c0 + (c1 - c0) * b;
            }
        }
        // Per-step voxel widths and volumes are the same for every ray of the step
        // (fill_idd_and_sigma_params.cuh:56-80).
        for (int k = tid; k < g.steps; k += 256) {
            const float zk = g.fanCorner.z + float(k) * g.fanDelta.z;
            const float vwx = g.fanDelta.x * (1.0f - zk / g.sourceDist.x);
            const float vwy = g.fanDelta.y * (1.0f - zk / g.sourceDist.y);
            const unsigned int ku = static_cast<unsigned int>(k);
            stepGeo[k] = make_float2(0.5f * (vwx + vwy),
                                     g.volConst + float(ku) * g.volLin + float(ku * ku) * g.volSq);
        }
        if (tid < kBuckets) {
            shHist[tid] = 0;
            shLive[tid] = 0;
        }
        if (tid == 0) shEnd = first;
    }
    __syncthreads();

    // Nuclear halo of this ray (idd_sigma.cu:88-98, 131-142): only rays under a
    // halo lattice cell carry a halo value; the cell's raw spot weight is its
    // weight. Every ray's primary dose keeps the (1 - nuclear weight) share.
    const bool nucOn = kNuclear && p.spotDist > 0.0f;
    int nucIdx = -1;  // the cell's source in the halo's tile-major planes
    float nucRayWeight = 0.0f;
    if (nucOn && real) {
        const int cell = rayToNuc[ridx];
        if (cell >= 0) {
            const int cx = cell % g.nucX, cy = cell / g.nucX;
            nucRayWeight = lattice[(static_cast<size_t>(l) * g.latNy + cy) * g.latNx + cx];
            nucIdx = ((cy / kTileY) * (g.nucX / kTileX) + cx / kTileX) * kTileSources + (cy % kTileY) * kTileX +
                     cx % kTileX;
        }
    }
    const size_t nucPlane = static_cast<size_t>(g.nucX) * g.nucY;
    float2* nucL = nucSources + lc * static_cast<size_t>(g.steps) * nucPlane;
    const float spotDist = p.spotDist;
    const float entrySigmaSq = ls[l].entrySigmaSq;
    const float eRefSq = nucOn ? g.eRefSq : 198.81f;
    const float sigmaDelta = nucOn ? g.sigmaDelta : 0.21f;
    const bool suppressDip = nucOn && g.suppressDistalDip;

    const float stepLength = fabsf(g.fanDelta.z);
    const float quad = p.sigmaSqAirQuad;
    float cumulSpOld = 0.0f, cumulDoseOld = 0.0f;
    float incScat = 0.0f, incincScat = 0.0f;
    float incDiv = p.sigmaSqAirLin + (2.0f * float(first) - 1.0f) * quad;
    float sigmaSq = -incDiv;

    // WEPL and material are loaded two steps ahead: where few tiles leave the SMs to one
    // CTA each, a step waits for its loads (3 layers of 96 x 72 rays, 235 steps: 96 us with
    // one step, 78 with two, three and four; full chips are as fast with one). One ahead
    // with the halo, whose registers would cost a CTA per SM (400 against 408 us).
    constexpr int kIddAhead = kNuclear ? 1 : 2;
    const float* nextW = wepl + static_cast<size_t>(first) * rayPlane + ridx;
    const float2* nextM = material + static_cast<size_t>(first) * rayPlane + ridx;
    float aheadSp[kIddAhead];
    float2 aheadMat[kIddAhead];
#pragma unroll
    for (int i = 0; i < kIddAhead; ++i) {
        aheadSp[i] = 0.0f;
        aheadMat[i] = make_float2(0.0f, 0.0f);
        if (live && first + i < afterLastL) {
            aheadSp[i] = nextW[static_cast<size_t>(i) * rayPlane];
            aheadMat[i] = nextM[static_cast<size_t>(i) * rayPlane];
        }
    }
    nextW += static_cast<size_t>(kIddAhead - 1) * rayPlane;
    nextM += static_cast<size_t>(kIddAhead - 1) * rayPlane;
    float2* dst = srcL;
    float runMax = 0.0f;  // largest IDD of this ray (fixed-point range of the superposition)
    int stepNo = first;
#pragma unroll 2
    for (; stepNo < afterLastL; ++stepNo) {
        // Once no ray of the row is live, every later step is (0, +inf): the fill
        // below writes those without the per-step walk (looked at every fourth step).
        if (!((stepNo - first) & 3) && !__any_sync(0xffffffffu, live)) break;
        float res = 0.0f;
        float rSigmaEff = __int_as_float(0x7f800000);
        float nucRes = 0.0f;
        float nucRSigmaEff = __int_as_float(0x7f800000);
        // WEPL of this step for the profile model (the reference reads the traced
        // value of every step, live or not).
        const float nextProfileSp = kProfile && real ? wepl[static_cast<size_t>(stepNo) * rayPlane + ridx] : 0.0f;
        if (live) {
            const float cumulSp = aheadSp[0];
            const float dens = aheadMat[0].x, rRl = aheadMat[0].y;
#pragma unroll
            for (int i = 0; i + 1 < kIddAhead; ++i) {
                aheadSp[i] = aheadSp[i + 1];
                aheadMat[i] = aheadMat[i + 1];
            }
            if (stepNo + kIddAhead < afterLastL) {
                nextW += rayPlane;
                nextM += rayPlane;
                aheadSp[kIddAhead - 1] = *nextW;
                aheadMat[kIddAhead - 1] = *nextM;
            }
            const float cumulDose = lut_linear_clamp_padded(ciddRow, luts.nS, cumulSp * p.energyScaleFact + 0.5f);
            if (cumulSp < p.peakDepth) {
                const float resE = kECoef * pow_normal(p.peakDepth - 0.5f * (cumulSp + cumulSpOld), kPInv);
                const float betaP = resE + 938.3f - div_normal(938.3f * 938.3f, resE + 938.3f);
                const float thetaSq = div_normal(eRefSq, betaP * betaP) * stepLength * rRl;
                sigmaSq += incScat + incDiv;
                incincScat += 2.0f * thetaSq * stepLength * stepLength;
                incScat += incincScat;
                incDiv += 2.0f * quad;
            } else if (!suppressDip) {
                sigmaSq -= 1.5f * (incScat + incDiv) * dens;
            }
            const float2 geo = stepGeo[stepNo];
            rSigmaEff = div_normal(geo.x, kSqrt2 * (sqrtf(sigmaSq) + sigmaDelta));
            const float mass = dens * geo.y;
            if (nucOn) {
                const float depthMidIdx = 0.5f * (cumulSp + cumulSpOld) * p.energyScaleFact + 0.5f;
                if (mass > 1e-2f) {
                    const float nucWeight = lut_linear_clamp_smem(nucWRow, luts.nS, depthMidIdx);
                    res = div_normal((1.0f - nucWeight) * rayWeight * (cumulDose - cumulDoseOld), mass);
                    if (nucIdx >= 0)
                        nucRes = __fdividef(nucWeight * nucRayWeight * (cumulDose - cumulDoseOld), mass * spotDist * spotDist);
                }
                if (nucIdx >= 0) {
                    const float nucSqSigma = lut_linear_clamp_smem(nucSRow, luts.nS, depthMidIdx);
                    nucRSigmaEff = 0.5f * spotDist * (2.0f * stepGeo[stepNo].x) /
                                   (kSqrt2 * sqrtf(sigmaSq + nucSqSigma + entrySigmaSq));
                }
            } else if (mass > 1e-2f) {
                res = div_normal(rayWeight * (cumulDose - cumulDoseOld), mass);
            }
            cumulSpOld = cumulSp;
            cumulDoseOld = cumulDose;
            if (cumulSp > p.rangeStopDepth || static_cast<unsigned int>(stepNo) == afterLast) {
                live = false;
                afterLast = static_cast<unsigned int>(stepNo);
            }
        }
        if (!live || stepNo < firstIn - 1) {
            res = 0.0f;
            rSigmaEff = __int_as_float(0x7f800000);
            nucRes = 0.0f;
            nucRSigmaEff = __int_as_float(0x7f800000);
        }
        if (kProfile && real) {
            // CarbonPBS lateral profile model on the filled step, in the reference's
            // order: the sigma override (overrideRSigmaFromCarbonProfileKernel,
            // wrapper.cu:2080-2152), then the overall weight
            // (applyCarbonProfileOverallWeightKernel, wrapper.cu:2154-2187).
            const int nGauss = (g.profileChannels - 1) / 2;
            const float depthIdx = (nextProfileSp - g.profileDepth0) / g.profileDepthStep;
            const float dIdx = fminf(fmaxf(depthIdx, 0.0f), float(g.profileDepthN - 1));
            const float rIdx = p.profileRow;
            if (g.profileMode & 1) {
                if (!(res > 0.0f)) {
                    rSigmaEff = __int_as_float(0x7f800000);
                } else {
                    float sumW = 0.0f, sumS2 = 0.0f;
                    for (int gi = 0; gi < nGauss; ++gi) {
                        const float w = profile_sample(g.profile, g.profileDepthN, g.profileChannels, g.profileRows,
                                                       gi, dIdx, rIdx);
                        const float sr = profile_sample(g.profile, g.profileDepthN, g.profileChannels, g.profileRows,
                                                        gi + nGauss, dIdx, rIdx);
                        sumW += w;
                        sumS2 += w * sr * sr;
                    }
                    if (!(sumW > 1.0e-8f)) {
                        rSigmaEff = __int_as_float(0x7f800000);
                    } else {
                        // CarbonPBS geometric depth: distance from the virtual source along
                        // this divergent ray minus the source-to-beam-parameter distance.
                        const float sad = 0.5f * (g.sourceDist.x + g.sourceDist.y);
                        const float fanX = g.fanCorner.x + float(x) * g.fanDelta.x;
                        const float fanY = g.fanCorner.y + float(y) * g.fanDelta.y;
                        const float fanZ = g.fanCorner.z + float(stepNo) * g.fanDelta.z;
                        const float proj = (sad - fanZ) * sqrtf(1.0f + (fanX * fanX) / (g.sourceDist.x * g.sourceDist.x) +
                                                                (fanY * fanY) / (g.sourceDist.y * g.sourceDist.y));
                        const float phy = proj - (sad - g.beamParaPos);
                        const float initR2 = p.bp0 + 2.0f * p.bp1 * phy + p.bp2 * phy * phy;
                        const float axisSq = 0.5f * fmaxf(0.0f, initR2 + sumS2 / sumW);
                        const float axis = sqrtf(fmaxf(0.0f, axisSq));
                        rSigmaEff = 0.5f * stepGeo[stepNo].x / (kSqrt2 * (axis + 0.21f));
                    }
                }
            }
            if ((g.profileMode & 2) && res > 0.0f) {
                const float ow = profile_sample(g.profile, g.profileDepthN, g.profileChannels, g.profileRows,
                                                g.profileChannels - 1, dIdx, rIdx);
                res *= fmaxf(0.0f, ow);
            }
        }
        runMax = fmaxf(runMax, res);
        *dst = make_float2(res, rSigmaEff);
        dst += padPlane;
        const int zr = stepNo - first;
        if (nucIdx >= 0) nucL[static_cast<size_t>(zr) * nucPlane + nucIdx] = make_float2(nucRes, nucRSigmaEff);

        // Warp minimum over all rays and range over the depositing ones, on the bits of the
        // floats, which order like them as long as they are positive (rSigmaEff is; the
        // device's canonical NaN lies above +inf and drops out of the minimum, as it does
        // under fminf). The smallest depositing value is the minimum unless a ray without
        // dose has a finite value too.
        const bool deposits = res > 0.0f;
        const int bits = __float_as_int(rSigmaEff);
        const int mk = __reduce_min_sync(0xffffffffu, bits);
        const int hi = __reduce_max_sync(0xffffffffu, deposits ? bits : 0);
        int lo = mk;
        if (__any_sync(0xffffffffu, !deposits && bits < 0x7f800000))
            lo = __reduce_min_sync(0xffffffffu, deposits ? bits : 0x7fffffff);
        if (lane == 0) {
            partMin[zr * 8 + warp] = __int_as_float(mk);
            partRange[zr * 8 + warp] = hi > 0 ? range_word(lo, hi) : 0u;
        }
    }
    // The row's remaining steps: no dose, rSigmaEff = +inf, nothing live (the halo's planes
    // start out like that). Past the tile's
    // last walked step no tile is live and nothing reads its sources.
    if (lane == 0) atomicMax(&shEnd, stepNo);
    __syncthreads();
    const int fillEnd = g.fillDeadTiles ? afterLastL : shEnd;
    for (int k = stepNo; k < fillEnd; ++k)
        srcL[static_cast<size_t>(k - first) * padPlane] = make_float2(0.0f, __int_as_float(0x7f800000));
    for (int zr = stepNo - first + lane; zr < afterLastL - first; zr += 32) {
        partMin[zr * 8 + warp] = __int_as_float(0x7f800000);
        partRange[zr * 8 + warp] = 0;
    }

    {
        const unsigned mb = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(runMax, 0.0f)));
        if (lane == 0 && mb) atomicMax(&ls[l].maxIddBits, mb);
    }
    int fp = real ? static_cast<int>(afterLast) : INT_MIN;
    if (real && firstPassiveOut) firstPassiveOut[static_cast<size_t>(lc) * rayPlane + ridx] = fp;
    for (int off = 16; off > 0; off >>= 1) fp = max(fp, __shfl_xor_sync(0xffffffffu, fp, off));
    if (lane == 0) shPassive[warp] = fp;
    __syncthreads();

    // Tile codes of every step and the tile's histogram contribution.
    const int nSteps = max(afterLastL - first, 0);
    uint8_t* codeL = codes + static_cast<size_t>(lc) * g.steps * g.tilesX * g.tilesY;
    const int tiles = g.tilesX * g.tilesY;
    for (int zr = tid; zr < nSteps; zr += 256) {
        float tm = partMin[zr * 8];
        unsigned tl = partRange[zr * 8];
#pragma unroll
        for (int w = 1; w < 8; ++w) {
            tm = fminf(tm, partMin[zr * 8 + w]);
            tl = merge_range(tl, partRange[zr * 8 + w]);
        }
        const int R = tile_radius_bucket(tm);
        const size_t ti = static_cast<size_t>(zr) * tiles + ty * g.tilesX + tx;
        codeL[ti] = static_cast<uint8_t>(R | (tl ? 0x80 : 0));
        if (tl) tileRange[static_cast<size_t>(lc) * g.steps * tiles + ti] = tl;
        atomicAdd(&shHist[R], 1);
        if (tl) atomicAdd(&shLive[R], 1);
    }
    __syncthreads();
    if (tid < kBuckets) {
        if (shHist[tid]) atomicAdd(&ls[l].histAll[tid], shHist[tid]);
        if (shLive[tid]) atomicAdd(&ls[l].liveHist[tid], shLive[tid]);
    }
    if (tid == 0) {
        int v = shPassive[0];
        for (int w = 1; w < 8; ++w) v = max(v, shPassive[w]);
        if (v != INT_MIN) atomicMax(&ls[l].maxFirstPassive, v);
    }
}

// Per layer of the chunk: passive step (wrapper.cu:4975-4990), histogram over [first,
// calcPassive) (tiles at steps >= calcPassive hold only dead rays and fall in bucket 0),
// overflow merge into R=32 (complete_superposition.cu:412-460) and batching of sparse
// buckets into the radius above them (complete_superposition.cu:476-483). Then the chunk's
// work list is laid out in descending radius.
//
// With `primaryLs` set the kernel plans the nuclear halo of the chunk instead
// (performNuclearTileBasedSuperposition, complete_superposition.cu:558-708): the
// halo histogram already covers [first, calcPassive) of the primary layer, and a
// radius above 32 is an error (the reference throws) rather than a merge.
//
// One block, latency bound. A warp reads and writes a layer's tables, lane = bucket, and a
// thread per layer batches them in shared memory; with a thread per layer throughout, each
// access to the tables was one sector per thread: 11.6 us in place of 9.6 (40 layers).
constexpr int kPlanThreads = 1024;

__global__ void __launch_bounds__(kPlanThreads)
layer_plan_kernel(BeamGeomDev g, int layer0, int nLayers, LayerStateDev* __restrict__ ls,
                  BeamStateDev* __restrict__ beam, int workCapacity, const LayerStateDev* __restrict__ primaryLs,
                  const BeamStateDev* __restrict__ primaryBeam) {
    constexpr int kStride = kBuckets + 1 - kBuckets % 2;  // odd
    __shared__ int sHist[kMaxChunkLayers][kStride];  // tiles per bucket; the list's offsets in the end
    __shared__ int sMap[kMaxChunkLayers][kStride];   // live tiles per bucket, then its batched radius
    __shared__ int sBatched[kMaxChunkLayers][kMaxR + 1];
    __shared__ int sLive[kMaxChunkLayers][kMaxR + 1];  // live items per batched radius
    __shared__ int sWarpSum[kPlanThreads / 32];
    __shared__ unsigned long long sFma;
    __shared__ unsigned sMaxIdd;
    __shared__ int sMaxCalc;
    pdl_trigger();
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const bool nuclear = primaryLs != nullptr;
    const int first = nuclear ? primaryBeam->firstInside : beam->firstInside;
    const int tiles = g.tilesX * g.tilesY;
    int calc = 0, afterLast = 0;
    unsigned maxIdd = 0;
    if (t < nLayers) {
        const LayerStateDev& st = ls[layer0 + t];
        afterLast = st.afterLast;
        calc = nuclear ? primaryLs[layer0 + t].calcPassive : st.maxFirstPassive;
        maxIdd = st.maxIddBits;
    }
    if (t == 0) {
        sFma = 0;
        sMaxIdd = 0;
        sMaxCalc = INT_MIN;
    }
    for (int q = warp; q < nLayers; q += kPlanThreads / 32)
        for (int i = lane; i < kBuckets; i += 32) {
            sHist[q][i] = ls[layer0 + q].histAll[i];
            sMap[q][i] = ls[layer0 + q].liveHist[i];
            if (i <= kMaxR) {
                sBatched[q][i] = 0;
                sLive[q][i] = 0;
            }
        }
    __syncthreads();
    if (t < nLayers) {
        LayerStateDev& st = ls[layer0 + t];
        int* hist = sHist[t];
        int* map = sMap[t];
        if (nuclear) {
            st.afterLast = calc;
            if (hist[kMaxR + 1] > 0) atomicOr(&beam->errorFlags, 4);
        } else {
            if (calc < first + 1) calc = first + 1;
            if (calc < 0) calc = first + 1;
            if (calc > afterLast) calc = afterLast;
            if (calc > g.steps) calc = g.steps;
            if (afterLast > calc && afterLast > first) hist[0] -= (afterLast - max(calc, first)) * tiles;
        }
        st.calcPassive = calc;
        atomicMax(&sMaxCalc, calc);
        if (maxIdd) atomicMax(&sMaxIdd, maxIdd);
        // Batches from the widest radius down: a batch, named by its widest radius `top`,
        // takes radii until it holds kMinTilesInBatch tiles. The overflow bucket counts as
        // the widest radius.
        int live = 0, top = 0, held = 0, heldLive = 0;
        bool met = false;
#pragma unroll 4
        for (int rad = kMaxR; rad > 0; --rad) {
            const int h = hist[rad] + (rad == kMaxR ? hist[kMaxR + 1] : 0);
            const int l = map[rad] + (rad == kMaxR ? map[kMaxR + 1] : 0);
            live += l;
            if (!met && h > 0) {
                met = true;
                top = rad;
            }
            map[rad] = met ? top : rad;
            if (rad == kMaxR) map[kMaxR + 1] = map[rad];
            held += h;
            heldLive += l;
            if (met) {
                sBatched[t][top] = held;
                sLive[t][top] = heldLive;
                if (held >= kMinTilesInBatch) {
                    top = rad - 1;
                    held = 0;
                    heldLive = 0;
                }
            }
        }
        live += map[0];
        sBatched[t][0] = hist[0];
        sLive[t][0] = map[0];
        map[0] = 0;
        st.liveTiles = live;
    }
    __syncthreads();
    for (int q = warp; q < nLayers; q += kPlanThreads / 32) {
        LayerStateDev& st = ls[layer0 + q];
        for (int i = lane; i < kBuckets; i += 32) {
            st.hist[i] = sHist[q][i];
            st.batchedR[i] = sMap[q][i];
            if (i <= kMaxR) {
                st.batchedCounts[i] = sBatched[q][i];
                st.liveR[i] = sLive[q][i];
                st.curR[i] = 0;
            }
        }
    }

    // Work-list offsets: radius groups in descending radius, each with its layers in
    // order, i.e. position p = (kMaxR - r) * nLayers + q. Each thread sums a run of
    // positions, the block scans the runs, then each thread sets its offsets.
    const int total = (kMaxR + 1) * nLayers;
    const int per = (total + kPlanThreads - 1) / kPlanThreads;
    const int p0 = min(t * per, total), p1 = min(p0 + per, total);
    int runSum = 0;
    long long runFma = 0;
    for (int p = p0; p < p1; ++p) {
        const int r = kMaxR - p / nLayers, q = p % nLayers;
        const int v = sLive[q][r];
        runSum += v;
        runFma += static_cast<long long>(v) * 256 * (2 * r + 1) * (2 * r + 1);
    }
    int incl = runSum;
    for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
    }
    for (int o = 16; o > 0; o >>= 1) runFma += __shfl_xor_sync(0xffffffffu, runFma, o);
    if (lane == 31) sWarpSum[warp] = incl;
    if (lane == 0 && runFma) atomicAdd(&sFma, static_cast<unsigned long long>(runFma));
    __syncthreads();
    // Items before this warp's positions, and in all.
    const int sum = sWarpSum[lane];
    int acc = __reduce_add_sync(0xffffffffu, lane < warp ? sum : 0) + incl - runSum;
    int items = __reduce_add_sync(0xffffffffu, sum);
    for (int p = p0; p < p1; ++p) {
        const int r = kMaxR - p / nLayers, q = p % nLayers;
        sHist[q][r] = acc;
        if (q == 0) beam->rStart[r] = acc;
        acc += sLive[q][r];
    }
    if (t <= kMaxR) beam->mergedR[t] = 0;
    if (t == 0) {
        if (nuclear) {
            // The halo transfer spans the same steps as the primary one.
            beam->firstInside = first;
            beam->maxCalcPassive = primaryBeam->maxCalcPassive;
        }
        beam->maxCalcPassive = max(beam->maxCalcPassive, sMaxCalc);
        if (items > workCapacity) {
            atomicOr(&beam->errorFlags, 1);
            items = workCapacity;
        }
        beam->workCount = items;
        beam->workNext = 0;
        beam->workNextSmall = 0;
        beam->workNextTiny = 0;
        // Fixed-point range of the chunk's BEV: a cell sums at most `items` tile
        // footprints (merged items sum several of them), each at most 256 x the
        // largest IDD of the chunk, so with that IDD below 2^ex every cell stays below
        // 2^(ex + 8 + ceil(log2 items)); the shift puts that bound at 2^61.
        int ex = 0;
        frexpf(__uint_as_float(sMaxIdd), &ex);
        int lg = 0;
        while ((1LL << lg) < static_cast<long long>(max(items, 1))) ++lg;
        beam->fixedShift = sMaxIdd ? min(61 - ex - 8 - lg, 120) : 0;
        beam->liveTiles += items;
        beam->superposeFma += static_cast<long long>(sFma);
    }
    __syncthreads();
    for (int q = warp; q < nLayers; q += kPlanThreads / 32)
        for (int i = lane; i <= kMaxR; i += 32) ls[layer0 + q].offR[i] = sHist[q][i];
}

// One thread per (layer, step, tile) code of the chunk: live tiles are written to
// their layer's radius group of the work list as one-layer items in the forward
// superposition's format. Each
// layer's box of the cells its items can write (LayerStateDev::liveLo/liveHi) is
// reduced per warp (a warp's 32 consecutive codes span at most a few layers) before
// its atomics.
__global__ void work_scatter_kernel(BeamGeomDev g, int layer0, int nLayers, const uint8_t* __restrict__ codes,
                                    LayerStateDev* __restrict__ ls, const BeamStateDev* __restrict__ beam,
                                    int4* __restrict__ work, int workCapacity) {
    const int tiles = g.tilesX * g.tilesY;
    const int first = beam->firstInside;
    const size_t perLayer = static_cast<size_t>(g.steps) * tiles;
    const size_t total = perLayer * nLayers;
    const int lane = threadIdx.x & 31;
    // Warp-uniform trip count: every lane takes part in the reductions.
    for (size_t i0 = blockIdx.x * size_t(blockDim.x) + threadIdx.x - lane; i0 < total;
         i0 += size_t(gridDim.x) * blockDim.x) {
        const size_t i = i0 + lane;
        int key = -1, R = 0, tile = 0, zr = 0;
        if (i < total) {
            const int lc = int(i / perLayer);
            const int rem = int(i - size_t(lc) * perLayer);
            zr = rem / tiles;
            tile = rem - zr * tiles;
            LayerStateDev& st = ls[layer0 + lc];
            const int c = codes[i];
            if (zr < st.afterLast - first && (c & 0x80)) {
                R = st.batchedR[c & 0x3f];
                const int slot = st.offR[R] + atomicAdd(&st.curR[R], 1);
                if (slot < workCapacity)
                    work[slot] = make_int4(static_cast<int>(1u << (lc & 31)), tile, zr, R | ((lc & ~31) << 8));
                key = lc;
            }
        }
        if (!__any_sync(0xffffffffu, key >= 0)) continue;
        const unsigned same = __match_any_sync(0xffffffffu, key);
        const int tx = tile % g.tilesX, ty = tile / g.tilesX;
        const int lo0 = key >= 0 ? tx * kTileX - R + kMaxR : INT_MAX;
        const int lo1 = key >= 0 ? ty * kTileY - R + kMaxR : INT_MAX;
        const int lo2 = key >= 0 ? zr : INT_MAX;
        const int hi0 = key >= 0 ? tx * kTileX + kTileX - 1 + R + kMaxR : INT_MIN;
        const int hi1 = key >= 0 ? ty * kTileY + kTileY - 1 + R + kMaxR : INT_MIN;
        const int hi2 = key >= 0 ? zr : INT_MIN;
        const int mlo0 = __reduce_min_sync(same, lo0), mlo1 = __reduce_min_sync(same, lo1);
        const int mlo2 = __reduce_min_sync(same, lo2);
        const int mhi0 = __reduce_max_sync(same, hi0), mhi1 = __reduce_max_sync(same, hi1);
        const int mhi2 = __reduce_max_sync(same, hi2);
        if (key >= 0 && lane == __ffs(same) - 1) {
            LayerStateDev& st = ls[layer0 + key];
            atomicMin(&st.liveLo[0], mlo0);
            atomicMin(&st.liveLo[1], mlo1);
            atomicMin(&st.liveLo[2], mlo2);
            atomicMax(&st.liveHi[0], mhi0);
            atomicMax(&st.liveHi[1], mhi1);
            atomicMax(&st.liveHi[2], mhi2);
        }
    }
}

// Appends a merged item to the block of its radius, [blockStart[R], blockStart[R - 1])
// (R = 0: up to blockStart[kMaxR + 1], the item count). Merging only joins items of one
// radius, so the merged items of R fit in the block its unmerged items occupy.
__device__ __forceinline__ void emit_merged(BeamStateDev* beam, const int* blockStart, int4* work, unsigned layers,
                                            int base, int tile, int zr, int R) {
    const int begin = blockStart[R];
    const int end = R > 0 ? blockStart[R - 1] : blockStart[kMaxR + 1];
    const int slot = begin + atomicAdd(&beam->mergedR[R], 1);
    if (slot < end) work[slot] = make_int4(static_cast<int>(layers), tile, zr, R | (base << 8));
}

// The forward superposition's work list: one warp per (step, tile) of the chunk,
// a lane per chunk layer (two passes for chunks of more than 32 layers), takes the
// tile's live items at that step (the same items, radii and step ranges as
// work_scatter_kernel) and makes one item of all layers with equal batched radius: the
// superposition's convolutions are done once per item whatever its layers. Each item
// goes to the block of its radius (so the superposition's warps run one radius at a
// time); the order within a block is arbitrary, and the superposition's fixed-point BEV
// makes the dose independent of it.
__global__ void work_merge_kernel(BeamGeomDev g, int layer0, int nLayers, const uint8_t* __restrict__ codes,
                                  const LayerStateDev* __restrict__ ls, BeamStateDev* __restrict__ beam,
                                  int4* __restrict__ work) {
    // The block's extent of the cells its items write (min x, y, z; max x, y, z), and
    // the radius blocks of the list (read once: the claims below are atomics on the
    // same beam state, which later reads of it would wait behind).
    __shared__ int sExt[6];
    __shared__ int sStart[kMaxR + 2];
    pdl_wait();
    if (threadIdx.x < 6) sExt[threadIdx.x] = threadIdx.x < 3 ? INT_MAX : INT_MIN;
    if (threadIdx.x <= kMaxR) sStart[threadIdx.x] = beam->rStart[threadIdx.x];
    if (threadIdx.x == kMaxR + 1) sStart[kMaxR + 1] = beam->workCount;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int tiles = g.tilesX * g.tilesY;
    const int first = beam->firstInside;
    const size_t perLayer = static_cast<size_t>(g.steps) * tiles;
    const size_t warps = (size_t(gridDim.x) * blockDim.x) >> 5;
    for (size_t i = (blockIdx.x * size_t(blockDim.x) + threadIdx.x) >> 5; i < perLayer; i += warps) {
        const int zr = int(i / tiles);
        const int tile = int(i - size_t(zr) * tiles);
        int rMax = -1;
        for (int base = 0; base < nLayers; base += 32) {
            const int lc = base + lane;
            int R = -1;
            if (lc < nLayers) {
                const LayerStateDev& st = ls[layer0 + lc];
                const int c = codes[size_t(lc) * perLayer + i];
                if (zr < st.afterLast - first && (c & 0x80)) R = st.batchedR[c & 0x3f];
            }
            rMax = max(rMax, R);
            // The lanes of one radius are one item; its first lane writes it.
            const unsigned same = __match_any_sync(0xffffffffu, R);
            if (R >= 0 && lane == __ffs(same) - 1) emit_merged(beam, sStart, work, same, base, tile, zr, R);
        }
        rMax = __reduce_max_sync(0xffffffffu, rMax);
        if (lane == 0 && rMax >= 0) {
            const int tx = tile % g.tilesX, ty = tile / g.tilesX;
            atomicMin(&sExt[0], tx * kTileX - rMax + kMaxR);
            atomicMin(&sExt[1], ty * kTileY - rMax + kMaxR);
            atomicMin(&sExt[2], zr);
            atomicMax(&sExt[3], tx * kTileX + kTileX - 1 + rMax + kMaxR);
            atomicMax(&sExt[4], ty * kTileY + kTileY - 1 + rMax + kMaxR);
            atomicMax(&sExt[5], zr);
        }
    }
    __syncthreads();
    if (threadIdx.x < 3 && sExt[threadIdx.x] != INT_MAX) atomicMin(&beam->liveLo[threadIdx.x], sExt[threadIdx.x]);
    if (threadIdx.x >= 3 && threadIdx.x < 6 && sExt[threadIdx.x] != INT_MIN)
        atomicMax(&beam->liveHi[threadIdx.x - 3], sExt[threadIdx.x]);
}

// Halo cells start empty: IDD 0 and rSigmaEff +inf (wrapper.cu:4124-4135).
__global__ void nuc_fill_kernel(float2* __restrict__ sources, size_t n) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        sources[i] = make_float2(0.0f, __int_as_float(0x7f800000));
}

// One warp per (layer, step, halo tile) over [first, calcPassive) of the layer:
// the tile's radius bucket and liveness (tileRadCalc, complete_superposition.cu:
// 198-255, on the halo grid), its code, and its count in the halo histogram.
__global__ void nuc_codes_kernel(BeamGeomDev gn, int layer0, int nLayers, const float2* __restrict__ sources,
                                 const LayerStateDev* __restrict__ primaryLs,
                                 const BeamStateDev* __restrict__ primaryBeam, LayerStateDev* __restrict__ nucLs,
                                 unsigned* __restrict__ tileRange, uint8_t* __restrict__ codes) {
    const int lane = threadIdx.x & 31;
    const int tiles = gn.tilesX * gn.tilesY;
    const int first = primaryBeam->firstInside;
    const size_t plane = static_cast<size_t>(gn.pitchX) * gn.pitchY;
    const size_t perLayer = static_cast<size_t>(gn.steps) * tiles;
    const size_t total = perLayer * nLayers;
    const size_t warps = (size_t(gridDim.x) * blockDim.x) >> 5;
    for (size_t i = (blockIdx.x * size_t(blockDim.x) + threadIdx.x) >> 5; i < total; i += warps) {
        const int lc = int(i / perLayer);
        const int rem = int(i - size_t(lc) * perLayer);
        const int zr = rem / tiles, tile = rem - zr * tiles;
        if (zr >= primaryLs[layer0 + lc].calcPassive - first) continue;
        const float2* ti = sources + (lc * static_cast<size_t>(gn.steps) + zr) * plane + size_t(tile) * kTileSources + lane;
        unsigned key = 0xffffffffu, range = 0;
        bool live = false;
        float mx = 0.0f;
#pragma unroll
        for (int r = 0; r < kTileY; ++r) {
            const float2 v = ti[r * kTileX];
            key = min(key, float_order_key(v.y));
            if (v.x > 0.0f && v.y > 0.0f) range = merge_range(range, range_word(__float_as_int(v.y), __float_as_int(v.y)));
            live |= v.x > 0.0f;
            mx = fmaxf(mx, v.x);
        }
        key = __reduce_min_sync(0xffffffffu, key);
        const unsigned hi = __reduce_max_sync(0xffffffffu, range >> 16);
        const unsigned lo = __reduce_min_sync(0xffffffffu, range ? range & 0xffffu : 0xffffu);
        live = __any_sync(0xffffffffu, live);
        const unsigned mb = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
        if (lane == 0 && mb) atomicMax(&nucLs[layer0 + lc].maxIddBits, mb);
        if (lane == 0) {
            const int R = tile_radius_bucket(float_from_order_key(key));
            codes[i] = static_cast<uint8_t>(R | (live ? 0x80 : 0));
            if (live) tileRange[i] = hi ? hi << 16 | lo : 0u;
            atomicAdd(&nucLs[layer0 + lc].histAll[R], 1);
            if (live) atomicAdd(&nucLs[layer0 + lc].liveHist[R], 1);
        }
    }
}

}  // namespace

// Table rows, per-step widths and volumes, and the warps' partials of every step.
size_t idd_smem_bytes(const BeamGeomDev& g, const LutsDev& luts) {
    const size_t tableFloats = static_cast<size_t>(luts.nS) * (g.nucOn ? 3 : 1) + 2;
    return (tableFloats + 2 * static_cast<size_t>(g.steps)) * sizeof(float) +
           static_cast<size_t>(g.steps) * 8 * (sizeof(float) + sizeof(unsigned));
}

cudaError_t launch_nuc_prepare(const BeamGeomDev& gn, int nLayers, float2* sources, cudaStream_t s) {
    const size_t n = static_cast<size_t>(nLayers) * gn.steps * gn.pitchX * gn.pitchY;
    const int blocks = int(std::min<size_t>((n + 255) / 256, 148 * 16));
    nuc_fill_kernel<<<blocks, 256, 0, s>>>(sources, n);
    return cudaGetLastError();
}

cudaError_t launch_nuc_codes(const BeamGeomDev& gn, int layer0, int nLayers, const float2* sources,
                             const LayerStateDev* primaryLs, const BeamStateDev* primaryBeam, LayerStateDev* nucLs,
                             unsigned* tileRange, uint8_t* codes, cudaStream_t s) {
    const size_t warps = static_cast<size_t>(nLayers) * gn.steps * gn.tilesX * gn.tilesY;
    const int blocks = int(std::min<size_t>((warps + 7) / 8, 148 * 16));
    nuc_codes_kernel<<<blocks, 256, 0, s>>>(gn, layer0, nLayers, sources, primaryLs, primaryBeam, nucLs, tileRange, codes);
    return cudaGetLastError();
}

cudaError_t launch_idd(const BeamGeomDev& g, const LutsDev& luts, int layer0, int nLayers, const float2* material,
                       const float* wepl, const int* firstInside, const int* firstOutside, const float* rayW,
                       const LayerParamsDev* lp, LayerStateDev* ls, const BeamStateDev* beam, float2* sources,
                       unsigned* tileRange, uint8_t* codes, int* firstPassive, const int* rayToNuc, const float* lattice,
                       float2* nucSources, cudaStream_t s) {
    dim3 grid(g.tilesX, g.tilesY, nLayers);
    dim3 block(32, 8);
    const size_t smem = idd_smem_bytes(g, luts);
    auto k = g.nucOn ? (g.profileMode ? idd_kernel<true, true> : idd_kernel<true, false>)
                     : (g.profileMode ? idd_kernel<false, true> : idd_kernel<false, false>);
    cudaError_t e = set_smem_limit(reinterpret_cast<const void*>(k), smem);
    if (e != cudaSuccess) return e;
    k<<<grid, block, smem, s>>>(g, luts, layer0, material, wepl, firstInside, firstOutside, rayW, lp, ls, beam, sources,
                                tileRange, codes, firstPassive, rayToNuc, lattice, nucSources);
    return cudaGetLastError();
}

cudaError_t launch_bin_plan(const BeamGeomDev& g, int layer0, int nLayers, const uint8_t* codes, LayerStateDev* ls,
                            BeamStateDev* beam, int4* work, int workCapacity, bool merged,
                            const LayerStateDev* primaryLs, const BeamStateDev* primaryBeam, cudaStream_t s) {
    if (nLayers > kMaxChunkLayers) return cudaErrorInvalidValue;
    layer_plan_kernel<<<1, kPlanThreads, 0, s>>>(g, layer0, nLayers, ls, beam, workCapacity, primaryLs,
                                                    primaryBeam);
    if (merged) {
        const size_t warps = static_cast<size_t>(g.steps) * g.tilesX * g.tilesY;
        const int blocks = int(std::min<size_t>((warps + 7) / 8, 148 * 16));
        cudaError_t e = launch_pdl(work_merge_kernel, dim3(blocks), dim3(256), 0, s, g, layer0, nLayers, codes,
                                   static_cast<const LayerStateDev*>(ls), beam, work);
        if (e != cudaSuccess) return e;
    } else {
        const size_t total = static_cast<size_t>(g.steps) * g.tilesX * g.tilesY * nLayers;
        const int blocks = int(std::min<size_t>((total + 255) / 256, 148 * 8));
        work_scatter_kernel<<<blocks, 256, 0, s>>>(g, layer0, nLayers, codes, ls, beam, work, workCapacity);
    }
    return cudaGetLastError();
}

}  // namespace pbs
