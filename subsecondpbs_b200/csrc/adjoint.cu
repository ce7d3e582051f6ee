// Adjoint of the dose with respect to the beam's ray weights: the transposes of
// the BEV -> dose transfer and of the tile superposition, followed by the IDD
// scaling. Dose is linear in the spot weights: for a live ray
//   idd[l][k][ray] = rayW[l][ray] * g[l][k][ray]      (idd_sigma.cu:194-201),
//   BEV = S(idd)  (tile superposition, complete_superposition.cu:264-335),
//   D  += T(BEV)  (divergent trilinear transfer, prim_transf_kernel.cu:11-44),
// so for a dose gradient Gd the ray-weight gradient is
//   rbar[l][ray] = sum_k g[l][k][ray] * (S^T T^T Gd)[l][k][ray]
//               = (sum_k idd[l][k][ray] * (S^T T^T Gd)[l][k][ray]) / rayW[l][ray].
// The tile radii, the live-ray mask and rSigmaEff do not depend on the weights'
// values, so they come from the same IDD and binning kernels as the forward pass.
#include <algorithm>

#include "device_util.cuh"
#include "work_blocks.cuh"
#include "kernels.h"
#include "launch_util.h"
#include "node_spread.cuh"
#include "transfer_walk.cuh"

namespace pbs {

namespace {

// T^T: every dose voxel of the transfer box spreads its gradient over the eight
// BEV texels its forward sample interpolated (bev_sample in transfer.cu), with the
// same weights. The forward adds a sample only where it is positive, and BEV cells are
// not negative: a sum of interpolated footprints that ends below zero is taken as zero.
// The transpose ignores that, so the two match to within the interpolation's residue,
// 2.5e-7 of the peaks of the sources that reach the cell (node_spread.cuh).
// A lane takes one dose column and 8 consecutive z (walk_box; the box is known only on
// the device).
__global__ void __launch_bounds__(256)
transfer_adjoint_kernel(BeamGeomDev g, const double* __restrict__ gradDose, const BeamStateDev* __restrict__ beam,
                        float* __restrict__ gradBev) {
    if (!beam->transferValid) return;
    const int sx = beam->transferStart[0], sy = beam->transferStart[1], sz = beam->transferStart[2];
    const int mx = beam->transferMax[0], my = beam->transferMax[1], mz = beam->transferMax[2];
    const int nxCols = min(((mx - sx + 1 + 31) / 32) * 32, g.doseX - sx);
    const int nyCols = min(((my - sy + 1 + 7) / 8) * 8, g.doseY - sy);
    const int nzc = (mz - sz + 8) / 8;
    if (nxCols <= 0 || nyCols <= 0 || nzc <= 0) return;
    const TransferParams T = beam->transfer;
    const float zShift = g.compatBevZShift ? float(beam->firstInside) : 0.0f;
    const size_t slice = static_cast<size_t>(g.doseX) * g.doseY;
    const int nx = g.bevX, ny = g.bevY, nz = g.steps;
    walk_box(T, sx, sy, nxCols, nyCols, nzc, [&](int x, int y, int chunk) {
        const int z0 = sz + chunk * 8;
        const int z1 = min(mz, z0 + 7);
        const V3 start = transfer_start(T, x, y);
        for (int z = z0; z <= z1; ++z) {
            const V3 f = transfer_fan_idx(T, start, z);
            if (f.x + 0.5f < 0.0f || f.y + 0.5f < 0.0f || f.z + 0.5f < 0.0f) continue;
            const float gd = float(gradDose[static_cast<size_t>(z) * slice + static_cast<size_t>(y) * g.doseX + x]);
            if (gd == 0.0f) continue;
            const float px = fminf(fmaxf(f.x, -2.0f), float(nx) + 1.0f);
            const float py = fminf(fmaxf(f.y, -2.0f), float(ny) + 1.0f);
            const float pz = fminf(fmaxf(f.z - zShift, -2.0f), float(nz) + 1.0f);
            const float fx = floorf(px), fy = floorf(py), fz = floorf(pz);
            const int x0 = int(fx), y0 = int(fy), z0i = int(fz);
            const float tx = px - fx, ty = py - fy, tz = pz - fz;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const int xi = x0 + (c & 1), yi = y0 + ((c >> 1) & 1), zi = z0i + (c >> 2);
                if (xi < 0 || yi < 0 || zi < 0 || xi >= nx || yi >= ny || zi >= nz) continue;
                const float w =
                    ((c & 1) ? tx : 1.0f - tx) * (((c >> 1) & 1) ? ty : 1.0f - ty) * ((c >> 2) ? tz : 1.0f - tz);
                atomicAdd(gradBev + (static_cast<size_t>(zi) * ny + yi) * nx + xi, w * gd);
            }
        }
    });
}

// S^T. A source's gradient is the BEV gradient gathered over its footprint with the
// forward's weights, and those are interpolated between nodes of rSigma as there
// (node_spread.cuh):
//   sum_{dy,dx} e_r(dy) e_r(dx) G = sum_j L_j(r) Q_j,  Q_j = E_j(y) * G * E_j(x).
// One warp takes one item of the forward's merged work list, a tile at one step with all
// its layers of one radius. The separable convolutions Q_j do not depend on the layer and
// are done once per item, two nodes (+-x_p) at a time:
//   * columns: lane = one footprint column, its rows in registers; both nodes' eight
//     output rows, as the pairs (y, 7 - y), go to shared memory;
//   * rows: lane = one (node, row pair, eight columns); the results replace the rows;
//   * lane = source column: A_p = C_p x_p (Q+ + Q-), D_p = C_p (Q+ - Q-);
// then every layer's sources add idd sum_p B_p(t^2) (A_p + t D_p) to their rays. Bound by
// FMA issue in the convolutions. Gathering (2R+1)^2 cells for every source and layer, as
// pair sums, took 342 us in place of 99 us (36 layers on 64 x 64 x 128 voxels of 2 mm).
template <int R>
__device__ __forceinline__ void gather_columns(const float* __restrict__ src, int bevX, const float2* __restrict__ e,
                                               float2* __restrict__ rows, int lane) {
    constexpr int W = kTileX + 2 * R, H = kTileY + 2 * R, N = H / 2;
#pragma unroll 1
    for (int x = lane; x < W; x += 32) {
        float2 t[N];
#pragma unroll
        for (int i = 0; i < N; ++i) t[i] = make_float2(__ldg(src + i * bevX + x), __ldg(src + (H - 1 - i) * bevX + x));
#pragma unroll 1
        for (int j = 0; j < 2; ++j) {
            float2 acc[kPairs];
#pragma unroll
            for (int y = 0; y < kPairs; ++y) acc[y] = make_float2(0.0f, 0.0f);
            const float4* e4 = reinterpret_cast<const float4*>(e + j * kTableStride<R>);
#pragma unroll
            for (int q = 0; q < (R + 2) / 2; ++q) {
                const float4 w = e4[q];
                const float2 wk[2] = {make_float2(w.x, w.y), make_float2(w.z, w.w)};
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int k = 2 * q + c;
                    if (k <= R) {
#pragma unroll
                        for (int y = 0; y < kPairs; ++y) {
                            const int i0 = y + R - k, i1 = y + R + k;
                            const float2 lo = i0 < N ? t[i0 < N ? i0 : 0] : make_float2(t[H - 1 - i0].y, t[H - 1 - i0].x);
                            const float2 hi = i1 < N ? t[i1 < N ? i1 : 0] : make_float2(t[H - 1 - i1].y, t[H - 1 - i1].x);
                            acc[y] = __ffma2_rn(lo, wk[c], acc[y]);
                            if (k > 0) acc[y] = __ffma2_rn(hi, wk[c], acc[y]);
                        }
                    }
                }
            }
#pragma unroll
            for (int y = 0; y < kPairs; ++y) rows[(j * kPairs + y) * kRowStride<R> + x] = acc[y];
        }
    }
}

// The eight rows of two nodes, each convolved along x over its 32 sources: the result of
// source column sx lies at sx. Lanes of one half-warp read distinct banks (odd stride).
template <int R>
__device__ __forceinline__ void gather_rows(float2* __restrict__ rows, const float2* __restrict__ e, int lane) {
    constexpr int kOut = kTileX / 4;
    const int row = lane & 7;
    float2 k[kTableStride<R>];
    const float4* e4 = reinterpret_cast<const float4*>(e + (row / kPairs) * kTableStride<R>);
#pragma unroll
    for (int q = 0; q < (R + 2) / 2; ++q) {
        const float4 v = e4[q];
        k[2 * q] = make_float2(v.x, v.y);
        k[2 * q + 1] = make_float2(v.z, v.w);
    }
    float2* p = rows + row * kRowStride<R> + (lane >> 3) * kOut;
    float2 acc[kOut];
#pragma unroll
    for (int o = 0; o < kOut; ++o) acc[o] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < kOut + 2 * R; ++i) {
        const float2 v = p[i];
#pragma unroll
        for (int o = 0; o < kOut; ++o) {
            const int d = i - o - R, a = d < 0 ? -d : d;
            if (a <= R) acc[o] = __ffma2_rn(v, k[a <= R ? a : 0], acc[o]);
        }
    }
    __syncwarp();
#pragma unroll
    for (int o = 0; o < kOut; ++o) p[o] = acc[o];
}

template <int R, int RHi>
__device__ __forceinline__ void gather_item(int r, const float* src, int bevX, const float2* e, float2* rows, int lane) {
    if (r == R) {
        gather_columns<R>(src, bevX, e, rows, lane);
        __syncwarp();
        gather_rows<R>(rows, e, lane);
        return;
    }
    if constexpr (R < RHi) gather_item<R + 1, RHi>(r, src, bevX, e, rows, lane);
}

// The sources of an item's layers: idd times the interpolated gradient into their rays.
struct SourceGradients {
    const TileSource& s;
    const NodeRange& n;
    unsigned layers;
    const float2* ad;  // (A_p, D_p) [p][2][4][32]
    float* rbar;       // the lane's ray of row 0 in the first layer of the item's group
    size_t rayPlane;
    int rayX, lane;

    template <int J>
    __device__ __forceinline__ void run() const {
        const float2 shift = make_float2(n.shift, n.shift), inv = make_float2(n.invHalf, n.invHalf);
        float2 a[kPairs][J / 2], d[kPairs][J / 2];
#pragma unroll
        for (int p = 0; p < J / 2; ++p)
#pragma unroll
            for (int y = 0; y < kPairs; ++y) {
                a[y][p] = ad[((p * 2) * kPairs + y) * kTileX + lane];
                d[y][p] = ad[((p * 2 + 1) * kPairs + y) * kTileX + lane];
            }
#pragma unroll 1
        for (unsigned m = layers; m; m &= m - 1u) {
            const int l = __ffs(m) - 1;
            const float2* f = s.first + l * s.layerStride + lane;
            float* out = rbar + l * rayPlane;
            float2 src[kTileY];
#pragma unroll
            for (int y = 0; y < kTileY; ++y) src[y] = f[y * kTileX];
#pragma unroll
            for (int y = 0; y < kPairs; ++y) {
                const float2 u = src[y], v = src[kTileY - 1 - y];
                float2 dose;
                dose.x = u.y > n.from && u.y <= n.to ? fmaxf(u.x, 0.0f) : 0.0f;
                dose.y = v.y > n.from && v.y <= n.to ? fmaxf(v.x, 0.0f) : 0.0f;
                const float2 t = __ffma2_rn(make_float2(fminf(u.y, n.top), fminf(v.y, n.top)), inv, shift);
                float2 b[J / 2];
                pair_products<J>(__fmul2_rn(t, t), b);
                float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
                for (int p = 0; p < J / 2; ++p) acc = __ffma2_rn(b[p], __ffma2_rn(t, d[y][p], a[y][p]), acc);
                // Rays outside the ray grid carry no dose.
                if (dose.x > 0.0f) atomicAdd(out + y * rayX, dose.x * acc.x);
                if (dose.y > 0.0f) atomicAdd(out + (kTileY - 1 - y) * rayX, dose.y * acc.y);
            }
        }
    }
};

// Shared memory of a warp (pairs): two nodes' tables, their eight rows, and A and D.
template <int RMax>
constexpr int kAdjWarpPairs = 2 * kTableStride<RMax> + 2 * kPairs * kRowStride<RMax> + kMaxNodes * kPairs * kTileX;

// Persistent warps over the items of radii RLo..RHi, claimed through the range's counter.
// The three instances of a beam overlap as the forward's do: each CTA lets the next
// instance launch at once (their items only add into the rays' accumulators) and waits
// for the previous instance before it exits.
template <int RLo, int RHi, int Warps, int MinBlocks>
__global__ void __launch_bounds__(Warps * 32, MinBlocks)
superpose_adjoint_kernel(BeamGeomDev g, const float2* __restrict__ sources, const unsigned* __restrict__ tileRange,
                         const int4* __restrict__ work, BeamStateDev* __restrict__ beam,
                         const float* __restrict__ gradBev, float* __restrict__ rbar) {
    pdl_trigger();
    extern __shared__ __align__(16) float2 adjSm[];
    __shared__ RadiusBlocks<RLo, RHi> sBlocks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int* counter = RLo > kSplitWide ? &beam->workNext : (RLo > kSplitR ? &beam->workNextSmall : &beam->workNextTiny);
    const int tiles = g.tilesX * g.tilesY;
    const size_t padPlane = static_cast<size_t>(tiles) * kTileSources;
    const size_t bevPlane = static_cast<size_t>(g.bevX) * g.bevY;
    const size_t rayPlane = static_cast<size_t>(g.rayX) * g.rayY;
    float2* e = adjSm + warp * kAdjWarpPairs<RHi>;
    float2* rows = e + 2 * kTableStride<RHi>;
    float2* ad = rows + 2 * kPairs * kRowStride<RHi>;

    load_blocks<RLo, RHi>(beam, sBlocks);
    __syncthreads();
    const int total = sBlocks.total, warps = gridDim.x * Warps;
    // The first item of every warp is fixed; the counter deals out the others.
    for (int c = blockIdx.x + warp * gridDim.x; c < total;) {
        int claim = 0;
        if (lane == 0) claim = warps + atomicAdd(counter, 1);
        const int4 it = work[block_slot<RLo, RHi>(sBlocks, c)];
        c = __shfl_sync(0xffffffffu, claim, 0);
        const unsigned layers = static_cast<unsigned>(it.x);
        const int tile = it.y, zRel = it.z, R = it.w & 0xff, base = it.w >> 8;
        if (R < RLo || R > RHi) {
            if (lane == 0) atomicOr(&beam->errorFlags, 2);
            continue;
        }
        unsigned range = 0;
        if (layers >> lane & 1u)
            range = tileRange[(static_cast<size_t>(base + lane) * g.steps + zRel) * tiles + tile];
        TileSource s;
        s.layerStride = static_cast<size_t>(g.steps) * padPlane;
        s.first = sources + base * s.layerStride + zRel * padPlane + tile * kTileSources;
        prefetch_tile(s, layers, lane);
        float lo, hi;
        if (!item_range(range, lo, hi)) continue;
        const int tx = tile % g.tilesX, ty = tile / g.tilesX;
        const float* src = gradBev + static_cast<size_t>(zRel) * bevPlane +
                           static_cast<size_t>(ty * kTileY - R + kMaxR) * g.bevX + (tx * kTileX - R + kMaxR);
        float* out = rbar + base * rayPlane + static_cast<size_t>(ty * kTileY) * g.rayX + tx * kTileX + lane;
        const int stride = kTileX + 2 * R + 1, eStride = ((R + 2) / 2 | 1) * 2;
        for (float from = 0.0f;;) {
            const NodeRange n = node_range(from, lo, hi);
#pragma unroll 1
            for (int p = 0; p < n.count / 2; ++p) {
                node_tables(n, 2 * p, 2, R, e, eStride, lane);
                __syncwarp();
                gather_item<RLo, RHi>(R, src, g.bevX, e, rows, lane);
                __syncwarp();
                const float cp = kNodeC[n.count / 2 - 2][p], cx = cp * kNodeX[n.count / 2 - 2][p];
#pragma unroll
                for (int y = 0; y < kPairs; ++y) {
                    const float2 qp = rows[y * stride + lane], qm = rows[(kPairs + y) * stride + lane];
                    ad[((p * 2) * kPairs + y) * kTileX + lane] = make_float2(cx * (qp.x + qm.x), cx * (qp.y + qm.y));
                    ad[((p * 2 + 1) * kPairs + y) * kTileX + lane] = make_float2(cp * (qp.x - qm.x), cp * (qp.y - qm.y));
                }
                __syncwarp();
            }
            with_nodes(n.count, SourceGradients{s, n, layers, ad, out, rayPlane, g.rayX, lane});
            if (n.top >= hi) break;
            from = lo = n.top;
        }
    }
    pdl_wait();
}

template <int RLo, int RHi, int Warps, int MinBlocks>
cudaError_t launch_adjoint_range(const BeamGeomDev& g, const float2* sources, const unsigned* tileRange,
                                 const int4* work, BeamStateDev* beam, const float* gradBev, float* rbar, int numSMs,
                                 bool overlap, cudaStream_t s) {
    auto k = superpose_adjoint_kernel<RLo, RHi, Warps, MinBlocks>;
    const size_t smem = size_t(Warps) * kAdjWarpPairs<RHi> * sizeof(float2);
    cudaError_t e = set_smem_limit(reinterpret_cast<const void*>(k), smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(numSMs * MinBlocks);
    cfg.blockDim = dim3(Warps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k, g, sources, tileRange, work, beam, gradBev, rbar);
}

}  // namespace

cudaError_t launch_transfer_adjoint(const BeamGeomDev& g, const double* gradDose, const BeamStateDev* beam,
                                    float* gradBev, cudaStream_t s) {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long cap = (static_cast<long long>(g.doseX) * g.doseY * ((g.doseZ + 7) / 8) + 255) / 256;
    const int blocks = static_cast<int>(std::max<long long>(1, std::min<long long>(cap, sms * 8)));
    transfer_adjoint_kernel<<<blocks, 256, 0, s>>>(g, gradDose, beam, gradBev);
    return cudaGetLastError();
}

cudaError_t launch_superpose_adjoint(const BeamGeomDev& g, const float2* sources, const unsigned* tileRange,
                                     const int4* work, BeamStateDev* beam, const float* gradBev, float* rbar,
                                     int numSMs, cudaStream_t s) {
    cudaError_t e = launch_adjoint_range<kSplitWide + 1, kMaxR, 4, 2>(g, sources, tileRange, work, beam, gradBev, rbar,
                                                                      numSMs, false, s);
    if (e != cudaSuccess) return e;
    e = launch_adjoint_range<kSplitR + 1, kSplitWide, 4, 3>(g, sources, tileRange, work, beam, gradBev, rbar, numSMs,
                                                            true, s);
    if (e != cudaSuccess) return e;
    return launch_adjoint_range<0, kSplitR, 4, 4>(g, sources, tileRange, work, beam, gradBev, rbar, numSMs, true, s);
}

}  // namespace pbs
