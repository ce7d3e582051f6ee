// BEV -> dose transfer and dose-grid helpers.
//
// The layer-summed BEV dose of a beam is sampled once at the divergent fan index
// of every dose voxel inside the transfer box and accumulated in FP64. The
// reference transfers every layer separately into an FP32 grid
// (wrapper.cu:5343-5505); the transfer is linear in the BEV dose, so one pass over
// the summed volume gives the same sum up to rounding.
#include <algorithm>

#include "device_util.cuh"
#include "kernels.h"
#include "launch_util.h"
#include "transfer_walk.cuh"

namespace pbs {

namespace {

// Trilinear sample with texel centres at i + 0.5 and zero outside the volume,
// at texel-space coordinates (x, y, z) = texture coordinate - 0.5.
__device__ __forceinline__ float bev_sample(const float* __restrict__ v, int nx, int ny, int nz, float x, float y,
                                            float z) {
    x = fminf(fmaxf(x, -2.0f), float(nx) + 1.0f);
    y = fminf(fmaxf(y, -2.0f), float(ny) + 1.0f);
    z = fminf(fmaxf(z, -2.0f), float(nz) + 1.0f);
    const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
    const int x0 = int(fx), y0 = int(fy), z0 = int(fz);
    const float tx = x - fx, ty = y - fy, tz = z - fz;
    float c000, c100, c010, c110, c001, c101, c011, c111;
    if (x0 >= 0 && y0 >= 0 && z0 >= 0 && x0 + 1 < nx && y0 + 1 < ny && z0 + 1 < nz) {
        // All eight texels inside: one base address.
        const size_t plane = static_cast<size_t>(nx) * ny;
        const float* p = v + (static_cast<size_t>(z0) * ny + y0) * nx + x0;
        c000 = __ldg(p);
        c100 = __ldg(p + 1);
        c010 = __ldg(p + nx);
        c110 = __ldg(p + nx + 1);
        c001 = __ldg(p + plane);
        c101 = __ldg(p + plane + 1);
        c011 = __ldg(p + plane + nx);
        c111 = __ldg(p + plane + nx + 1);
    } else {
        auto at = [&](int xi, int yi, int zi) -> float {
            if (xi < 0 || yi < 0 || zi < 0 || xi >= nx || yi >= ny || zi >= nz) return 0.0f;
            return __ldg(v + (static_cast<size_t>(zi) * ny + yi) * nx + xi);
        };
        c000 = at(x0, y0, z0);
        c100 = at(x0 + 1, y0, z0);
        c010 = at(x0, y0 + 1, z0);
        c110 = at(x0 + 1, y0 + 1, z0);
        c001 = at(x0, y0, z0 + 1);
        c101 = at(x0 + 1, y0, z0 + 1);
        c011 = at(x0, y0 + 1, z0 + 1);
        c111 = at(x0 + 1, y0 + 1, z0 + 1);
    }
    const float c00 = c000 + (c100 - c000) * tx;
    const float c10 = c010 + (c110 - c010) * tx;
    const float c01 = c001 + (c101 - c001) * tx;
    const float c11 = c011 + (c111 - c011) * tx;
    const float c0 = c00 + (c10 - c00) * ty;
    const float c1 = c01 + (c11 - c01) * ty;
    return c0 + (c1 - c0) * tz;
}

// Transfer box from the eight BEV corners (wrapper.cu:5343-5394) over the steps
// [first, passive). With `live` the corners are those of the cells the superposition
// items can have written (liveLo/liveHi, one cell of trilinear reach added): every
// voxel outside samples only zero cells, so the transfer and the box's readers skip
// it. Returns whether the box holds a voxel; no live cell gives an empty box.
__device__ bool plan_transfer_box(const BeamGeomDev& g, int first, int passive, bool live, const int* liveLo,
                                  const int* liveHi, int start[3], int maxi[3]) {
    start[0] = start[1] = start[2] = 0;
    maxi[0] = maxi[1] = maxi[2] = -1;
    float xs[2] = {-float(kMaxR), float(g.pitchX + kMaxR - 1)};
    float ys[2] = {-float(kMaxR), float(g.pitchY + kMaxR - 1)};
    float zs[2] = {float(first), float(passive - 1)};
    if (live) {
        if (liveLo[0] > liveHi[0]) return false;
        // Padded BEV cell c is ray coordinate c - kMaxR.
        xs[0] = fmaxf(xs[0], float(liveLo[0] - kMaxR - 1));
        xs[1] = fminf(xs[1], float(liveHi[0] - kMaxR + 1));
        ys[0] = fmaxf(ys[0], float(liveLo[1] - kMaxR - 1));
        ys[1] = fminf(ys[1], float(liveHi[1] - kMaxR + 1));
        zs[0] = fmaxf(zs[0], float(first + liveLo[2] - 1));
        zs[1] = fminf(zs[1], float(first + liveHi[2] + 1));
    }
    V3 mx = v3(-1.0f, -1.0f, -1.0f), mn = v3(100000.0f, 100000.0f, 100000.0f);
    for (int zi = 0; zi < 2; ++zi)
        for (int yi = 0; yi < 2; ++yi)
            for (int xi = 0; xi < 2; ++xi) {
                const V3 p = apply(g.rayIdxToDoseIdx, v3(xs[xi], ys[yi], zs[zi]));
                mx.x = fmaxf(mx.x, p.x);
                mx.y = fmaxf(mx.y, p.y);
                mx.z = fmaxf(mx.z, p.z);
                mn.x = fminf(mn.x, p.x);
                mn.y = fminf(mn.y, p.y);
                mn.z = fminf(mn.z, p.z);
            }
    start[0] = max((int(floorf(mn.x)) / 32) * 32, 0);
    start[1] = max(int(floorf(mn.y)), 0);
    start[2] = max(int(floorf(mn.z)), 0);
    maxi[0] = min(int(ceilf(mx.x)), g.doseX - 1);
    maxi[1] = min(int(ceilf(mx.y)), g.doseY - 1);
    maxi[2] = min(int(ceilf(mx.z)), g.doseZ - 1);
    return passive > first && start[0] <= maxi[0] && start[1] <= maxi[1] && start[2] <= maxi[2];
}

// The beam's transfer box: over the deepest superposed step of all layers, or of
// `layer` alone when it is given (plan_transfer_box), and the transfer parameters.
__global__ void transfer_planner_kernel(BeamGeomDev g, BeamStateDev* beam, const LayerStateDev* layer, int live) {
    pdl_trigger();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    // Last kernel of the beam's work list with one thread: hand the beam's error
    // flags to the context's error word, which outlives the beam state.
    if (g.errWord && beam->errorFlags) atomicOr(g.errWord, beam->errorFlags);
    const int first = beam->firstInside;
    const int passive = layer ? layer->calcPassive : beam->maxCalcPassive;
    // The live box is read before any field of the beam state is written.
    int lo[3], hi[3], start[3], maxi[3];
    for (int i = 0; i < 3; ++i) {
        lo[i] = beam->liveLo[i];
        hi[i] = beam->liveHi[i];
    }
    const int valid = plan_transfer_box(g, first, passive, live != 0, lo, hi, start, maxi);
    const ToFan t = invert_and_shift(g.rayIdxToDoseIdx, v3(float(kMaxR), float(kMaxR), -float(first)));
    beam->transfer = make_transfer_params(t);
    for (int i = 0; i < 3; ++i) {
        beam->transferStart[i] = start[i];
        beam->transferMax[i] = maxi[i];
    }
    beam->transferValid = valid;
}

// Batched influence columns: every layer of the chunk [layer0, layer0 + nCols) gets
// the transfer box of its own live cells (LayerStateDev::colStart/colMax/colValid);
// the beam gets the transfer parameters, which do not depend on the layer.
__global__ void column_transfer_planner_kernel(BeamGeomDev g, BeamStateDev* beam, LayerStateDev* ls, int nCols) {
    const int q = threadIdx.x;
    const int first = beam->firstInside;
    if (q == 0) {
        if (g.errWord && beam->errorFlags) atomicOr(g.errWord, beam->errorFlags);
        const ToFan t = invert_and_shift(g.rayIdxToDoseIdx, v3(float(kMaxR), float(kMaxR), -float(first)));
        beam->transfer = make_transfer_params(t);
    }
    if (q < nCols) {
        LayerStateDev& st = ls[q];
        st.colValid = plan_transfer_box(g, first, st.calcPassive, true, st.liveLo, st.liveHi, st.colStart, st.colMax);
    }
}

constexpr int kTransferZChunk = 4;
constexpr int kTransferBlocksPerSM = 8;

// BEV cells [lo, hi] outside of which a volume is zero. `reaches`: whether the sample at
// BEV index (x, y, z) reads a cell of the box.
struct BevBox {
    float lo[3], hi[3];
    __device__ __forceinline__ BevBox(const int l[3], const int h[3]) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            lo[i] = float(l[i] - 1);
            hi[i] = float(h[i] + 1);
        }
    }
    __device__ __forceinline__ bool reaches(float x, float y, float z) const {
        return x >= lo[0] && x <= hi[0] && y >= lo[1] && y <= hi[1] && z >= lo[2] && z <= hi[2];
    }
};

// A column's BEV samples at kTransferZChunk consecutive z from z0 on (0 past `mz` and
// outside the fan): independent loads, so that their latencies overlap. A chunk that only
// reads zero cells is left out as a whole (a test for each voxel would come between the
// loads), and the divergence's divisions are done once where the beam runs across z.
// 512 x 512 x 200 voxels, gantry 240: 237 -> 181 us with both, 227 with the latter alone;
// 20,000 spots along x 187 -> 177. With 2 or 8 voxels in a chunk 206 and 248.
__device__ __forceinline__ void sample_chunk(const BeamGeomDev& g, const float* __restrict__ bev, const BevBox& box,
                                             const TransferParams& T, float zShift, int x, int y, int z0, int mz,
                                             float (&v)[kTransferZChunk]) {
    const V3 start = transfer_start(T, x, y);
    float fx, fy;
    transfer_divergence(T, start, z0, fx, fy);
    V3 f[kTransferZChunk];
    bool any = false;
#pragma unroll
    for (int k = 0; k < kTransferZChunk; ++k) {
        if (k > 0 && T.inc.z != 0.0f) transfer_divergence(T, start, z0 + k, fx, fy);
        f[k] = transfer_fan_idx(T, start, z0 + k, fx, fy);
        any = any || box.reaches(f[k].x, f[k].y, f[k].z - zShift);
        v[k] = 0.0f;
    }
    if (!any) return;
#pragma unroll
    for (int k = 0; k < kTransferZChunk; ++k)
        if (z0 + k <= mz && !(f[k].x + 0.5f < 0.0f || f[k].y + 0.5f < 0.0f || f[k].z + 0.5f < 0.0f))
            v[k] = bev_sample(bev, g.bevX, g.bevY, g.steps, f[k].x, f[k].y, f[k].z - zShift);
}

// primTransfDiv (src/algorithms/prim_transf_kernel.cu:11-44). The reference launches
// ceil(width/32) x ceil(height/8) blocks from the box start, so columns up to the
// next block boundary inside the dose grid are transferred too. Every voxel is
// independent: a persistent grid walks the box, which is known only on the device.
__global__ void __launch_bounds__(256)
transfer_kernel(BeamGeomDev g, const float* __restrict__ bev, const BeamStateDev* __restrict__ beam,
                double* __restrict__ dose) {
    pdl_wait();
    if (!beam->transferValid) return;
    const int sx = beam->transferStart[0], sy = beam->transferStart[1], sz = beam->transferStart[2];
    const int mx = beam->transferMax[0], my = beam->transferMax[1], mz = beam->transferMax[2];
    // Columns of the launch box that lie inside the dose grid.
    const int nx = min(((mx - sx + 1 + 31) / 32) * 32, g.doseX - sx);
    const int ny = min(((my - sy + 1 + 7) / 8) * 8, g.doseY - sy);
    const int nzc = (mz - sz + kTransferZChunk) / kTransferZChunk;
    if (nx <= 0 || ny <= 0 || nzc <= 0) return;
    const TransferParams T = beam->transfer;
    const float zShift = g.compatBevZShift ? float(beam->firstInside) : 0.0f;
    const size_t slice = static_cast<size_t>(g.doseX) * g.doseY;
    const BevBox box(beam->liveLo, beam->liveHi);
    walk_box(T, sx, sy, nx, ny, nzc, [&](int x, int y, int chunk) {
        const int z0 = sz + chunk * kTransferZChunk;
        float v[kTransferZChunk];
        sample_chunk(g, bev, box, T, zShift, x, y, z0, mz, v);
        double* col = dose + static_cast<size_t>(y) * g.doseX + x;
#pragma unroll
        for (int k = 0; k < kTransferZChunk; ++k)
            if (v[k] > 0.0f) col[static_cast<size_t>(z0 + k) * slice] += double(v[k]);
    });
}

__global__ void dose_init_kernel(double* dose, const float* init, size_t n) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        dose[i] = init ? double(init[i]) : 0.0;
}

__global__ void dose_to_float_kernel(const double* dose, float* out, size_t n) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        out[i] = float(dose[i]);
}

// Box [lo, lo + ext) of a [dims.z][dims.y][dims.x] grid: zeroes the FP64 dose there
// (out == nullptr) or converts it to float into the same voxels of `out` and
// sets *nonFinite (if given) where a value is not finite.
__global__ void dose_box_kernel(double* dose, float* out, int3 dims, int3 lo, int3 ext, int* nonFinite) {
    walk_rows(ext.x, ext.y, ext.z, [&](int x, int y, int z) {
        const size_t v = (size_t(z + lo.z) * dims.y + (y + lo.y)) * size_t(dims.x) + (x + lo.x);
        if (out) {
            const float f = float(dose[v]);
            out[v] = f;
            if (nonFinite && !isfinite(f)) *nonFinite = 1;
        } else {
            dose[v] = 0.0;
        }
    });
}

// Batched influence columns: column q (blockIdx.y) samples its own BEV volume
// (bev + q * bevStride) over its layer's transfer box (column_written_box) and adds
// into its own FP64 dose buffer laid out over `fb`. Items and sampling as in
// transfer_kernel; the blocks of a column stride over its items.
__global__ void __launch_bounds__(256)
column_transfer_kernel(BeamGeomDev g, const float* __restrict__ bev, size_t bevStride,
                       const BeamStateDev* __restrict__ beam, const LayerStateDev* __restrict__ ls, ColBox fb,
                       double* __restrict__ colDose) {
    const int q = blockIdx.y;
    int lo[3], hi[3];
    if (!column_written_box(ls[q], g.doseX, g.doseY, fb, lo, hi)) return;
    const int nx = hi[0] - lo[0] + 1, ny = hi[1] - lo[1] + 1;
    const int nzc = (hi[2] - lo[2] + kTransferZChunk) / kTransferZChunk;
    const TransferParams T = beam->transfer;
    const float* v0 = bev + static_cast<size_t>(q) * bevStride;
    const size_t fbN = static_cast<size_t>(fb.ext[0]) * fb.ext[1] * fb.ext[2];
    double* out = colDose + static_cast<size_t>(q) * fbN;
    const size_t slice = static_cast<size_t>(fb.ext[0]) * fb.ext[1];
    const BevBox box(ls[q].liveLo, ls[q].liveHi);
    walk_box(T, lo[0], lo[1], nx, ny, nzc, [&](int x, int y, int chunk) {
        const int z0 = lo[2] + chunk * kTransferZChunk;
        float v[kTransferZChunk];
        sample_chunk(g, v0, box, T, 0.0f, x, y, z0, hi[2], v);
        double* col = out + static_cast<size_t>(y - fb.lo[1]) * fb.ext[0] + (x - fb.lo[0]);
#pragma unroll
        for (int k = 0; k < kTransferZChunk; ++k)
            if (v[k] > 0.0f) col[static_cast<size_t>(z0 + k - fb.lo[2]) * slice] += double(v[k]);
    });
}

// Batched influence columns, row norms: every voxel's samples in the columns whose box
// holds it, squared and added up in column order into the voxel's norm. The sampling
// coordinates are the same in all columns. Against transferring the columns into dose
// buffers of their own and adding those up, no column is written, read and cleared
// again (64 columns on 256 x 256 x 160 voxels: 181 + 434 -> 85 us; with the
// registers of an unbounded kernel, one block per SM, 209).
__global__ void __launch_bounds__(256, 4)
column_norm_kernel(BeamGeomDev g, const float* __restrict__ bev, size_t bevStride,
                   const BeamStateDev* __restrict__ beam, const LayerStateDev* __restrict__ ls, int nCols, ColBox fb,
                   double* __restrict__ norm) {
    extern __shared__ int sBox[];  // [nCols][6]: lo and hi of the column's box (hi < lo: none)
    __shared__ int sAll[6];
    if (threadIdx.x < 6) sAll[threadIdx.x] = threadIdx.x < 3 ? 0x7fffffff : -1;
    __syncthreads();
    for (int q = threadIdx.x; q < nCols; q += blockDim.x) {
        int lo[3], hi[3];
        const bool any = column_written_box(ls[q], g.doseX, g.doseY, fb, lo, hi);
        for (int i = 0; i < 3; ++i) {
            sBox[q * 6 + i] = any ? lo[i] : 0x7fffffff;
            sBox[q * 6 + 3 + i] = any ? hi[i] : -1;
            if (any) {
                atomicMin(&sAll[i], lo[i]);
                atomicMax(&sAll[3 + i], hi[i]);
            }
        }
    }
    __syncthreads();
    if (sAll[3] < sAll[0]) return;
    const TransferParams T = beam->transfer;
    walk_box(T, sAll[0], sAll[1], sAll[3] - sAll[0] + 1, sAll[4] - sAll[1] + 1, sAll[5] - sAll[2] + 1,
             [&](int x, int y, int chunk) {
                 const int z = sAll[2] + chunk;
                 const V3 f = transfer_fan_idx(T, transfer_start(T, x, y), z);
                 if (f.x + 0.5f < 0.0f || f.y + 0.5f < 0.0f || f.z + 0.5f < 0.0f) return;
                 double acc = 0.0;
#pragma unroll 4
                 for (int q = 0; q < nCols; ++q) {
                     const int* b = sBox + q * 6;
                     if (x < b[0] || y < b[1] || z < b[2] || x > b[3] || y > b[4] || z > b[5]) continue;
                     const double v = fmaxf(bev_sample(bev + static_cast<size_t>(q) * bevStride, g.bevX, g.bevY,
                                                       g.steps, f.x, f.y, f.z),
                                            0.0f);
                     acc += v * v;
                 }
                 if (acc != 0.0) norm[(static_cast<size_t>(z) * g.doseY + y) * g.doseX + x] += acc;
             });
}

// Batched influence columns: zeroes column q's float BEV volume over its layer's
// live cells (the only cells its superposition wrote), so every volume is zero for
// the next batch.
__global__ void __launch_bounds__(256) column_bev_clear_kernel(BeamGeomDev g, float* __restrict__ bev, size_t bevStride,
                                                               const LayerStateDev* __restrict__ ls) {
    const int q = blockIdx.y;
    const LayerStateDev& st = ls[q];
    if (st.liveLo[0] > st.liveHi[0]) return;
    const int x0 = max(st.liveLo[0], 0), x1 = min(st.liveHi[0], g.bevX - 1);
    const int y0 = max(st.liveLo[1], 0), y1 = min(st.liveHi[1], g.bevY - 1);
    const int z0 = max(st.liveLo[2], 0), z1 = min(st.liveHi[2], g.steps - 1);
    if (x1 < x0 || y1 < y0 || z1 < z0) return;
    const int w = x1 - x0 + 1, rows = y1 - y0 + 1;
    float* v0 = bev + static_cast<size_t>(q) * bevStride;
    walk_rows(w, rows, z1 - z0 + 1, [&](int x, int y, int z) {
        v0[(static_cast<size_t>(z0 + z) * g.bevY + y0 + y) * g.bevX + x0 + x] = 0.0f;
    });
}

// Box [lo, lo + ext) of the FP64 grid initialised from the same voxels of a float grid.
__global__ void dose_box_init_kernel(double* dose, const float* init, int3 dims, int3 lo, int3 ext) {
    walk_rows(ext.x, ext.y, ext.z, [&](int x, int y, int z) {
        const size_t v = (size_t(z + lo.z) * dims.y + (y + lo.y)) * size_t(dims.x) + (x + lo.x);
        dose[v] = double(init[v]);
    });
}

}  // namespace

cudaError_t launch_dose_box_init(double* dose, const float* init, const int dims[3], const int lo[3], const int hi[3],
                                 cudaStream_t s) {
    for (int i = 0; i < 3; ++i)
        if (lo[i] < 0 || hi[i] >= dims[i] || hi[i] < lo[i]) return cudaErrorInvalidValue;
    const int3 d = make_int3(dims[0], dims[1], dims[2]);
    const int3 l = make_int3(lo[0], lo[1], lo[2]);
    const int3 e = make_int3(hi[0] - lo[0] + 1, hi[1] - lo[1] + 1, hi[2] - lo[2] + 1);
    const size_t total = size_t(e.x) * e.y * e.z;
    const int blocks = int(std::min<size_t>((total + 255) / 256, 148 * 32));
    dose_box_init_kernel<<<blocks, 256, 0, s>>>(dose, init, d, l, e);
    return cudaGetLastError();
}

cudaError_t launch_column_transfer(const BeamGeomDev& g, const float* bev, size_t bevStride, BeamStateDev* beam,
                                   LayerStateDev* ls, int nCols, const ColBox& fb, double* colDose, cudaStream_t s) {
    if (nCols <= 0) return cudaSuccess;
    if (nCols > 1024) return cudaErrorInvalidValue;
    column_transfer_planner_kernel<<<1, ((nCols + 31) / 32) * 32, 0, s>>>(g, beam, ls, nCols);
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // Blocks per column: a few waves over all columns together.
    const int per = std::max(1, (sms * kTransferBlocksPerSM) / nCols);
    column_transfer_kernel<<<dim3(per, nCols), 256, 0, s>>>(g, bev, bevStride, beam, ls, fb, colDose);
    return cudaGetLastError();
}

cudaError_t launch_column_norms(const BeamGeomDev& g, const float* bev, size_t bevStride, BeamStateDev* beam,
                                LayerStateDev* ls, int nCols, const ColBox& fb, double* norm, cudaStream_t s) {
    if (nCols <= 0) return cudaSuccess;
    if (nCols > 1024) return cudaErrorInvalidValue;
    column_transfer_planner_kernel<<<1, ((nCols + 31) / 32) * 32, 0, s>>>(g, beam, ls, nCols);
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = size_t(nCols) * 6 * sizeof(int);
    column_norm_kernel<<<sms * kTransferBlocksPerSM, 256, smem, s>>>(g, bev, bevStride, beam, ls, nCols, fb, norm);
    return cudaGetLastError();
}

cudaError_t launch_column_bev_clear(const BeamGeomDev& g, float* bev, size_t bevStride, const LayerStateDev* ls,
                                    int nCols, cudaStream_t s) {
    if (nCols <= 0) return cudaSuccess;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int per = std::max(1, (sms * 8) / nCols);
    column_bev_clear_kernel<<<dim3(per, nCols), 256, 0, s>>>(g, bev, bevStride, ls);
    return cudaGetLastError();
}

cudaError_t launch_transfer_planner(const BeamGeomDev& g, BeamStateDev* beam, const LayerStateDev* layer, int live,
                                    cudaStream_t s) {
    transfer_planner_kernel<<<1, 32, 0, s>>>(g, beam, layer, live);
    return cudaGetLastError();
}

cudaError_t launch_transfer(const BeamGeomDev& g, const float* bev, const BeamStateDev* beam, double* dose,
                            cudaStream_t s) {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // No more CTAs than the whole grid could need (small grids).
    const long long cap = ((static_cast<long long>(g.doseX) * g.doseY) * ((g.doseZ + kTransferZChunk - 1) / kTransferZChunk) +
                           255) / 256;
    const int blocks = static_cast<int>(std::max<long long>(1, std::min<long long>(cap, sms * kTransferBlocksPerSM)));
    cudaError_t e = launch_pdl(transfer_kernel, dim3(blocks), dim3(256), 0, s, g, bev, beam, dose);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

cudaError_t launch_dose_init(double* dose, const float* init, size_t n, cudaStream_t s) {
    const int blocks = int(std::min<size_t>((n + 255) / 256, 148 * 32));
    dose_init_kernel<<<blocks, 256, 0, s>>>(dose, init, n);
    return cudaGetLastError();
}

cudaError_t launch_dose_to_float(const double* dose, float* out, size_t n, cudaStream_t s) {
    const int blocks = int(std::min<size_t>((n + 255) / 256, 148 * 32));
    dose_to_float_kernel<<<blocks, 256, 0, s>>>(dose, out, n);
    return cudaGetLastError();
}

cudaError_t launch_dose_box(double* dose, float* out, const int dims[3], const int lo[3], const int hi[3],
                            cudaStream_t s, int* nonFinite) {
    for (int i = 0; i < 3; ++i)
        if (lo[i] < 0 || hi[i] >= dims[i] || hi[i] < lo[i]) return cudaErrorInvalidValue;
    const int3 d = make_int3(dims[0], dims[1], dims[2]);
    const int3 l = make_int3(lo[0], lo[1], lo[2]);
    const int3 e = make_int3(hi[0] - lo[0] + 1, hi[1] - lo[1] + 1, hi[2] - lo[2] + 1);
    const size_t total = size_t(e.x) * e.y * e.z;
    const int blocks = int(std::min<size_t>((total + 255) / 256, 148 * 32));
    dose_box_kernel<<<blocks, 256, 0, s>>>(dose, out, d, l, e, nonFinite);
    return cudaGetLastError();
}

}  // namespace pbs
