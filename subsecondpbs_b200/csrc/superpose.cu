// Tile-based Gaussian superposition of the per-ray IDD into the padded BEV dose.
//
// Each work item is one 32x8 tile of source rays at one step with its batched radius
// R (kernelSuperposition<R>, complete_superposition.cu:264-335) and a set of layers
// whose tile has that radius at that step (their footprints land on the same BEV
// cells). Every source s spreads idd_s * e_s(dy) * e_s(dx) over a (2R+1)^2 footprint.
//
// One warp takes one item at a time (persistent grid, no CTA barrier):
//   * range: the item's smallest and largest rSigma, hence its interpolation nodes
//     (node_spread.cuh: 4 or 6 on most items, 8 at most);
//   * weights: lane x holds source column x and adds every layer's idd_s L_j(r_s) into
//     the node weights w_j[sy][x];
//   * rows: lane = one (node, source row); a transposed FIR filter walks the row once,
//     two taps per |d|, and overwrites w_j[sy] with its spread T_j[sy][0 .. 32+2R);
//   * columns: lane = one footprint column (or one half of it: the footprint is
//     symmetric under y -> H-1-y, sy -> 7-sy, so the halves run the same code); the
//     column's rows are summed over nodes and source rows in registers, with one
//     shared-memory load per (node, source row);
//   * write-out: the rows are added to the BEV dose of the item's step (all layers of
//     the beam share one BEV volume) in 64-bit fixed point: a BEV cell sums many
//     items, and integer adds commute, so the dose does not depend on the order in
//     which the items land. The chunk's exponent (layer_plan_kernel) bounds every cell
//     below 2^62; a last pass adds the chunk to the float BEV and clears it.
#include <algorithm>

#include "device_util.cuh"
#include "kernels.h"
#include "launch_util.h"
#include "node_spread.cuh"
#include "work_blocks.cuh"

namespace pbs {

namespace {

// Nodes whose rows a warp holds at a time; 8 nodes go in two halves.
constexpr int kRowNodes = 6;
__device__ __forceinline__ int batch_nodes(int count) { return count > kRowNodes ? count / 2 : count; }

// Shared memory of one warp for radii up to RMax: the node tables, then kRowNodes x 4
// rows of pairs (source rows y and 7 - y of one node, as the two halves of packed FP32
// operations). Rows and tables have odd strides (in 8 and 16 bytes), so that the lanes
// of the row pass, one row each, read distinct banks.
template <int RMax>
constexpr int kWarpPairs = kRowNodes * (kTableStride<RMax> + kPairs * kRowStride<RMax>);

// Node weights of a tile: rows[((j - node0) * 4 + y) * stride + lane] for the row pair
// (y, 7 - y) and the batch of nodes from node0 on. Per source the even and odd parts
// E_p = sum idd B_p(t^2), S_p = sum idd t B_p(t^2) of each node pair are summed over the
// layers; the weights are C_p (x_p E_p +- S_p). The layers' sources are copied into the
// shared memory of the rows, which are written only after the last layer, as many
// layers at a time as fit: all their loads are in flight at once, where loads into
// registers would hold two row pairs of one layer.
struct WeightPass {
    const TileSource& s;
    const NodeRange& n;
    unsigned layers;
    int node0;
    float2* rows;
    int room;  // layers that fit
    int stride, lane;

    template <int J>
    __device__ __forceinline__ void run() const {
        const float2 shift = make_float2(n.shift, n.shift), inv = make_float2(n.invHalf, n.invHalf);
        float2 even[kPairs][J / 2], odd[kPairs][J / 2];
#pragma unroll
        for (int y = 0; y < kPairs; ++y)
#pragma unroll
            for (int p = 0; p < J / 2; ++p) even[y][p] = odd[y][p] = make_float2(0.0f, 0.0f);
#pragma unroll 1
        for (unsigned m = layers; m;) {
            int staged = 0;
#pragma unroll 1
            for (; m && staged < room; m &= m - 1u, ++staged)
                copy_tile(s, __ffs(m) - 1, rows + staged * kTileSources, lane);
            async_copies_wait();
            __syncwarp();
            const float2* f = rows + lane;
#pragma unroll 1
            for (; staged > 0; --staged, f += kTileSources) {
#pragma unroll
                for (int y = 0; y < kPairs; ++y) {
                    const float2 u = f[y * kTileX], v = f[(kTileY - 1 - y) * kTileX];
                    float2 dose;
                    dose.x = u.y > n.from && u.y <= n.to ? fmaxf(u.x, 0.0f) : 0.0f;
                    dose.y = v.y > n.from && v.y <= n.to ? fmaxf(v.x, 0.0f) : 0.0f;
                    // Every t is finite: sources outside the range carry no dose.
                    const float2 t = __ffma2_rn(make_float2(fminf(u.y, n.top), fminf(v.y, n.top)), inv, shift);
                    float2 b[J / 2];
                    pair_products<J>(__fmul2_rn(t, t), b);
#pragma unroll
                    for (int p = 0; p < J / 2; ++p) {
                        const float2 q = __fmul2_rn(dose, b[p]);
                        even[y][p] = __fadd2_rn(even[y][p], q);
                        odd[y][p] = __ffma2_rn(q, t, odd[y][p]);
                    }
                }
            }
            __syncwarp();
        }
#pragma unroll
        for (int p = 0; p < J / 2; ++p) {
            const int j = 2 * p - node0;
            if (J > kRowNodes && (j < 0 || j >= J / 2)) continue;
            const float c = kNodeC[J / 2 - 2][p], cx = c * kNodeX[J / 2 - 2][p];
#pragma unroll
            for (int y = 0; y < kPairs; ++y) {
                const float2 ev = __fmul2_rn(even[y][p], make_float2(cx, cx));
                rows[(j * kPairs + y) * stride + lane] = __ffma2_rn(odd[y][p], make_float2(c, c), ev);
                rows[((j + 1) * kPairs + y) * stride + lane] = __ffma2_rn(odd[y][p], make_float2(-c, -c), ev);
            }
        }
    }
};

// Rows: every row is convolved with its node's e in place. After source column x the
// pending sums a[i] belong to columns x + 1 + i; column x is complete. Up to radius 15 a
// lane takes one row pair in packed operations; above, where the pending sums of a pair
// do not fit the registers, one row.
template <int R>
__device__ __forceinline__ void spread_rows(float2* __restrict__ rows, const float2* __restrict__ e, int nodes,
                                            int lane) {
    constexpr int U = 2;  // source columns per step: more would crowd the instruction cache
    if constexpr (R <= 15) {
        if (lane < nodes * kPairs) {
            float2 k[kTableStride<R>];
            const float4* e4 = reinterpret_cast<const float4*>(e + (lane / kPairs) * kTableStride<R>);
#pragma unroll
            for (int q = 0; q < (R + 2) / 2; ++q) {
                const float4 v = e4[q];
                k[2 * q] = make_float2(v.x, v.y);
                k[2 * q + 1] = make_float2(v.z, v.w);
            }
            float2* p = rows + lane * kRowStride<R>;
            float2 a[2 * R + 1];
#pragma unroll
            for (int i = 0; i <= 2 * R; ++i) a[i] = make_float2(0.0f, 0.0f);
#pragma unroll 1
            for (int x = 0; x < kTileX; x += U) {
                float2 v[U], out[U];
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = p[x + u];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    out[u] = __ffma2_rn(v[u], k[R], a[0]);
#pragma unroll
                    for (int i = 0; i < 2 * R; ++i)
                        a[i] = __ffma2_rn(v[u], k[i + 1 < R ? R - 1 - i : i + 1 - R], a[i + 1]);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) p[x + u] = out[u];
            }
#pragma unroll
            for (int i = 0; i < 2 * R; ++i) p[kTileX + i] = a[i];
        }
    } else {
#pragma unroll 1
        for (int row = lane; row < nodes * kTileY; row += 32) {
            float k[kTableStride<R>];
            const float4* e4 = reinterpret_cast<const float4*>(e + (row / kTileY) * kTableStride<R>);
#pragma unroll
            for (int q = 0; q < (R + 2) / 2; ++q) {
                const float4 v = e4[q];
                k[2 * q] = v.x;
                k[2 * q + 1] = v.z;
            }
            float* p = reinterpret_cast<float*>(rows + (row >> 1) * kRowStride<R>) + (row & 1);
            float a[2 * R + 1];
#pragma unroll
            for (int i = 0; i <= 2 * R; ++i) a[i] = 0.0f;
#pragma unroll 1
            for (int x = 0; x < kTileX; x += U) {
                float v[U], out[U];
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = p[2 * (x + u)];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    out[u] = fmaf(v[u], k[R], a[0]);
#pragma unroll
                    for (int i = 0; i < 2 * R; ++i)
                        a[i] = fmaf(v[u], k[i + 1 < R ? R - 1 - i : i + 1 - R], a[i + 1]);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) p[2 * (x + u)] = out[u];
            }
#pragma unroll
            for (int i = 0; i < 2 * R; ++i) p[2 * (kTileX + i)] = a[i];
        }
    }
}

// Adds a footprint value (scaled to the BEV's fixed point) to a BEV cell. A batch of
// nodes, or the rounding of the interpolation, can make it negative: the cells are
// two's complement and their sum is taken as zero where it ends below it.
__device__ __forceinline__ void add_to_bev(unsigned long long* cell, float v) {
    if (fabsf(v) >= 0.5f) atomicAdd(cell, static_cast<unsigned long long>(__float2ll_rn(v)));
}

// A BEV cell as a float.
__device__ __forceinline__ float from_bev(unsigned long long cell, double unit) {
    return fmaxf(float(double(static_cast<long long>(cell)) * unit), 0.0f);
}

// Columns: a lane takes one footprint column, rows y and H-1-y as a pair (under
// y -> H-1-y, sy -> 7-sy the footprint's form does not change), 32 columns at a time.
// The last W % 32 columns go to several groups of lanes, each with every G-th node, whose
// sums are added up. A finished strip of columns is laid over the rows it came from
// (each column is read by its own pass only) and added to the BEV by a loop: the same
// straight-line code for every footprint row would not fit the instruction cache.
template <int R>
__device__ __forceinline__ void spread_columns(float2* __restrict__ rows, const float2* __restrict__ e, int nodes,
                                               int lane, unsigned long long* __restrict__ dst, int bevX,
                                               float scale) {
    constexpr int W = kTileX + 2 * R, H = kTileY + 2 * R, N = H / 2;
    constexpr int kLast = W % 32;
    constexpr int kLastShift = kLast == 0 ? 0 : (kLast <= 4 ? 3 : (kLast <= 8 ? 2 : (kLast <= 16 ? 1 : 0)));
    constexpr int kSlots = kRowNodes * kPairs;  // rows of the strip
#pragma unroll 1
    for (int base = 0; base < W; base += 32) {
        const bool last = kLast > 0 && base + 32 > W;
        const int shift = last ? kLastShift : 0;
        const int groups = 1 << shift, width = 32 >> shift;
        const int group = lane >> (5 - shift), xi = lane & (width - 1);
        const int n = last ? kLast : 32;
        const int x = base + min(xi, n - 1);
        float2 acc[N];
#pragma unroll
        for (int i = 0; i < N; ++i) acc[i] = make_float2(0.0f, 0.0f);
#pragma unroll 1
        for (int j = group; j < nodes; j += groups) {
            const float2* p = rows + j * kPairs * kRowStride<R> + x;
            float2 t[kTileY];
#pragma unroll
            for (int y = 0; y < kPairs; ++y) {
                const float2 v = p[y * kRowStride<R>];
                t[y] = v;
                t[kTileY - 1 - y] = make_float2(v.y, v.x);
            }
            const float4* e4 = reinterpret_cast<const float4*>(e + j * kTableStride<R>);
#pragma unroll
            for (int q = 0; q < (R + 2) / 2; ++q) {
                // Keeps later table entries out of the registers until they are needed.
                if (q > 0 && q % 2 == 0) asm volatile("" ::: "memory");
                const float4 w = e4[q];
                const float2 wk[2] = {make_float2(w.x, w.y), make_float2(w.z, w.w)};
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int k = 2 * q + c;
                    if (k <= R) {
#pragma unroll
                        for (int y = 0; y < kTileY; ++y) {
                            if (y + R + k < N) acc[y + R + k] = __ffma2_rn(t[y], wk[c], acc[y + R + k]);
                            if (k > 0 && y + R - k < N) acc[y + R - k] = __ffma2_rn(t[y], wk[c], acc[y + R - k]);
                        }
                    }
                }
            }
        }
        __syncwarp();
#pragma unroll 1
        for (int o = 16; o >= width; o >>= 1)
#pragma unroll
            for (int i = 0; i < N; ++i) {
                acc[i].x += __shfl_down_sync(0xffffffffu, acc[i].x, o);
                acc[i].y += __shfl_down_sync(0xffffffffu, acc[i].y, o);
            }
#pragma unroll
        for (int i0 = 0; i0 < N; i0 += kSlots) {
            __syncwarp();
            if (lane < n)
#pragma unroll
                for (int i = i0; i < N && i < i0 + kSlots; ++i) rows[(i - i0) * kRowStride<R> + x] = acc[i];
            __syncwarp();
            const int end = min(N, i0 + kSlots);
            unsigned lo = (i0 + group) * bevX + x, hi = (H - 1 - i0 - group) * bevX + x;
            const float2* f = rows + group * kRowStride<R> + x;
#pragma unroll 1
            for (int i = i0 + group; i < end; i += groups) {
                const float2 v = *f;
                if (xi < n) {
                    add_to_bev(dst + lo, v.x * scale);
                    add_to_bev(dst + hi, v.y * scale);
                }
                f += groups * kRowStride<R>;
                lo += groups * bevX;
                hi -= groups * bevX;
            }
        }
    }
}

// The convolutions of an item at its radius.
template <int R, int RHi>
__device__ __forceinline__ void spread_item(int r, float2* rows, float2* e, int nodes, int lane,
                                            unsigned long long* dst, int bevX, float scale) {
    if (r == R) {
        spread_rows<R>(rows, e, nodes, lane);
        __syncwarp();
        spread_columns<R>(rows, e, nodes, lane, dst, bevX, scale);
        return;
    }
    if constexpr (R < RHi) spread_item<R + 1, RHi>(r, rows, e, nodes, lane, dst, bevX, scale);
}

// An item as a warp takes it from the work list, with the tile ranges of its layers
// (lane = layer).
struct Item {
    unsigned layers;
    int tile, zRel, R, base;
    unsigned range;
};

// Persistent warps over the items of radii RLo..RHi, claimed one at a time through the
// range's counter. A claim is made two items ahead, and the next item is read and its
// layers fetched into L2 while the current one runs, so that their latencies are hidden.
// Items are taken radius block by radius block, so the warps of an SM mostly run the
// code of one radius at a time.
//
// The three instances of a beam (radii 24..32, 16..23 and 0..15, by the registers and
// shared memory they need) are launched back to back with programmatic dependent launch: every CTA lets
// the next instance start at once (its items are independent of this instance's: both
// only add to the fixed-point BEV), so the next instance's CTAs take the SMs this
// instance's CTAs leave at its tail. Before it exits a CTA waits for the previous
// instance to complete, so an instance is complete only once the earlier one is, and the
// kernel after the last one sees every item's adds. An instance of its own for radii up
// to 7 (20 warps per SM instead of 16) was 2 to 9 % slower: its launch and tail cost more.
template <int RLo, int RHi, int Warps, int MinBlocks>
__global__ void __launch_bounds__(Warps * 32, MinBlocks)
superpose_kernel(BeamGeomDev g, const float2* __restrict__ sources, const unsigned* __restrict__ tileRange,
                 const int4* __restrict__ work, BeamStateDev* __restrict__ beam, unsigned long long* __restrict__ bev,
                 int shiftOffset, size_t layerBevStride) {
    extern __shared__ __align__(16) float2 sm[];
    __shared__ RadiusBlocks<RLo, RHi> sBlocks;

    pdl_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int* counter = RLo > kSplitWide ? &beam->workNext : (RLo > kSplitR ? &beam->workNextSmall : &beam->workNextTiny);
    const int tiles = g.tilesX * g.tilesY;
    const size_t padPlane = static_cast<size_t>(tiles) * kTileSources;
    const size_t bevPlane = static_cast<size_t>(g.bevX) * g.bevY;
    float2* e = sm + warp * kWarpPairs<RHi>;
    float2* rows = e + kRowNodes * kTableStride<RHi>;
    constexpr int kRoom = kRowNodes * kPairs * kRowStride<RHi> / kTileSources;  // layers, 256 pairs each

    load_blocks<RLo, RHi>(beam, sBlocks);
    __syncthreads();
    const float scale = ldexpf(1.0f, beam->fixedShift + shiftOffset);
    const int total = sBlocks.total;

    TileSource s;
    s.layerStride = static_cast<size_t>(g.steps) * padPlane;
    auto source = [&](const Item& it) {
        s.first = sources + it.base * s.layerStride + it.zRel * padPlane + it.tile * kTileSources;
    };
    auto fetch = [&](int c) {
        Item it = {};
        if (c < total) {
            const int4 w = work[block_slot<RLo, RHi>(sBlocks, c)];
            it.layers = static_cast<unsigned>(w.x);
            it.tile = w.y;
            it.zRel = w.z;
            it.R = w.w & 0xff;
            it.base = w.w >> 8;
            if (it.layers >> lane & 1u)
                it.range = tileRange[(static_cast<size_t>(it.base + lane) * g.steps + it.zRel) * tiles + it.tile];
        }
        return it;
    };
    // The first item of every warp is fixed; the counter deals out the others. The blocks of
    // an SM, every sms-th one, start on neighbouring items, so that its warps run the code of
    // one radius: the straight-line code of several does not fit the instruction cache. Where
    // radii are many and items few (7500 of radii 0..16, one layer each) a stride of the grid
    // left 3.3 of 9.5 stall cycles per instruction to that: 137 -> 130 us.
    // With fewer items than warps nothing is left to even out the SMs that got the wide radii:
    // the stride shares them out (one layer of 91 spots: 28.6 us, neighbours 30.7).
    const int warps = gridDim.x * Warps, sms = gridDim.x / MinBlocks;
    int claim = 0;
    if (lane == 0) claim = warps + atomicAdd(counter, 1);
    Item next = fetch(total < warps ? blockIdx.x + warp * gridDim.x
                                    : ((blockIdx.x % sms) * MinBlocks + blockIdx.x / sms) * Warps + warp);
    while (next.layers) {
        const Item it = next;
        next = fetch(__shfl_sync(0xffffffffu, claim, 0));
        if (lane == 0) claim = warps + atomicAdd(counter, 1);
        if (next.layers) {
            source(next);
            prefetch_tile(s, next.layers, lane);
        }
        const int R = it.R;
        if (R < RLo || R > RHi) {
            if (lane == 0) atomicOr(&beam->errorFlags, 2);
            continue;
        }
        float lo, hi;
        if (!item_range(it.range, lo, hi)) continue;
        source(it);
        const int tx = it.tile % g.tilesX, ty = it.tile / g.tilesX;
        // One BEV volume per layer when layerBevStride is set (one-layer items: batched
        // influence columns), else one volume for all layers.
        unsigned long long* dst = bev + (it.base + __ffs(it.layers) - 1) * layerBevStride +
                                  static_cast<size_t>(it.zRel) * bevPlane +
                                  static_cast<size_t>(ty * kTileY - R + kMaxR) * g.bevX + (tx * kTileX - R + kMaxR);
        const int stride = kTileX + 2 * R + 1, eStride = ((R + 2) / 2 | 1) * 2;
        for (float from = 0.0f;;) {
            const NodeRange n = node_range(from, lo, hi);
            const int batch = batch_nodes(n.count);
            for (int node0 = 0; node0 < n.count; node0 += batch) {
                node_tables(n, node0, batch, R, e, eStride, lane);
                with_nodes(n.count, WeightPass{s, n, it.layers, node0, rows, kRoom, stride, lane});
                __syncwarp();
                spread_item<RLo, RHi>(R, rows, e, batch, lane, dst, g.bevX, scale);
                __syncwarp();
            }
            if (n.top >= hi) break;
            from = lo = n.top;
        }
    }
    pdl_wait();
}

// `overlap`: launch as a programmatic dependent of the previous kernel on `s` (the
// previous superposition instance).
template <int RLo, int RHi, int Warps, int MinBlocks>
cudaError_t launch_range(const BeamGeomDev& g, const float2* sources, const unsigned* tileRange, const int4* work,
                         BeamStateDev* beam, unsigned long long* bev, int shiftOffset, int numSMs, bool overlap,
                         size_t layerBevStride, cudaStream_t s) {
    auto k = superpose_kernel<RLo, RHi, Warps, MinBlocks>;
    const size_t smem = size_t(Warps) * kWarpPairs<RHi> * sizeof(float2);
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
    return cudaLaunchKernelEx(&cfg, k, g, sources, tileRange, work, beam, bev, shiftOffset, layerBevStride);
}

// Adds the fixed-point BEV of the chunk to the float BEV and clears it for the next
// superposition, over the cells the items can have written: the box of live cells
// (BeamStateDev::liveLo/liveHi, from work_merge_kernel) within the planes written so
// far, [0, maxCalcPassive - firstInside). Every cell is converted once, so the float BEV is
// the same on every run.
__global__ void __launch_bounds__(256) bev_fixed_to_float_kernel(BeamGeomDev g, const BeamStateDev* __restrict__ beam,
                                                                 unsigned long long* __restrict__ fixed,
                                                                 float* __restrict__ bev, int shiftOffset) {
    pdl_wait();
    const int planes = min(beam->maxCalcPassive - beam->firstInside, g.steps);
    if (planes <= 0 || beam->liveLo[0] > beam->liveHi[0]) return;
    // bevX is even (the padded ray pitch plus 2 kMaxR), so cells go in aligned pairs.
    const int x0 = max(beam->liveLo[0], 0) & ~1, x1 = min(beam->liveHi[0], g.bevX - 1) | 1;
    const int y0 = max(beam->liveLo[1], 0), y1 = min(beam->liveHi[1], g.bevY - 1);
    const int z0 = max(beam->liveLo[2], 0), z1 = min(beam->liveHi[2], planes - 1);
    if (x1 < x0 || y1 < y0 || z1 < z0) return;
    const int pw = (x1 - x0 + 1) / 2, rows = y1 - y0 + 1;
    const double unit = ldexp(1.0, -(beam->fixedShift + shiftOffset));
    ulonglong2* f2 = reinterpret_cast<ulonglong2*>(fixed);
    float2* b2 = reinterpret_cast<float2*>(bev);
    walk_rows(pw, rows, z1 - z0 + 1, [&](int xp, int y, int z) {
        const size_t pr = ((static_cast<size_t>(z0 + z) * g.bevY + y0 + y) * g.bevX + x0) / 2 + xp;
        const ulonglong2 v = f2[pr];
        if (v.x | v.y) {
            float2 o = b2[pr];
            o.x += from_bev(v.x, unit);
            o.y += from_bev(v.y, unit);
            b2[pr] = o;
            f2[pr] = make_ulonglong2(0ull, 0ull);
        }
    });
}

// Warps per CTA and resident CTAs per SM of the instances.
constexpr int kWidestWarps = 5, kWidestBlocks = 2;
constexpr int kWideWarps = 4, kWideBlocks = 3;
constexpr int kNarrowWarps = 4, kNarrowBlocks = 4;

}  // namespace

namespace {

// The three instances over `work` (items sorted by range: the wide radii first).
cudaError_t launch_instances(const BeamGeomDev& g, const float2* sources, const unsigned* tileRange, const int4* work,
                             BeamStateDev* beam, unsigned long long* bevFixed, int shiftOffset, int numSMs,
                             size_t layerBevStride, cudaStream_t s) {
    cudaError_t e = launch_range<kSplitWide + 1, kMaxR, kWidestWarps, kWidestBlocks>(
        g, sources, tileRange, work, beam, bevFixed, shiftOffset, numSMs, false, layerBevStride, s);
    if (e != cudaSuccess) return e;
    e = launch_range<kSplitR + 1, kSplitWide, kWideWarps, kWideBlocks>(g, sources, tileRange, work, beam, bevFixed,
                                                                       shiftOffset, numSMs, true, layerBevStride, s);
    if (e != cudaSuccess) return e;
    return launch_range<0, kSplitR, kNarrowWarps, kNarrowBlocks>(g, sources, tileRange, work, beam, bevFixed, shiftOffset,
                                                                 numSMs, true, layerBevStride, s);
}

// A superposition over the chunk's whole one-layer work list (work_scatter_kernel):
// radius block R is [rStart[R], rStart[R - 1]) (or up to workCount), and the claim
// counters restart.
__global__ void one_layer_list_view_kernel(BeamStateDev* __restrict__ beam) {
    const int t = threadIdx.x;
    if (t <= kMaxR) {
        const int end = t > 0 ? beam->rStart[t - 1] : beam->workCount;
        beam->mergedR[t] = max(end - beam->rStart[t], 0);
    }
    if (t == 0) {
        beam->workNext = 0;
        beam->workNextSmall = 0;
        beam->workNextTiny = 0;
    }
}

// Batched influence columns: bev_fixed_to_float_kernel for volume q (blockIdx.y) over
// its layer's live cells (LayerStateDev::liveLo/liveHi).
__global__ void __launch_bounds__(256) column_fixed_to_float_kernel(BeamGeomDev g, const BeamStateDev* __restrict__ beam,
                                                                    const LayerStateDev* __restrict__ ls,
                                                                    unsigned long long* __restrict__ fixed,
                                                                    float* __restrict__ bev, size_t stride) {
    const int q = blockIdx.y;
    const LayerStateDev& st = ls[q];
    if (st.liveLo[0] > st.liveHi[0]) return;
    const int x0 = max(st.liveLo[0], 0) & ~1, x1 = min(st.liveHi[0], g.bevX - 1) | 1;
    const int y0 = max(st.liveLo[1], 0), y1 = min(st.liveHi[1], g.bevY - 1);
    const int z0 = max(st.liveLo[2], 0), z1 = min(st.liveHi[2], g.steps - 1);
    if (x1 < x0 || y1 < y0 || z1 < z0) return;
    const int pw = (x1 - x0 + 1) / 2, rows = y1 - y0 + 1;
    const double unit = ldexp(1.0, -beam->fixedShift);
    // stride is even (bevX is), so every volume starts on a cell pair.
    ulonglong2* f2 = reinterpret_cast<ulonglong2*>(fixed + static_cast<size_t>(q) * stride);
    float2* b2 = reinterpret_cast<float2*>(bev + static_cast<size_t>(q) * stride);
    walk_rows(pw, rows, z1 - z0 + 1, [&](int xp, int y, int z) {
        const size_t pr = ((static_cast<size_t>(z0 + z) * g.bevY + y0 + y) * g.bevX + x0) / 2 + xp;
        const ulonglong2 v = f2[pr];
        if (v.x | v.y) {
            float2 o = b2[pr];
            o.x += from_bev(v.x, unit);
            o.y += from_bev(v.y, unit);
            b2[pr] = o;
            f2[pr] = make_ulonglong2(0ull, 0ull);
        }
    });
}

}  // namespace

cudaError_t launch_superpose(const BeamGeomDev& g, const float2* sources, const unsigned* tileRange, const int4* work,
                             BeamStateDev* beam, float* bev, unsigned long long* bevFixed, int shiftOffset, int numSMs,
                             cudaStream_t s) {
    cudaError_t e = launch_instances(g, sources, tileRange, work, beam, bevFixed, shiftOffset, numSMs, 0, s);
    if (e != cudaSuccess) return e;
    e = launch_pdl(bev_fixed_to_float_kernel, dim3(numSMs * 8), dim3(256), 0, s, g,
                   static_cast<const BeamStateDev*>(beam), bevFixed, bev, shiftOffset);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

cudaError_t launch_superpose_columns(const BeamGeomDev& g, const float2* sources, const unsigned* tileRange,
                                     const int4* work,
                                     BeamStateDev* beam, const LayerStateDev* ls, int nCols, float* bev,
                                     unsigned long long* bevFixed, size_t stride, int numSMs, cudaStream_t s) {
    if (nCols <= 0) return cudaSuccess;
    if (stride % 2) return cudaErrorInvalidValue;
    one_layer_list_view_kernel<<<1, 64, 0, s>>>(beam);
    cudaError_t e = launch_instances(g, sources, tileRange, work, beam, bevFixed, 0, numSMs, stride, s);
    if (e != cudaSuccess) return e;
    const int per = std::max(1, (numSMs * 8) / nCols);
    column_fixed_to_float_kernel<<<dim3(per, nCols), 256, 0, s>>>(g, beam, ls, bevFixed, bev, stride);
    return cudaGetLastError();
}

}  // namespace pbs
