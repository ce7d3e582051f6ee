// Lateral spread of a tile's sources by interpolation in rSigma, shared by the tile
// superposition and its adjoint.
//
// A source s of a tile spreads over e_s(|dy|) e_s(|dx|) with e_s(0) = erf(r/2),
// e_s(k) = (erf((k+1/2) r) - erf((k-1/2) r)) / 2 and r = rSigma of the source
// (complete_superposition.cu:298-307). That product is a smooth function of r alone,
// so over the range [lo, hi] of a tile's r it equals, to rounding, its polynomial
// interpolant through a few Chebyshev nodes r_j:
//   e_r(dy) e_r(dx) = sum_j L_j(r) e_{r_j}(dy) e_{r_j}(dx).
// The tile's footprint is then a sum over the nodes of plain separable convolutions,
//   F = sum_j E_j(y) * (sum_s idd_s L_j(r_s) delta_s) * E_j(x),
// of node weights that all layers of an item add into: the work per source and layer
// is one polynomial basis instead of 2R+1 footprint rows, and the convolutions are
// done once per item whatever its layers.
//
// Error: the largest deviation of the interpolant over all (dy, dx), relative to the
// source's own peak e_r(0)^2, is bounded by hi/lo alone, whatever r and R; node_count
// takes the fewest nodes that keep it below 2.5e-7 (in 64 bits, R <= 32: 2.32e-7 with 4
// nodes, at r = 3.9, 1.91e-7 with 6, 2.11e-7 with 8). The erf differences of one source
// in 32-bit arithmetic are good to about 1e-6 of that peak.
#pragma once

#include <cuda_runtime.h>

#include "pbs_types.h"

namespace pbs {

constexpr int kMaxNodes = 8;
constexpr int kSplitWide = 23;  // widest radius of the second of the three instances

// Rows of a tile in pairs (y and 7 - y, the two halves of packed FP32 operations), and
// strides of a pair's row and of a node's table in shared memory.
constexpr int kPairs = kTileY / 2;
template <int R>
constexpr int kRowStride = kTileX + 2 * R + 1;
template <int R>
constexpr int kTableStride = ((R + 2) / 2 | 1) * 2;

// r above which e_r is (1, 0, 0, ...) in 32 bits: larger values (a zero sigma) are
// taken as this.
constexpr float kMaxRSigma = 12.0f;
// A range of r wider than kNodeRatio is cut into ranges of that ratio, small r included:
// one range from 0.001 to 0.02 would miss the peak of a source at its lower end by 2e-4.
constexpr float kNodeRatio = 1.6f;

// Chebyshev nodes +-cos((2p+1) pi / 2J), p < J/2, of J = 4, 6, 8 nodes, and
// 1 / (2 x_p prod_{q != p} (x_p^2 - x_q^2)). Node 2p is +x_p, node 2p+1
// is -x_p. Even counts only: the two nodes of a pair share their basis product.
static __constant__ float kNodeX[kMaxNodes / 2 - 1][kMaxNodes / 2] = {{0.9238795f, 0.38268343f},
                                                           {0.9659258f, 0.70710677f, 0.25881904f},
                                                           {0.98078525f, 0.8314696f, 0.55557024f, 0.19509032f}};
static __constant__ float kNodeC[kMaxNodes / 2 - 1][kMaxNodes / 2] = {{0.76536694f, -1.84775922f},
                                                           {1.38036833f, -3.77123645f, 5.15160478f},
                                                           {3.12144614f, -8.88912625f, 13.3035158f, -15.6925653f}};

// Nodes for a range of r with ratio hi/lo (interpolation error below 2.5e-7 of the peak;
// up to kNodeRatio, 8 nodes keep it).
__device__ __forceinline__ int node_count(float ratio) {
    const float d = ratio - 1.0f;
    return 4 + 2 * (d > 0.075f) + 2 * (d > 0.285f);
}

// e_r(k) for r >= 1, out of line: few tiles have sources that narrow.
static __device__ __noinline__ float narrow_spread_weight(float r, int k) {
    const float c = float(k);
    return k == 0 ? erff(0.5f * r) : 0.5f * (erfcf((c - 0.5f) * r) - erfcf((c + 0.5f) * r));
}

// e_r(k). For r < 1 the mean of the Gaussian over the unit cell by Gauss-Legendre
// quadrature (3 points up to r = 0.3, else 5): the difference of two erf values of nearly
// equal size loses its leading digits. In exact arithmetic its error is below 4.4e-8 of
// e_r(0); relative to e_r(k) itself it grows along the tail, to 2.7e-7 at r k = 2.1 and
// 4.5e-6 at r k = 3 (r = 0.3; 4.1e-7 there with 5 points). __expf adds 1e-7 at the centre
// and 1e-6 where e^-9 is left.
__device__ __forceinline__ float spread_weight(float r, int k) {
    if (r >= 1.0f) return narrow_spread_weight(r, k);
    const float c = float(k), r2 = -r * r;
    auto g = [&](float u) { return __expf(r2 * (c + u) * (c + u)); };
    float s;
    if (r < 0.3f)
        s = 0.44444445f * g(0.0f) + 0.27777778f * (g(0.38729834f) + g(-0.38729834f));
    else
        s = 0.28444445f * g(0.0f) + 0.23931434f * (g(0.26923466f) + g(-0.26923466f)) +
            0.11846344f * (g(0.45308992f) + g(-0.45308992f));
    return 0.56418958f * r * s;
}

// The sources (idd, rSigma) of one 32 x 8 tile at one step: 256 consecutive pairs per
// layer, row by row.
struct TileSource {
    const float2* first;  // the tile in the first layer of the item's group
    size_t layerStride;   // pairs between layers
};

// Starts the L2 fetch of a tile's layers, 2 KB each (they come from DRAM on large beams).
__device__ __forceinline__ void prefetch_tile(const TileSource& s, unsigned layers, int lane) {
    if (lane < 16)
#pragma unroll 1
        for (unsigned m = layers; m; m &= m - 1u)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(s.first + static_cast<size_t>(__ffs(m) - 1) * s.layerStride +
                                                          lane * 16));
}

// Starts the copy of a layer's sources to shared memory (16-byte aligned) by the lanes
// of a warp.
__device__ __forceinline__ void copy_tile(const TileSource& s, int layer, float2* dst, int lane) {
    const float2* src = s.first + static_cast<size_t>(layer) * s.layerStride + lane * 2;
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst + lane * 2));
    asm volatile(
        "cp.async.cg.shared.global [%0], [%1], 16;\n\t"
        "cp.async.cg.shared.global [%0 + 512], [%1 + 512], 16;\n\t"
        "cp.async.cg.shared.global [%0 + 1024], [%1 + 1024], 16;\n\t"
        "cp.async.cg.shared.global [%0 + 1536], [%1 + 1536], 16;" ::"r"(d),
        "l"(src)
        : "memory");
}
__device__ __forceinline__ void async_copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Range [lo, hi] of r over the layers of an item from the tile ranges the IDD kernel
// left (lane = layer, range_word); false if no source has a valid r > 0.
__device__ __forceinline__ bool item_range(unsigned laneRange, float& lo, float& hi) {
    const unsigned h = __reduce_max_sync(0xffffffffu, laneRange >> 16);
    const unsigned l = __reduce_min_sync(0xffffffffu, laneRange ? laneRange & 0xffffu : 0xffffu);
    hi = fminf(__uint_as_float(h << 15), kMaxRSigma);  // (NaN too)
    lo = fminf(fmaxf(__uint_as_float(l << 15), 1.0e-12f), kMaxRSigma);
    return h != 0u && hi >= lo;
}

// One range of r and its nodes: r = mid + half t, t in [-1, 1].
struct NodeRange {
    float from, to;  // sources with from < r <= to; r above `top` is taken as `top`
    float top;
    float mid, half;
    float invHalf, shift;  // t = r invHalf + shift
    int count;
};

// The range that starts at lo (sources above `from`), at most up to hi. The last range
// takes every larger r.
__device__ __forceinline__ NodeRange node_range(float from, float lo, float hi) {
    NodeRange n;
    n.from = from;
    n.top = fminf(hi, kNodeRatio * lo);
    n.to = n.top >= hi ? __int_as_float(0x7f800000) : n.top;
    n.mid = 0.5f * (lo + n.top);
    n.half = 0.5f * (n.top - lo);
    n.invHalf = n.half > 0.0f ? 1.0f / n.half : 0.0f;
    n.shift = -n.mid * n.invHalf;
    n.count = node_count(n.top / lo);
    return n;
}

// prod_{q != p} (u - x_q^2) for the pairs p of J nodes, two values of u at a time: the
// basis of node +-x_p at t is C_p (t +- x_p) times this, up to the node's sign.
template <int J>
__device__ __forceinline__ void pair_products(float2 u, float2 (&b)[J / 2]) {
    float2 f[J / 2];
#pragma unroll
    for (int p = 0; p < J / 2; ++p) {
        const float q = -kNodeX[J / 2 - 2][p] * kNodeX[J / 2 - 2][p];
        f[p] = __fadd2_rn(u, make_float2(q, q));
    }
    if constexpr (J == 4) {
        b[0] = f[1];
        b[1] = f[0];
    } else if constexpr (J == 6) {
        b[0] = __fmul2_rn(f[1], f[2]);
        b[1] = __fmul2_rn(f[0], f[2]);
        b[2] = __fmul2_rn(f[0], f[1]);
    } else {
        const float2 f01 = __fmul2_rn(f[0], f[1]), f23 = __fmul2_rn(f[2], f[3]);
        b[0] = __fmul2_rn(f[1], f23);
        b[1] = __fmul2_rn(f[0], f23);
        b[2] = __fmul2_rn(f01, f[3]);
        b[3] = __fmul2_rn(f01, f[2]);
    }
}

// Position of node j of n.count.
__device__ __forceinline__ float node_at(const NodeRange& n, int j) {
    const float x = kNodeX[n.count / 2 - 2][j >> 1];
    return fmaf(n.half, j & 1 ? -x : x, n.mid);
}

// Node tables of `count` nodes from `node0` on: (e_{r_j}(k), e_{r_j}(k)) at
// e[(j - node0) * stride + k], k = 0..R, by the lanes of a warp.
__device__ __forceinline__ void node_tables(const NodeRange& n, int node0, int count, int R, float2* __restrict__ e,
                                            int stride, int lane) {
    const int per = R + 1;
    const unsigned inv = 65536u / per + 1u;  // i / per = i inv / 65536 for i < 8 (kMaxR + 1)
#pragma unroll 1
    for (int i = lane; i < count * per; i += 32) {
        const int j = static_cast<int>(i * inv >> 16), k = i - j * per;
        const float v = spread_weight(node_at(n, node0 + j), k);
        e[j * stride + k] = make_float2(v, v);
    }
}

// Calls f.template run<J>() for the range's node count J.
template <int J = 4, typename F>
__device__ __forceinline__ void with_nodes(int count, F&& f) {
    if (count == J || J == kMaxNodes) {
        f.template run<J>();
        return;
    }
    if constexpr (J < kMaxNodes) with_nodes<J + 2>(count, f);
}

}  // namespace pbs
