// gpu_build.cu -- binned SAH BVH build on the GPU, breadth first (one pass of
// kernels per tree level), producing the same tree as the host builder
// (bvh_build.cpp, the reference's algorithm family: src/scene/bvhBuilder.cpp:115-312).
//
// Why the trees match: every quantity that decides a split is order independent or
// computed with the host's operations in the host's order -- node and centroid
// bounds are exact minima / maxima, bin indices are int((c - c0) * (B / ext)) with
// each operation rounded alone, bin boxes are exact, and the SAH sweep runs on one
// thread in the host's axis / bin order with the same FP64 area and cost formulas.
// The partition is stable, so every node's triangle range stays sorted by triangle
// index (the ranges start as 0..N-1); the host's median fallback (all centroids
// equal: nth_element on (centroid, index)) is then the first half of the range.
// Only the order of triangles inside a leaf differs from the host build (which
// partitions with std::partition).
//
// Per level: big nodes (more than kWarpMax triangles) get their bounds and bins from
// grid-wide atomics (warp-aggregated), small nodes one warp each with bins in shared
// memory; then flags, one exclusive scan over all positions, a stable scatter, and
// child allocation.  Nodes are numbered breadth first on the device.  One
// device-to-host read per level (the next level's node count); no kernel waits on
// another.
//
// The rest of a scene's set-up runs here too: triangle boxes and centroids before the
// build, the collapse to 4-wide nodes after it (one pass down that opens children, one up
// that counts subtrees, one down that numbers and writes the nodes depth first, as the
// host's collapse does), and the search for coincident faces of opposite winding.  On the
// host they took three quarters of a set-up with a GPU-built tree: 133k triangles, boxes
// 1.7, transfers 2.3, renumbering 5.5, collapse 3.3, triangle records 4.1 and the search
// 9.7 of 30 ms.
#include <algorithm>
#include <cfloat>
#include <vector>

#include "bvh_build.hpp"
#include "common.hpp"
#include "devpool.hpp"

namespace sbr {
namespace {

constexpr int kMaxBins = 32;
constexpr int kWarpMax = 512;   // nodes up to this many triangles are built by one warp
constexpr int kKeys = 7;        // per bin: lo x/y/z keys, hi x/y/z keys, count
constexpr int kScanBlock = 1024;

// Order-preserving map of floats to unsigned keys (min / max by integer atomics).
__device__ __forceinline__ unsigned fkey(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fval(unsigned k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

struct Level {
    // active nodes of the level
    int32_t* node;          // global node id
    int32_t* s;             // triangle range [s, e)
    int32_t* e;
    unsigned* bounds;       // [12]: box lo keys, box hi keys, centroid lo keys, centroid hi keys
    int32_t* kind;          // 0 leaf, 1 SAH split, 2 median split
    int32_t* axis;
    int32_t* bin;
    int32_t* big_rank;      // -1: built by one warp
    int32_t* left_count;
    int32_t* child_slot;    // first of two slots in the next level
};

struct Work {
    const float* lo;        // [N * 3] triangle boxes
    const float* hi;
    const float* cen;       // [N * 3] centroids
    int32_t* idx;           // [N] position -> triangle
    int32_t* tmp;           // [N]
    int32_t* node_of;       // [N] position -> active slot (-1: in a finished leaf)
    int32_t* flag;          // [N]
    int32_t* scan;          // [N + 1]
    int32_t* block_sums;    // [N / kScanBlock + 2]
    unsigned* big_bins;     // [big nodes][3][B][kKeys]
    int32_t* counters;      // [0] big nodes, [1] next-level nodes, [2] node count
    // node records (breadth first ids)
    float* nlo;             // [2N * 3]
    float* nhi;
    int32_t* nleft;         // child ids, -1 for leaves
    int32_t* nright;
    int32_t* nfirst;
    int32_t* ncount;
    int n, bins, leaf_size, max_leaf;
};

__device__ __forceinline__ int bin_of(float c, float c0, float scl, int B) {
    const int b = __float2int_rz(__fmul_rn(__fsub_rn(c, c0), scl));
    return min(B - 1, max(0, b));
}

// Box area as the host computes it (Box::area, FP64, each operation rounded alone).
__device__ __forceinline__ double area_keys(const unsigned* lo, const unsigned* hi) {
    double d[3];
    for (int a = 0; a < 3; ++a) d[a] = fmax(0.0, __dsub_rn(double(fval(hi[a])), double(fval(lo[a]))));
    return __dmul_rn(2.0, __dadd_rn(__dadd_rn(__dmul_rn(d[0], d[1]), __dmul_rn(d[1], d[2])), __dmul_rn(d[2], d[0])));
}

// The host builder's split decision (Builder::split) from filled bins [3][B][kKeys], by
// one warp: lane b holds bin b, boxes and counts are accumulated from the left and from
// the right by scans (exact minima, maxima and integer sums, whatever their order), every
// lane costs the split after its bin with the host's formula, and the warp keeps the
// cheapest, the first in the host's axis / bin order where several cost the same.  One
// lane doing all of it took 55 us a level of small nodes and 17 us of big ones.
__device__ void sah_decide(const unsigned* bins, int B, const unsigned* bounds, int n, int leaf_size, int max_leaf,
                           int& kind, int& axis, int& bin) {
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    kind = 0;
    axis = -1;
    bin = -1;
    if (n <= leaf_size) return;
    const double inf = __longlong_as_double(0x7ff0000000000000LL);
    const double parent = fmax(area_keys(bounds, bounds + 3), 1e-300);
    double best = inf;
    int bestAx = -1, bestBin = -1;
    for (int ax = 0; ax < 3; ++ax) {
        const float c0 = fval(bounds[6 + ax]), ext = __fsub_rn(fval(bounds[9 + ax]), c0);
        if (!(ext > 0.0f)) continue;
        const unsigned* bx = bins + (ax * B + lane) * kKeys;
        unsigned l[kKeys], r[kKeys];  // lo keys, hi keys, count: of bins 0..lane and lane..B-1
#pragma unroll
        for (int k = 0; k < kKeys; ++k)
            l[k] = r[k] = lane < B ? bx[k] : k < 3 ? fkey(FLT_MAX) : k < 6 ? fkey(-FLT_MAX) : 0u;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
#pragma unroll
            for (int k = 0; k < kKeys; ++k) {
                const unsigned u = __shfl_up_sync(FULL, l[k], off), d = __shfl_down_sync(FULL, r[k], off);
                if (lane >= off) l[k] = k < 3 ? min(l[k], u) : k < 6 ? max(l[k], u) : l[k] + u;
                if (lane + off < 32) r[k] = k < 3 ? min(r[k], d) : k < 6 ? max(r[k], d) : r[k] + d;
            }
        }
        unsigned q[kKeys];  // right of the split after this lane's bin
#pragma unroll
        for (int k = 0; k < kKeys; ++k) q[k] = __shfl_down_sync(FULL, r[k], 1);
        double cost = inf;
        if (lane < B - 1 && l[6] != 0 && q[6] != 0)
            cost = __ddiv_rn(__dadd_rn(__dmul_rn(area_keys(l, l + 3), double(int(l[6]))),
                                       __dmul_rn(area_keys(q, q + 3), double(int(q[6])))), parent);
        if (!(cost < inf)) cost = inf;
        int at = lane;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const double oc = __shfl_xor_sync(FULL, cost, off);
            const int oa = __shfl_xor_sync(FULL, at, off);
            if (oc < cost || (oc == cost && oa < at)) {
                cost = oc;
                at = oa;
            }
        }
        if (cost < best) {
            best = cost;
            bestAx = ax;
            bestBin = at;
        }
    }
    if (bestAx >= 0 && (best < double(n) || n > max_leaf)) {
        kind = 1;
        axis = bestAx;
        bin = bestBin;
    } else if (n > max_leaf) {
        kind = 2;  // all centroids equal: first half of the (index-sorted) range
    }
}

__device__ __forceinline__ void init_bins(unsigned* b, int count, int lane, int stride) {
    for (int i = lane; i < count; i += stride) {
        const int k = i % kKeys;
        b[i] = k < 3 ? fkey(FLT_MAX) : k < 6 ? fkey(-FLT_MAX) : 0u;
    }
}

__global__ void k_init(Work W, Level L) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < W.n) {
        W.idx[p] = p;
        W.node_of[p] = 0;
    }
    if (p == 0) {
        L.node[0] = 0;
        L.s[0] = 0;
        L.e[0] = W.n;
        W.counters[2] = 1;
    }
}

// Per active slot: reset bounds, pick big nodes; `words` words of big-node bins are reset
// alongside (none where no node can be big any more).
__global__ void k_level_begin(Work W, Level L, int nact, int words) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < words) {
        const int k = j % kKeys;
        W.big_bins[j] = k < 3 ? fkey(FLT_MAX) : k < 6 ? fkey(-FLT_MAX) : 0u;
    }
    if (j >= nact) return;
    for (int k = 0; k < 12; ++k) L.bounds[12 * j + k] = (k % 6) < 3 ? fkey(FLT_MAX) : fkey(-FLT_MAX);
    const int n = L.e[j] - L.s[j];
    L.big_rank[j] = n > kWarpMax ? atomicAdd(&W.counters[0], 1) : -1;
}

// Big nodes: bounds by atomics, one warp-level reduction first when a whole warp
// works on one node (contiguous ranges make that the common case).
__global__ void k_big_bounds(Work W, Level L) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = p < W.n ? W.node_of[p] : -1;
    const bool mine = j >= 0 && L.big_rank[j] >= 0;
    const unsigned m = __ballot_sync(0xffffffffu, mine);
    if (!mine) return;
    unsigned v[12];
    const int t = W.idx[p];
    for (int a = 0; a < 3; ++a) {
        v[a] = fkey(W.lo[3 * t + a]);
        v[3 + a] = fkey(W.hi[3 * t + a]);
        v[6 + a] = fkey(W.cen[3 * t + a]);
        v[9 + a] = v[6 + a];
    }
    const int j0 = __shfl_sync(m, j, __ffs(m) - 1);
    const bool uniform = __all_sync(m, j == j0);
    unsigned* B = L.bounds + 12 * j;
    if (uniform) {
        for (int k = 0; k < 12; ++k)
            v[k] = (k % 6) < 3 ? __reduce_min_sync(m, v[k]) : __reduce_max_sync(m, v[k]);
        if ((threadIdx.x & 31) != __ffs(m) - 1) return;
    }
    for (int k = 0; k < 12; ++k) {
        if ((k % 6) < 3) atomicMin(B + k, v[k]);
        else atomicMax(B + k, v[k]);
    }
}

// Big nodes: bins on the three axes (shared-memory bins when the block's positions
// all belong to one node, else global atomics).
__global__ void k_big_bins(Work W, Level L) {
    extern __shared__ unsigned sb[];
    const int B = W.bins;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int p0 = blockIdx.x * blockDim.x, p1 = min(W.n, p0 + (int)blockDim.x) - 1;
    const int jf = W.node_of[p0], jl = W.node_of[p1];
    const bool block_uniform = jf >= 0 && jf == jl && L.big_rank[jf] >= 0;
    if (block_uniform) init_bins(sb, 3 * B * kKeys, threadIdx.x, blockDim.x);
    __syncthreads();
    const int j = p < W.n ? W.node_of[p] : -1;
    if (j >= 0 && L.big_rank[j] >= 0) {
        unsigned* bins = block_uniform ? sb : W.big_bins + (size_t)L.big_rank[j] * 3 * B * kKeys;
        const unsigned* bd = L.bounds + 12 * j;
        const int t = W.idx[p];
        for (int ax = 0; ax < 3; ++ax) {
            const float c0 = fval(bd[6 + ax]), ext = __fsub_rn(fval(bd[9 + ax]), c0);
            if (!(ext > 0.0f)) continue;
            const float scl = __fdiv_rn(float(B), ext);
            unsigned* bb = bins + (ax * B + bin_of(W.cen[3 * t + ax], c0, scl, B)) * kKeys;
            for (int a = 0; a < 3; ++a) {
                atomicMin(bb + a, fkey(W.lo[3 * t + a]));
                atomicMax(bb + 3 + a, fkey(W.hi[3 * t + a]));
            }
            atomicAdd(bb + 6, 1u);
        }
    }
    __syncthreads();
    if (block_uniform) {
        unsigned* g = W.big_bins + (size_t)L.big_rank[jf] * 3 * B * kKeys;
        for (int i = threadIdx.x; i < 3 * B * kKeys; i += blockDim.x) {
            const int k = i % kKeys;
            if (k < 3) atomicMin(g + i, sb[i]);
            else if (k < 6) atomicMax(g + i, sb[i]);
            else if (sb[i]) atomicAdd(g + i, sb[i]);
        }
    }
}

// Big nodes: the split decision, a warp each.
__global__ void k_big_split(Work W, Level L, int nact) {
    const int j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (j >= nact || L.big_rank[j] < 0) return;
    int kind, ax, bin;
    sah_decide(W.big_bins + (size_t)L.big_rank[j] * 3 * W.bins * kKeys, W.bins, L.bounds + 12 * j, L.e[j] - L.s[j],
               W.leaf_size, W.max_leaf, kind, ax, bin);
    if ((threadIdx.x & 31) != 0) return;
    L.kind[j] = kind;
    L.axis[j] = ax;
    L.bin[j] = bin;
}

// Small nodes: one warp each -- bounds, bins in shared memory, split decision.
__global__ void k_small(Work W, Level L, int nact) {
    extern __shared__ unsigned sb[];
    const int B = W.bins;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j = blockIdx.x * (blockDim.x >> 5) + warp;
    if (j >= nact || L.big_rank[j] >= 0) return;
    unsigned* bins = sb + warp * 3 * B * kKeys;
    const int s = L.s[j], e = L.e[j], n = e - s;
    unsigned v[12];
    for (int k = 0; k < 12; ++k) v[k] = (k % 6) < 3 ? fkey(FLT_MAX) : fkey(-FLT_MAX);
    for (int p = s + lane; p < e; p += 32) {
        const int t = W.idx[p];
        for (int a = 0; a < 3; ++a) {
            v[a] = min(v[a], fkey(W.lo[3 * t + a]));
            v[3 + a] = max(v[3 + a], fkey(W.hi[3 * t + a]));
            const unsigned c = fkey(W.cen[3 * t + a]);
            v[6 + a] = min(v[6 + a], c);
            v[9 + a] = max(v[9 + a], c);
        }
    }
    for (int k = 0; k < 12; ++k)
        v[k] = (k % 6) < 3 ? __reduce_min_sync(0xffffffffu, v[k]) : __reduce_max_sync(0xffffffffu, v[k]);
    if (lane < 12) L.bounds[12 * j + lane] = v[lane];
    if (n <= W.leaf_size) {
        if (lane == 0) L.kind[j] = 0;
        return;
    }
    init_bins(bins, 3 * B * kKeys, lane, 32);
    __syncwarp();
    for (int p = s + lane; p < e; p += 32) {
        const int t = W.idx[p];
        for (int ax = 0; ax < 3; ++ax) {
            const float c0 = fval(v[6 + ax]), ext = __fsub_rn(fval(v[9 + ax]), c0);
            if (!(ext > 0.0f)) continue;
            const float scl = __fdiv_rn(float(B), ext);
            unsigned* bb = bins + (ax * B + bin_of(W.cen[3 * t + ax], c0, scl, B)) * kKeys;
            for (int a = 0; a < 3; ++a) {
                atomicMin(bb + a, fkey(W.lo[3 * t + a]));
                atomicMax(bb + 3 + a, fkey(W.hi[3 * t + a]));
            }
            atomicAdd(bb + 6, 1u);
        }
    }
    __syncwarp();
    int kind, ax, bin;
    sah_decide(bins, B, v, n, W.leaf_size, W.max_leaf, kind, ax, bin);
    if (lane == 0) {
        L.kind[j] = kind;
        L.axis[j] = ax;
        L.bin[j] = bin;
    }
}

__global__ void k_flags(Work W, Level L) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= W.n) return;
    const int j = W.node_of[p];
    int f = 0;
    if (j >= 0) {
        const int kind = L.kind[j];
        if (kind == 1) {
            const int ax = L.axis[j];
            const unsigned* bd = L.bounds + 12 * j;
            const float c0 = fval(bd[6 + ax]), ext = __fsub_rn(fval(bd[9 + ax]), c0);
            const float scl = __fdiv_rn(float(W.bins), ext);
            f = bin_of(W.cen[3 * W.idx[p] + ax], c0, scl, W.bins) <= L.bin[j];
        } else if (kind == 2) {
            const int s = L.s[j], n = L.e[j] - s;
            f = (p - s) < n / 2;
        }
    }
    W.flag[p] = f;
}

// Exclusive scan of W.flag into W.scan[0..n] (three passes).
__global__ void k_scan_blocks(const int32_t* in, int32_t* out, int32_t* sums, int n) {
    __shared__ int32_t sh[kScanBlock];
    const int p = blockIdx.x * kScanBlock + threadIdx.x;
    const int x = p < n ? in[p] : 0;
    sh[threadIdx.x] = x;
    __syncthreads();
    for (int off = 1; off < kScanBlock; off <<= 1) {
        const int y = threadIdx.x >= off ? sh[threadIdx.x - off] : 0;
        __syncthreads();
        sh[threadIdx.x] += y;
        __syncthreads();
    }
    if (p < n) out[p] = sh[threadIdx.x] - x;
    if (threadIdx.x == kScanBlock - 1) sums[blockIdx.x] = sh[threadIdx.x];
}
__global__ void k_scan_sums(int32_t* sums, int nb) {
    __shared__ int32_t carry;
    __shared__ int32_t sh[kScanBlock];
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < nb; base += kScanBlock) {
        const int i = base + threadIdx.x;
        const int x = i < nb ? sums[i] : 0;
        sh[threadIdx.x] = x;
        __syncthreads();
        for (int off = 1; off < kScanBlock; off <<= 1) {
            const int y = threadIdx.x >= off ? sh[threadIdx.x - off] : 0;
            __syncthreads();
            sh[threadIdx.x] += y;
            __syncthreads();
        }
        if (i < nb) sums[i] = carry + sh[threadIdx.x] - x;
        __syncthreads();
        if (threadIdx.x == kScanBlock - 1) carry += sh[threadIdx.x];
        __syncthreads();
    }
    if (threadIdx.x == 0) sums[nb] = carry;
}
__global__ void k_scan_add(int32_t* out, const int32_t* sums, int n, int nblk) {
    const int p = blockIdx.x * kScanBlock + threadIdx.x;
    if (p < n) out[p] += sums[blockIdx.x];
    if (p == n) out[n] = sums[nblk];  // the total
}

// Stable partition of every split node's range; other positions copy through.
__global__ void k_scatter(Work W, Level L) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= W.n) return;
    const int j = W.node_of[p];
    if (j < 0 || L.kind[j] == 0) {
        W.tmp[p] = W.idx[p];
        return;
    }
    const int s = L.s[j], e = L.e[j];
    const int base = W.scan[s];
    const int nl = W.scan[e] - base;
    const int lr = W.scan[p] - base;
    const int q = W.flag[p] ? s + lr : s + nl + (p - s - lr);
    W.tmp[q] = W.idx[p];
    if (p == s) L.left_count[j] = nl;
}

// Node records and the next level's active slots.
__global__ void k_emit(Work W, Level L, Level N, int nact, int cap) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nact) return;
    const int id = L.node[j];
    const unsigned* bd = L.bounds + 12 * j;
    for (int a = 0; a < 3; ++a) {
        W.nlo[3 * id + a] = fval(bd[a]);
        W.nhi[3 * id + a] = fval(bd[3 + a]);
    }
    const int s = L.s[j], e = L.e[j];
    if (L.kind[j] == 0) {
        W.nleft[id] = W.nright[id] = -1;
        W.nfirst[id] = s;
        W.ncount[id] = e - s;
        L.child_slot[j] = -1;
        return;
    }
    const int m = s + L.left_count[j];
    const int c = atomicAdd(&W.counters[1], 2);
    const int cid = atomicAdd(&W.counters[2], 2);
    if (c + 1 >= cap || cid + 1 >= 2 * W.n) {  // bounded by construction; never write past the arrays
        atomicOr(&W.counters[3], 1);
        L.child_slot[j] = -1;
        return;
    }
    W.nleft[id] = cid;
    W.nright[id] = cid + 1;
    W.nfirst[id] = 0;
    W.ncount[id] = 0;
    N.node[c] = cid;
    N.s[c] = s;
    N.e[c] = m;
    N.node[c + 1] = cid + 1;
    N.s[c + 1] = m;
    N.e[c + 1] = e;
    L.child_slot[j] = c;
}

__global__ void k_assign(Work W, Level L) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= W.n) return;
    const int j = W.node_of[p];
    if (j < 0) return;
    const int c = L.child_slot[j];
    W.node_of[p] = c < 0 ? -1 : (p < L.s[j] + L.left_count[j] ? c : c + 1);
}

// Conservative boxes of the triangles (covering the FP32 and the outward-rounded FP64
// vertices) and their centroids, in the host build's arithmetic.
__global__ void k_boxes(const float* __restrict__ xyz, const uint32_t* __restrict__ idx, int n, float sc32, double sc,
                        float* __restrict__ lo, float* __restrict__ hi, float* __restrict__ cen) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    float l[3] = {INFINITY, INFINITY, INFINITY}, h[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int c = 0; c < 3; ++c) {
        const size_t v = idx[3 * (size_t)t + c];
        for (int a = 0; a < 3; ++a) {
            const float x = xyz[3 * v + a], p = __fmul_rn(x, sc32);
            const double q = __dmul_rn(double(x), sc);
            l[a] = fminf(l[a], fminf(p, __double2float_rd(q)));
            h[a] = fmaxf(h[a], fmaxf(p, __double2float_ru(q)));
        }
    }
    for (int a = 0; a < 3; ++a) {
        lo[3 * (size_t)t + a] = l[a];
        hi[3 * (size_t)t + a] = h[a];
        cen[3 * (size_t)t + a] = __fmul_rn(0.5f, __fadd_rn(l[a], h[a]));
    }
}

// ------------------------------------------------------------------ collapse
// Work arrays of the collapse, by breadth-first number of the 4-wide node.
struct Collapse {
    int32_t* bin;      // binary node it stands for
    int32_t* need;     // stack entries a walker may hold on arrival
    int4* kids;        // binary nodes of its children, -1 for none
    int32_t* child;    // number of its first inner child
    int32_t* size;     // 4-wide nodes of its subtree
    int32_t* pre;      // 4-wide nodes allotted before it in depth-first order
    int32_t* slot;     // its final number
    int32_t* off;      // [levels + 2] first number of each level
    int32_t* tail;     // nodes so far
};
struct BinView {
    const float* lo;
    const float* hi;
    const int32_t* left;
    const int32_t* right;
    const int32_t* first;
    const int32_t* count;
};

__device__ __forceinline__ float box_area(const BinView& B, int b) {
    const float x = __fsub_rn(B.hi[3 * b], B.lo[3 * b]), y = __fsub_rn(B.hi[3 * b + 1], B.lo[3 * b + 1]),
                z = __fsub_rn(B.hi[3 * b + 2], B.lo[3 * b + 2]);
    return __fadd_rn(__fadd_rn(__fmul_rn(x, y), __fmul_rn(y, z)), __fmul_rn(z, x));
}

__global__ void k_collapse_root(Collapse C) {
    C.bin[0] = 0;
    C.need[0] = 0;
    C.off[0] = 0;
    C.off[1] = 1;
    *C.tail = 1;
}
// A 4-wide node takes a binary node's two children and keeps opening its largest (by
// surface area) inner child until it holds four or the walker's stack bound is reached.
__global__ void k_collapse_open(BinView B, Collapse C, int level, int stack_depth) {
    for (int i = C.off[level] + blockIdx.x * blockDim.x + threadIdx.x; i < C.off[level + 1]; i += gridDim.x * blockDim.x) {
        const int b = C.bin[i], need = C.need[i];
        int kid[4] = {b, -1, -1, -1};
        int nk = 1;
        if (B.left[b] >= 0) {
            kid[0] = B.left[b];
            kid[1] = B.right[b];
            nk = 2;
            while (nk < 4 && need + nk <= stack_depth) {
                int best = -1;
                float ba = -1.0f;
                for (int k = 0; k < nk; ++k) {
                    if (B.left[kid[k]] < 0) continue;
                    const float a = box_area(B, kid[k]);
                    if (a > ba) {
                        ba = a;
                        best = k;
                    }
                }
                if (best < 0) break;
                const int open = kid[best];
                for (int k = nk; k > best + 1; --k) kid[k] = kid[k - 1];
                kid[best] = B.left[open];
                kid[best + 1] = B.right[open];
                ++nk;
            }
        }
        int ni = 0;
        for (int k = 0; k < nk; ++k) ni += kid[k] != b && B.left[kid[k]] >= 0;
        int at = ni ? atomicAdd(C.tail, ni) : 0;
        C.kids[i] = make_int4(kid[0], kid[1], kid[2], kid[3]);
        C.child[i] = at;
        for (int k = 0; k < nk; ++k) {
            if (kid[k] == b || B.left[kid[k]] < 0) continue;
            C.bin[at] = kid[k];
            C.need[at] = need + nk - 1;
            ++at;
        }
    }
}
__global__ void k_collapse_level(Collapse C, int level) { C.off[level + 2] = *C.tail; }

__device__ __forceinline__ bool is_inner(const BinView& B, const Collapse& C, int i, int kid) {
    return kid >= 0 && kid != C.bin[i] && B.left[kid] >= 0;
}
__global__ void k_collapse_size(BinView B, Collapse C, int level) {
    for (int i = C.off[level] + blockIdx.x * blockDim.x + threadIdx.x; i < C.off[level + 1]; i += gridDim.x * blockDim.x) {
        const int4 q = C.kids[i];
        const int kid[4] = {q.x, q.y, q.z, q.w};
        int at = C.child[i], n = 1;
        for (int k = 0; k < 4; ++k)
            if (is_inner(B, C, i, kid[k])) n += C.size[at++];
        C.size[i] = n;
    }
}
// Numbers a node's inner children next to one another after all nodes that come before
// it depth first, and writes the node.
__global__ void k_collapse_emit(BinView B, Collapse C, int level, GNode4* nodes, int32_t* level_nodes) {
    for (int i = C.off[level] + blockIdx.x * blockDim.x + threadIdx.x; i < C.off[level + 1]; i += gridDim.x * blockDim.x) {
        const int pre = level == 0 ? 0 : C.pre[i], slot = level == 0 ? 0 : C.slot[i];
        const int4 q = C.kids[i];
        const int kid[4] = {q.x, q.y, q.z, q.w};
        GNode4 N;
        int ni = 0;
        for (int k = 0; k < 4; ++k) ni += is_inner(B, C, i, kid[k]);
        int at = C.child[i], num = 1 + pre, before = pre + ni;
        for (int k = 0; k < 4; ++k) {
            float lo[3] = {1e30f, 1e30f, 1e30f}, hi[3] = {1e30f, 1e30f, 1e30f};  // an empty slot's far box
            int ref = ~0;
            if (kid[k] >= 0) {
                for (int a = 0; a < 3; ++a) {
                    lo[a] = B.lo[3 * kid[k] + a];
                    hi[a] = B.hi[3 * kid[k] + a];
                }
                if (is_inner(B, C, i, kid[k])) {
                    ref = num;
                    C.slot[at] = num++;
                    C.pre[at] = before;
                    before += C.size[at] - 1;
                    ++at;
                } else {
                    ref = ~(B.first[kid[k]] * 16 + B.count[kid[k]]);
                }
            }
            (&N.lox.x)[k] = lo[0]; (&N.hix.x)[k] = hi[0];
            (&N.loy.x)[k] = lo[1]; (&N.hiy.x)[k] = hi[1];
            (&N.loz.x)[k] = lo[2]; (&N.hiz.x)[k] = hi[2];
            (&N.child.x)[k] = ref;
        }
        nodes[slot] = N;
        level_nodes[i] = slot;
    }
}

// ------------------------------------------------------------------ twins
// A triangle's three vertices in the order of their bits, and the parity of that order
// (-1: a repeated vertex), as has_opposed_twins compares them.
struct TwinKey {
    uint32_t v[9];
    int parity;
};
__device__ TwinKey twin_key(const float* xyz, const uint32_t* idx, size_t t) {
    uint32_t p[3][3];
    for (int c = 0; c < 3; ++c)
        for (int a = 0; a < 3; ++a) p[c][a] = __float_as_uint(xyz[3 * (size_t)idx[3 * t + c] + a]);
    int swaps = 0;
    auto order = [&](int a, int b) {  // p[a] before p[b]
        const bool less = p[b][0] != p[a][0] ? p[b][0] < p[a][0] : p[b][1] != p[a][1] ? p[b][1] < p[a][1] : p[b][2] < p[a][2];
        if (!less) return;
        ++swaps;
        for (int k = 0; k < 3; ++k) {
            const uint32_t x = p[a][k];
            p[a][k] = p[b][k];
            p[b][k] = x;
        }
    };
    order(0, 1);
    order(1, 2);
    order(0, 1);
    TwinKey key;
    bool r01 = true, r12 = true;
    for (int k = 0; k < 3; ++k) {
        key.v[k] = p[0][k];
        key.v[3 + k] = p[1][k];
        key.v[6 + k] = p[2][k];
        r01 = r01 && p[0][k] == p[1][k];
        r12 = r12 && p[1][k] == p[2][k];
    }
    key.parity = r01 || r12 ? -1 : swaps & 1;
    return key;
}
// Open addressing: every distinct key keeps the first triangle that came with it; a later
// one of the other parity is a twin.
__global__ void k_twins(const float* __restrict__ xyz, const uint32_t* __restrict__ idx, int n, int32_t* table,
                        uint32_t mask, int32_t* flag) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const TwinKey key = twin_key(xyz, idx, t);
    if (key.parity < 0) return;
    uint32_t h = 2166136261u;
    for (int k = 0; k < 9; ++k) h = (h ^ key.v[k]) * 16777619u;
    h ^= h >> 15;
    h *= 0x2c1b3c6du;
    h ^= h >> 12;
    for (uint32_t probe = 0; probe <= mask; ++probe) {
        const int other = atomicCAS(table + ((h + probe) & mask), -1, t);
        if (other == -1) return;
        const TwinKey o = twin_key(xyz, idx, other);
        bool same = true;
        for (int k = 0; k < 9; ++k) same = same && o.v[k] == key.v[k];
        if (same) {
            if (o.parity != key.parity) *flag = 1;
            return;
        }
    }
}

}  // namespace

size_t gpu_twins_table(size_t n) {
    size_t m = 64;
    while (m < 2 * n) m *= 2;
    return m;
}

cudaError_t gpu_opposed_twins(const float* d_xyz, const uint32_t* d_idx, size_t n, int32_t* table, int32_t* d_flag,
                              cudaStream_t stream) {
    const size_t m = gpu_twins_table(n);
    cudaError_t e = cudaMemsetAsync(table, 0xff, m * sizeof(int32_t), stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_flag, 0, sizeof(int32_t), stream);
    if (e != cudaSuccess) return e;
    k_twins<<<(unsigned)((n + 127) / 128), 128, 0, stream>>>(d_xyz, d_idx, (int)n, table, (uint32_t)(m - 1), d_flag);
    return cudaGetLastError();
}

void gpu_tree_free(GpuTree& t, cudaStream_t stream) {
    if (!t.block) return;
    if (cudaStreamSynchronize(stream) != cudaSuccess) cudaDeviceSynchronize();
    pool_free(t.device, t.block);
    pool_free(t.device, t.level_off);
    t.block = nullptr;
    t.level_off = nullptr;
}

cudaError_t gpu_tree_build(const float* d_xyz, const uint32_t* d_idx, int n, double scale, const BuildOptions& opt,
                           cudaStream_t stream, GpuTree& out) {
    out = GpuTree();
    out.n = n;
    const int B = std::min(std::max(2, opt.bin_count), kMaxBins);
    const int cap = std::min(n, 2 * (n / (opt.leaf_size + 1)) + 2);
    const int nblk = (n + kScanBlock - 1) / kScanBlock;

    Work W{};
    Level L[2]{};
    // all work arrays in one block: their sizes first, then their addresses
    Parts parts;
    std::vector<std::pair<void**, size_t>> owned;
    auto A = [&](auto** p, size_t count) {
        owned.emplace_back(reinterpret_cast<void**>(p), parts.add(sizeof(**p) * count));
    };
    float *lo, *hi, *ce;
    A(&lo, 3 * (size_t)n);
    A(&hi, 3 * (size_t)n);
    A(&ce, 3 * (size_t)n);
    A(&W.idx, n);
    A(&W.tmp, n);
    A(&W.node_of, n);
    A(&W.flag, n);
    A(&W.scan, (size_t)n + 1);
    A(&W.block_sums, (size_t)nblk + 2);
    A(&W.big_bins, (size_t)(n / kWarpMax + 2) * 3 * B * kKeys);
    A(&W.counters, 4);
    A(&W.nlo, 3 * (size_t)(2 * n));
    A(&W.nhi, 3 * (size_t)(2 * n));
    A(&W.nleft, 2 * (size_t)n);
    A(&W.nright, 2 * (size_t)n);
    A(&W.nfirst, 2 * (size_t)n);
    A(&W.ncount, 2 * (size_t)n);
    for (Level& l : L) {
        A(&l.node, cap);
        A(&l.s, cap);
        A(&l.e, cap);
        A(&l.bounds, 12 * (size_t)cap);
        A(&l.kind, cap);
        A(&l.axis, cap);
        A(&l.bin, cap);
        A(&l.big_rank, cap);
        A(&l.left_count, cap);
        A(&l.child_slot, cap);
    }
    // the collapse's work: a binary tree of n leaves at most has n - 1 inner nodes
    A(&out.work, 10 * (size_t)n);
    cudaError_t e = cudaGetDevice(&out.device);
    if (e == cudaSuccess) e = pool_alloc(out.device, &out.block, parts.size());
    if (e != cudaSuccess) return e;
    for (auto& o : owned) *o.first = out.block + o.second;
    W.lo = lo;
    W.hi = hi;
    W.cen = ce;
    W.n = n;
    W.bins = B;
    W.leaf_size = opt.leaf_size;
    W.max_leaf = opt.max_leaf;
    e = cudaMemsetAsync(W.counters, 0, 4 * sizeof(int32_t), stream);
    const int TB = 256;
    const int gp = (n + TB - 1) / TB;
    k_boxes<<<gp, TB, 0, stream>>>(d_xyz, d_idx, n, float(scale), scale, lo, hi, ce);
    k_init<<<gp, TB, 0, stream>>>(W, L[0]);
    const size_t bin_bytes = (size_t)3 * B * kKeys * sizeof(unsigned);
    int nact = 1, cur = 0;
    bool big = n > kWarpMax;
    while (nact > 0 && e == cudaSuccess) {
        Level& C = L[cur];
        Level& X = L[cur ^ 1];
        cudaMemsetAsync(W.counters, 0, 2 * sizeof(int32_t), stream);
        // big nodes only come from big nodes
        const int words = big ? (int)((size_t)(n / kWarpMax + 2) * 3 * B * kKeys) : 0;
        k_level_begin<<<(std::max(nact, words) + TB - 1) / TB, TB, 0, stream>>>(W, C, nact, words);
        if (big) {
            k_big_bounds<<<gp, TB, 0, stream>>>(W, C);
            k_big_bins<<<gp, TB, bin_bytes, stream>>>(W, C);
            k_big_split<<<(nact + 7) / 8, 256, 0, stream>>>(W, C, nact);
        }
        k_small<<<(nact + 7) / 8, 256, 8 * bin_bytes, stream>>>(W, C, nact);
        k_flags<<<gp, TB, 0, stream>>>(W, C);
        k_scan_blocks<<<nblk, kScanBlock, 0, stream>>>(W.flag, W.scan, W.block_sums, n);
        k_scan_sums<<<1, kScanBlock, 0, stream>>>(W.block_sums, nblk);
        k_scan_add<<<(n + 1 + kScanBlock - 1) / kScanBlock, kScanBlock, 0, stream>>>(W.scan, W.block_sums, n, nblk);
        k_scatter<<<gp, TB, 0, stream>>>(W, C);
        std::swap(W.idx, W.tmp);
        k_emit<<<(nact + TB - 1) / TB, TB, 0, stream>>>(W, C, X, nact, cap);
        k_assign<<<gp, TB, 0, stream>>>(W, C);
        int32_t cnt[4] = {0, 0, 0, 0};
        e = cudaMemcpyAsync(cnt, W.counters, sizeof(cnt), cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        if (e == cudaSuccess) e = cudaGetLastError();
        // cannot happen: each split node has more than leaf_size triangles
        if (e == cudaSuccess && (cnt[3] != 0 || cnt[1] > cap)) e = cudaErrorInvalidValue;
        big = cnt[0] > 0;
        nact = cnt[1];
        out.nnodes = cnt[2];
        ++out.levels;
        cur ^= 1;
    }
    if (e != cudaSuccess) {
        gpu_tree_free(out, stream);
        return e;
    }
    out.lo = W.nlo;
    out.hi = W.nhi;
    out.left = W.nleft;
    out.right = W.nright;
    out.first = W.nfirst;
    out.count = W.ncount;
    out.order = W.idx;
    return cudaSuccess;
}

namespace {

// The collapse's arrays in the tree's block: `work` is 10 words per triangle and a tree
// has fewer inner nodes (4-wide nodes) than triangles, but at least one node.
Collapse collapse_view(const GpuTree& t) {
    const size_t m = std::max(1, t.n);
    Collapse C;
    C.kids = reinterpret_cast<int4*>(t.work);
    C.bin = t.work + 4 * m;
    C.need = t.work + 5 * m;
    C.child = t.work + 6 * m;
    C.size = t.work + 7 * m;
    C.pre = t.work + 8 * m;
    C.slot = t.work + 9 * m;
    C.off = t.level_off;
    C.tail = t.level_off + t.levels + 2;
    return C;
}
BinView bin_view(const GpuTree& t) { return {t.lo, t.hi, t.left, t.right, t.first, t.count}; }
constexpr int kCollapseGrid = 592;  // 4 blocks of 128 per SM, striding over a level

}  // namespace

cudaError_t gpu_tree_collapse(GpuTree& t, int stack_depth, cudaStream_t stream) {
    cudaError_t e = pool_alloc(t.device, &t.level_off, (size_t)(t.levels + 3) * sizeof(int32_t));
    if (e != cudaSuccess) return e;
    const Collapse C = collapse_view(t);
    k_collapse_root<<<1, 1, 0, stream>>>(C);
    for (int l = 0; l < t.levels; ++l) {
        k_collapse_open<<<kCollapseGrid, 128, 0, stream>>>(bin_view(t), C, l, stack_depth);
        k_collapse_level<<<1, 1, 0, stream>>>(C, l);
    }
    for (int l = t.levels - 1; l >= 0; --l) k_collapse_size<<<kCollapseGrid, 128, 0, stream>>>(bin_view(t), C, l);
    e = cudaMemcpyAsync(&t.ncollapsed, C.tail, sizeof(int32_t), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e == cudaSuccess) e = cudaGetLastError();
    return e;
}

cudaError_t gpu_tree_emit(const GpuTree& t, void* d_nodes, int32_t* d_level_nodes, std::vector<int32_t>& level_off,
                          cudaStream_t stream) {
    const Collapse C = collapse_view(t);
    for (int l = 0; l < t.levels; ++l)
        k_collapse_emit<<<kCollapseGrid, 128, 0, stream>>>(bin_view(t), C, l, static_cast<GNode4*>(d_nodes), d_level_nodes);
    level_off.resize((size_t)t.levels + 2);
    cudaError_t e = cudaMemcpyAsync(level_off.data(), t.level_off, level_off.size() * sizeof(int32_t),
                                    cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e == cudaSuccess) e = cudaGetLastError();
    // levels below the collapsed tree's depth are empty
    while (level_off.size() > 2 && level_off[level_off.size() - 2] == level_off.back()) level_off.pop_back();
    return e;
}

cudaError_t gpu_tree_download(const GpuTree& t, cudaStream_t stream, BinTree& out) {
    out = BinTree();
    const size_t m = (size_t)t.nnodes;
    std::vector<float> nlo(3 * m), nhi(3 * m);
    std::vector<int32_t> nl(m), nr(m), nf(m), nc(m), order((size_t)t.n);
    cudaError_t e = cudaStreamSynchronize(stream);
    auto get = [&](void* dst, const void* src, size_t bytes) {
        if (e == cudaSuccess) e = cudaMemcpy(dst, src, bytes, cudaMemcpyDeviceToHost);
    };
    get(nlo.data(), t.lo, 12 * m);
    get(nhi.data(), t.hi, 12 * m);
    get(nl.data(), t.left, 4 * m);
    get(nr.data(), t.right, 4 * m);
    get(nf.data(), t.first, 4 * m);
    get(nc.data(), t.count, 4 * m);
    get(order.data(), t.order, 4 * (size_t)t.n);
    if (e != cudaSuccess) return e;
    // pre-order renumbering (left subtree before right), as the host builder's flatten
    out.nodes.reserve(m);
    struct Item {
        int32_t id, parent, depth;
        bool right;
    };
    std::vector<Item> stack{{0, -1, 0, false}};
    while (!stack.empty()) {
        const Item it = stack.back();
        stack.pop_back();
        const int me = (int)out.nodes.size();
        BinNode b;
        for (int a = 0; a < 3; ++a) {
            b.lo[a] = nlo[3 * (size_t)it.id + a];
            b.hi[a] = nhi[3 * (size_t)it.id + a];
        }
        b.left = b.right = -1;
        b.first = nl[it.id] < 0 ? nf[it.id] : 0;
        b.count = nl[it.id] < 0 ? nc[it.id] : 0;
        out.nodes.push_back(b);
        out.depth = std::max(out.depth, it.depth + 1);
        if (it.parent >= 0) {
            if (it.right) out.nodes[it.parent].right = me;
            else out.nodes[it.parent].left = me;
        }
        if (nl[it.id] >= 0) {
            stack.push_back({nr[it.id], me, it.depth + 1, true});
            stack.push_back({nl[it.id], me, it.depth + 1, false});
        }
    }
    out.order = std::move(order);
    return cudaSuccess;
}

}  // namespace sbr
