// Device build of the reference's binary BVH topology (BVH::build_node /
// compute_split, src/primitive/bvh.h:57-216), bit-identical to the host
// restatement build_ref_topology (bvh.cpp) and so to the reference.
//
// Level-synchronous: every node of one tree level is a segment [start,
// start + count) of the primitive array, processed by one CTA of 128
// threads (nodes of more than kBigSeg primitives by several, k_big_*; nodes of
// at most 32 by a warp, level_warp), which
//   1. reduces the node's bounds and centroid bounds,
//   2. bins the centroids into 5 equal-width bins per axis (a primitive
//      joins the first bin j with c < min + (max - min) * (j + 1) / 5) and
//      reduces each bin's count and box,
//   3. evaluates the 4 splits per axis (area(L) + area(R), +inf when a side
//      is empty; first strict minimum; the reference's nested axis choice),
//   4. writes its primitives into the other buffer in the bins'
//      concatenation order (bin 0's primitives, then bin 1's, ..., each bin
//      in input order), and emits the node and its two child segments (bins
//      0..split and the rest) for the next level.
// A segment of fewer than 4 primitives is a leaf (bvh.h:152-158).  Where the
// chosen split leaves one side empty the reference recurses without end
// (bvh.h:200); like the host build, one leaf then holds them all.
//
// The reference unites boxes in the primitives' order with
// min(a, b) = a < b ? a : b (and max likewise), so among equal values the
// later primitive's value is kept (this matters for -0.0 against +0.0).
// Each min / max is therefore a reduction of a 64-bit key -- the value
// mapped to an ordered integer with -0.0 and +0.0 equal, then the position
// (ties to the later one) -- and the winner's own float is read back.
// All float arithmetic is unfused (__fadd_rn / __fmul_rn) in the
// reference's order.
//
// Nodes are created level by level in no particular order; the pre-order
// numbering of the reference (parent, then the first partition's subtree,
// then the second's) follows from the subtree sizes, computed bottom-up.
#include <cuda_runtime.h>

#include <cstring>
#include <stdexcept>
#include <string>
#include <vector>

#include "gpu_bvh.h"

namespace cpppt_gb300 {

namespace {

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int kBins = 5;
constexpr int kBigSeg = 2048;     // nodes above this size are split by several CTAs
constexpr int kBigChunk = 2048;   // primitives per CTA there
constexpr int kBigThreads = 256;

struct PrimG {
    float lo[3], hi[3], c[3];
    int32_t id;
};

struct SegG {
    int32_t start, count, parent, side;  // parent: node id (-1: none); side 0 = first partition
};

struct NodeG {
    float lo[3], hi[3];
    int32_t parent, side;
    int32_t child[2];  // node ids, -1 for a leaf child
};

__device__ __forceinline__ uint32_t okey(float v) {
    if (v == 0.0f) v = 0.0f;  // -0.0 and +0.0 compare equal
    const uint32_t u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
// smallest value, then the later position
__device__ __forceinline__ unsigned long long kmin(float v, uint32_t pos) {
    return ((unsigned long long)okey(v) << 32) | (unsigned long long)(0xffffffffu - pos);
}
// largest value, then the later position
__device__ __forceinline__ unsigned long long kmax(float v, uint32_t pos) {
    return ((unsigned long long)okey(v) << 32) | (unsigned long long)pos;
}
__device__ __forceinline__ uint32_t kpos_min(unsigned long long k) { return 0xffffffffu - (uint32_t)(k & 0xffffffffu); }
__device__ __forceinline__ uint32_t kpos_max(unsigned long long k) { return (uint32_t)(k & 0xffffffffu); }

__device__ __forceinline__ unsigned long long warp_min64(unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
        v = w < v ? w : v;
    }
    return v;
}
__device__ __forceinline__ unsigned long long warp_max64(unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
        v = w > v ? w : v;
    }
    return v;
}

// AABB::area (aabb.h:77-82): 2.0 * (|dx| dy + |dz| dy + |dx| dz), the sum in
// float, doubled in double
__device__ __forceinline__ float ref_area(const float* lo, const float* hi) {
    const float dx = fabsf(__fsub_rn(hi[0], lo[0])), dy = __fsub_rn(hi[1], lo[1]);
    const float dz = fabsf(__fsub_rn(hi[2], lo[2])), dzy = __fsub_rn(hi[2], lo[2]);
    float s = __fmul_rn(dx, dy);
    s = __fadd_rn(s, __fmul_rn(dz, dy));
    s = __fadd_rn(s, __fmul_rn(dx, dzy));
    return (float)(2.0 * (double)s);
}

// a < b ? a : b and a > b ? a : b (the later operand kept on ties)
__device__ __forceinline__ float vmin1(float a, float b) { return a < b ? a : b; }
__device__ __forceinline__ float vmax1(float a, float b) { return a > b ? a : b; }

__device__ __forceinline__ int bin_of(float c, const float* thr) {
    int b = kBins - 1;
#pragma unroll
    for (int j = kBins - 2; j >= 0; j--)
        if (c < thr[j]) b = j;
    return b;
}

// Per-primitive records: Triangle::get_bounds (triangle.h:197-207) and
// AABB::center ((min + max) * 0.5, aabb.h:62-64).
__global__ void k_prims(const float* __restrict__ tv, int n, PrimG* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* v = tv + 9 * (size_t)i;
    PrimG p;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        p.lo[k] = vmin1(vmin1(v[k], v[3 + k]), v[6 + k]);
        p.hi[k] = vmax1(vmax1(v[k], v[3 + k]), v[6 + k]);
        p.c[k] = __fmul_rn(__fadd_rn(p.lo[k], p.hi[k]), 0.5f);
    }
    p.id = i;
    out[i] = p;
}

// A node of more than kBigSeg primitives: its segment, its chunks, and what the
// chunks accumulate -- bounds and centroid bounds, then each bin's box (keys)
// and count.
struct BigG {
    SegG seg;
    int32_t first, chunks;  // in the level's chunk list
    unsigned long long red[12];
    unsigned long long bin[3][kBins][6];
    int32_t cnt[3][kBins];
    int32_t axis, leaf;
};
struct ChunkG {
    int32_t big, index;  // kBigChunk primitives from index * kBigChunk on
};

// The next level's segments, those of at most 32 primitives in a list of
// their own, and its large nodes with their chunks.
// counts: [0] segments, [1] nodes, [2] large nodes, [3] chunks, [4] small segments
struct LevelOut {
    SegG* segs;
    SegG* small;
    BigG* big;
    ChunkG* chunks;
    int* counts;
};

__device__ __forceinline__ bool comp_is_min(int comp) { return comp < 3; }

__device__ void emit_seg(const LevelOut& L, const SegG& c) {
    if (c.count <= 32) {
        L.small[atomicAdd(L.counts + 4, 1)] = c;
        return;
    }
    L.segs[atomicAdd(L.counts, 1)] = c;
    if (c.count <= kBigSeg) return;
    const int bi = atomicAdd(L.counts + 2, 1), n = (c.count + kBigChunk - 1) / kBigChunk;
    BigG& B = L.big[bi];
    B.seg = c;
    B.first = atomicAdd(L.counts + 3, n);
    B.chunks = n;
    for (int j = 0; j < 12; j++) B.red[j] = (j % 6) < 3 ? ~0ull : 0ull;
    for (int j = 0; j < 3 * kBins * 6; j++) (&B.bin[0][0][0])[j] = comp_is_min(j % 6) ? ~0ull : 0ull;
    for (int j = 0; j < 3 * kBins; j++) (&B.cnt[0][0])[j] = 0;
    for (int j = 0; j < n; j++) L.chunks[B.first + j] = ChunkG{bi, j};
}

__global__ void k_root(LevelOut L, int n) { emit_seg(L, SegG{0, n, -1, 0}); }

// The 12 bounds keys of P[begin, end), reduced over a warp.
__device__ __forceinline__ void bounds_keys(const PrimG* __restrict__ P, int begin, int end, unsigned long long k[12]) {
#pragma unroll
    for (int j = 0; j < 3; j++) { k[j] = ~0ull; k[3 + j] = 0ull; k[6 + j] = ~0ull; k[9 + j] = 0ull; }
    for (int i = begin + (int)threadIdx.x; i < end; i += blockDim.x) {
        const PrimG p = P[i];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const unsigned long long a = kmin(p.lo[j], i), b = kmax(p.hi[j], i);
            const unsigned long long c = kmin(p.c[j], i), d = kmax(p.c[j], i);
            k[j] = a < k[j] ? a : k[j];
            k[3 + j] = b > k[3 + j] ? b : k[3 + j];
            k[6 + j] = c < k[6 + j] ? c : k[6 + j];
            k[9 + j] = d > k[9 + j] ? d : k[9 + j];
        }
    }
#pragma unroll
    for (int j = 0; j < 3; j++) {
        k[j] = warp_min64(k[j]);
        k[3 + j] = warp_max64(k[3 + j]);
        k[6 + j] = warp_min64(k[6 + j]);
        k[9 + j] = warp_max64(k[9 + j]);
    }
}

// The float that the winner of bounds key j (0-11) holds.
__device__ __forceinline__ float bounds_value(const PrimG* __restrict__ P, unsigned long long key, int j) {
    const PrimG& w = P[(j % 6) < 3 ? kpos_min(key) : kpos_max(key)];
    return j < 3 ? w.lo[j] : (j < 6 ? w.hi[j - 3] : w.c[j % 3]);
}

// Bin threshold lo + (hi - lo) * float(j + 1) / 5.
__device__ __forceinline__ float bin_threshold(float lo, float hi, int j) {
    return __fadd_rn(lo, __fdiv_rn(__fmul_rn(__fsub_rn(hi, lo), (float)(j + 1)), (float)kBins));
}

// Bins P[begin, end): counts and box keys, into shared memory.  A key is added
// only where it improves on what is there (64-bit shared minima are loops of
// compare and swap; most primitives improve nothing), counts once per warp.
__device__ __forceinline__ void fill_bins(const PrimG* __restrict__ P, int begin, int end,
                                          const float thr[3][kBins - 1],
                                          volatile unsigned long long s_bin[3][kBins][6], int s_cnt[3][kBins]) {
    const int lane = threadIdx.x & 31;
    int count[3] = {0, 0, 0};  // of bin `lane`
    for (int base = begin; base < end; base += blockDim.x) {
        const int i = base + (int)threadIdx.x;
        const bool on = i < end;
        PrimG p;
        if (on) p = P[i];
#pragma unroll
        for (int axis = 0; axis < 3; axis++) {
            const int b = on ? bin_of(p.c[axis], thr[axis]) : -1;
#pragma unroll
            for (int q = 0; q < kBins; q++) {
                const int c = __popc(__ballot_sync(0xffffffffu, b == q));
                if (lane == q) count[axis] += c;
            }
            if (on) {
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    const unsigned long long a = kmin(p.lo[j], i), d = kmax(p.hi[j], i);
                    if (a < s_bin[axis][b][j]) atomicMin((unsigned long long*)&s_bin[axis][b][j], a);
                    if (d > s_bin[axis][b][3 + j]) atomicMax((unsigned long long*)&s_bin[axis][b][3 + j], d);
                }
            }
        }
    }
    if (lane < kBins)
#pragma unroll
        for (int axis = 0; axis < 3; axis++)
            if (count[axis]) atomicAdd(&s_cnt[axis][lane], count[axis]);
}

// Split costs of one axis (bvh.h:57-149): the first strict minimum.
__device__ void axis_split(const PrimG* __restrict__ P, const unsigned long long bin[kBins][6], const int cnt[kBins],
                           float* cost, int* best) {
    float blo[kBins][3], bhi[kBins][3];
    for (int b = 0; b < kBins; b++)
        for (int j = 0; j < 3; j++) {
            if (cnt[b] > 0) {
                blo[b][j] = P[kpos_min(bin[b][j])].lo[j];
                bhi[b][j] = P[kpos_max(bin[b][3 + j])].hi[j];
            } else {
                blo[b][j] = __int_as_float(0x7f800000);
                bhi[b][j] = -__int_as_float(0x7f800000);
            }
        }
    float pc[kBins - 1];
    for (int i = 0; i < kBins - 1; i++) {
        float llo[3], lhi[3], rlo[3], rhi[3];
        for (int j = 0; j < 3; j++) {
            llo[j] = rlo[j] = __int_as_float(0x7f800000);
            lhi[j] = rhi[j] = -__int_as_float(0x7f800000);
        }
        int lc = 0, rc = 0;
        for (int b = 0; b < kBins; b++) {
            const int c = cnt[b];
            if (b <= i) {
                lc += c;
                if (c)
                    for (int j = 0; j < 3; j++) { llo[j] = vmin1(llo[j], blo[b][j]); lhi[j] = vmax1(lhi[j], bhi[b][j]); }
            } else {
                rc += c;
                if (c)
                    for (int j = 0; j < 3; j++) { rlo[j] = vmin1(rlo[j], blo[b][j]); rhi[j] = vmax1(rhi[j], bhi[b][j]); }
            }
        }
        pc[i] = (lc == 0 || rc == 0) ? __int_as_float(0x7f800000) : __fadd_rn(ref_area(llo, lhi), ref_area(rlo, rhi));
    }
    int m = 0;
    float mc = pc[0];
    for (int i = 1; i < kBins - 1; i++)
        if (pc[i] < mc) { mc = pc[i]; m = i; }
    *cost = mc;
    *best = m;
}

// The reference's nested axis choice (bvh.h:179-197).
__device__ __forceinline__ int pick_axis(const float cost[3]) {
    const float c1 = cost[0], c2 = cost[1], c3 = cost[2];
    if (c1 < c2) return (c1 < c3) ? 0 : (c2 < c3 ? 1 : 2);
    return (c2 < c3) ? 1 : 2;
}

// The node of a split segment and its children.
__device__ void emit_node(const SegG& seg, const float bounds[6], int nl, NodeG* __restrict__ nodes, const LevelOut& L) {
    const int nid = atomicAdd(L.counts + 1, 1);
    NodeG nd;
    for (int j = 0; j < 3; j++) { nd.lo[j] = bounds[j]; nd.hi[j] = bounds[3 + j]; }
    nd.parent = seg.parent;
    nd.side = seg.side;
    nd.child[0] = nd.child[1] = -1;
    nodes[nid] = nd;
    if (seg.parent >= 0) nodes[seg.parent].child[seg.side] = nid;
    emit_seg(L, SegG{seg.start, nl, nid, 0});
    emit_seg(L, SegG{seg.start + nl, seg.count - nl, nid, 1});
}

// P[begin, end) into Q in the bins' concatenation order (bin 0's primitives,
// then bin 1's, ..., each bin in input order): the first partition is bins
// 0..split, the second the rest (bvh.h:138-144).  run: where the range's first
// primitive of each bin goes.  All threads of the CTA.
__device__ __forceinline__ void scatter_bins(const PrimG* __restrict__ P, PrimG* __restrict__ Q, int begin, int end,
                                             int axis, const float* thr, int run[kBins], int (*s_wbin)[kBins]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    for (int base = begin; base < end; base += blockDim.x) {
        const int i = base + (int)threadIdx.x;
        PrimG p;
        int mb = -1;
        if (i < end) {
            p = P[i];
            mb = bin_of(p.c[axis], thr);
        }
        unsigned bal[kBins];
#pragma unroll
        for (int b = 0; b < kBins; b++) {
            bal[b] = __ballot_sync(0xffffffffu, mb == b);
            if (lane == b) s_wbin[warp][b] = __popc(bal[b]);
        }
        __syncthreads();
        if (i < end) {
            int pos = 0;
#pragma unroll
            for (int b = 0; b < kBins; b++)
                if (mb == b) pos = run[b] + __popc(bal[b] & ((1u << lane) - 1u));
            for (int w = 0; w < warp; w++) pos += s_wbin[w][mb];
            Q[pos] = p;
        }
#pragma unroll
        for (int b = 0; b < kBins; b++)
            for (int w = 0; w < warps; w++) run[b] += s_wbin[w][b];
        __syncthreads();
    }
}

__device__ __forceinline__ float okey_value(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// One level of the nodes of at most 32 primitives, a warp each with a primitive per
// lane and no barriers but the two around the CTA's additions to the counters.
// Children of fewer than 4 primitives become leaves at once.  Bound by the
// latency of its chain of warp reductions.  With a CTA of 128 threads, and two
// atomics on the counters, per node (and leaf) scene creation took 11.1 ms for
// the 192k-triangle room, now 10.4; 1M-triangle soup 22.8, now 18.9.
//
// The bounds are the reference's floats (the later of equal values); the bins'
// boxes only enter costs, where -0.0 and +0.0 give the same.
__device__ __forceinline__ void level_warp(const SegG* __restrict__ small, int n_small, int block,
                                           const PrimG* __restrict__ pin, PrimG* __restrict__ pout,
                                           NodeG* __restrict__ nodes, const LevelOut& L,
                                           int32_t* __restrict__ final_id, int32_t* __restrict__ leaf_parent) {
    constexpr unsigned full = 0xffffffffu;
    const float inf = __int_as_float(0x7f800000);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int w = block * kWarps + warp;
    SegG seg{0, 0, -1, 0};
    if (w < n_small) seg = small[w];
    const int n = seg.count;
    const bool on = lane < n;
    PrimG p{};
    if (on) p = pin[seg.start + lane];
    float bound[6];  // lo xyz, hi xyz
    int nl = 0, bin = -1;  // primitives of the first partition; this one's bin on the chosen axis
    if (n >= 4) {  // fewer: a leaf (bvh.h:152-158)
        uint32_t kl[3], kh[3];
        float cb[6];  // centroid bounds
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const uint32_t kc = okey(p.c[j]);
            kl[j] = okey(p.lo[j]);
            kh[j] = okey(p.hi[j]);
            auto later = [&](uint32_t key, uint32_t best, float v) {  // the last lane that holds the best key
                return __shfl_sync(full, v, 31 - __clz(__ballot_sync(full, on && key == best)));
            };
            bound[j] = later(kl[j], __reduce_min_sync(full, on ? kl[j] : full), p.lo[j]);
            bound[3 + j] = later(kh[j], __reduce_max_sync(full, on ? kh[j] : 0u), p.hi[j]);
            cb[j] = later(kc, __reduce_min_sync(full, on ? kc : full), p.c[j]);
            cb[3 + j] = later(kc, __reduce_max_sync(full, on ? kc : 0u), p.c[j]);
        }
        // thresholds: lane 4 axis + j
        const int ax = (lane >> 2) % 3;
        const float t = bin_threshold(ax == 0 ? cb[0] : (ax == 1 ? cb[1] : cb[2]),
                                      ax == 0 ? cb[3] : (ax == 1 ? cb[4] : cb[5]), lane & 3);
        // bins: lane kBins axis + b holds bin b's count and box
        int b[3], cnt = 0;
        float blo[3] = {inf, inf, inf}, bhi[3] = {-inf, -inf, -inf};
#pragma unroll
        for (int axis = 0; axis < 3; axis++) {
            float thr[kBins - 1];
#pragma unroll
            for (int j = 0; j < kBins - 1; j++) thr[j] = __shfl_sync(full, t, 4 * axis + j);
            b[axis] = on ? bin_of(p.c[axis], thr) : -1;
#pragma unroll
            for (int q = 0; q < kBins; q++) {
                const bool in = b[axis] == q, mine = lane == kBins * axis + q;
                const unsigned m = __ballot_sync(full, in);
                if (m == 0) continue;
                if (mine) cnt = __popc(m);
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    const uint32_t lo = __reduce_min_sync(full, in ? kl[j] : full);
                    const uint32_t hi = __reduce_max_sync(full, in ? kh[j] : 0u);
                    if (mine) {
                        blo[j] = okey_value(lo);
                        bhi[j] = okey_value(hi);
                    }
                }
            }
        }
        // split costs (bvh.h:57-149): lane 4 axis + i splits after bin i
        const int i = lane & 3;
        float llo[3] = {inf, inf, inf}, lhi[3] = {-inf, -inf, -inf}, rlo[3] = {inf, inf, inf}, rhi[3] = {-inf, -inf, -inf};
        int lc = 0, rc = 0;
#pragma unroll
        for (int q = 0; q < kBins; q++) {
            const int src = kBins * ax + q, c = __shfl_sync(full, cnt, src);
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const float lo = __shfl_sync(full, blo[j], src), hi = __shfl_sync(full, bhi[j], src);
                if (c == 0) continue;
                if (q <= i) {
                    llo[j] = vmin1(llo[j], lo);
                    lhi[j] = vmax1(lhi[j], hi);
                } else {
                    rlo[j] = vmin1(rlo[j], lo);
                    rhi[j] = vmax1(rhi[j], hi);
                }
            }
            if (q <= i) lc += c;
            else rc += c;
        }
        const float pc = (lc == 0 || rc == 0) ? inf : __fadd_rn(ref_area(llo, lhi), ref_area(rlo, rhi));
        float cost[3];
        int best[3];
#pragma unroll
        for (int axis = 0; axis < 3; axis++) {  // the first strict minimum
            cost[axis] = __shfl_sync(full, pc, 4 * axis);
            best[axis] = 0;
#pragma unroll
            for (int j = 1; j < kBins - 1; j++) {
                const float c = __shfl_sync(full, pc, 4 * axis + j);
                if (c < cost[axis]) {
                    cost[axis] = c;
                    best[axis] = j;
                }
            }
        }
        const int axis = pick_axis(cost);
        bin = axis == 0 ? b[0] : (axis == 1 ? b[1] : b[2]);
        const int last = axis == 0 ? best[0] : (axis == 1 ? best[1] : best[2]);
        nl = __popc(__ballot_sync(full, on && bin <= last));
    }
    const bool split = nl > 0 && nl < n;
    const int nr = n - nl;
    const int kids = split ? (nl >= 4) + (nr >= 4) : 0;
    __shared__ int s_split[kWarps], s_kids[kWarps], s_node, s_seg;
    if (lane == 0) {
        s_split[warp] = split;
        s_kids[warp] = kids;
    }
    __syncthreads();
    int node = 0, kid = 0, n_nodes = 0, n_kids = 0;
    for (int v = 0; v < kWarps; v++) {
        if (v < warp) {
            node += s_split[v];
            kid += s_kids[v];
        }
        n_nodes += s_split[v];
        n_kids += s_kids[v];
    }
    if (threadIdx.x == 0 && n_nodes > 0) s_node = atomicAdd(L.counts + 1, n_nodes);
    if (threadIdx.x == 32 && n_kids > 0) s_seg = atomicAdd(L.counts + 4, n_kids);
    __syncthreads();
    if (!split) {
        if (on) {
            final_id[seg.start + lane] = p.id;
            leaf_parent[seg.start + lane] = seg.parent;
        }
        return;
    }
    node += s_node;
    kid += s_seg;
    if (lane == 0) {
        NodeG nd;
        for (int j = 0; j < 3; j++) {
            nd.lo[j] = bound[j];
            nd.hi[j] = bound[3 + j];
        }
        nd.parent = seg.parent;
        nd.side = seg.side;
        nd.child[0] = nd.child[1] = -1;
        nodes[node] = nd;
        if (seg.parent >= 0) nodes[seg.parent].child[seg.side] = node;
        if (nl >= 4) L.small[kid++] = SegG{seg.start, nl, node, 0};
        if (nr >= 4) L.small[kid] = SegG{seg.start + nl, nr, node, 1};
    }
    // the bins' concatenation order (bvh.h:138-144)
    int pos = 0, before = 0;
#pragma unroll
    for (int q = 0; q < kBins; q++) {
        const unsigned m = __ballot_sync(full, bin == q);
        if (bin == q) pos = before + __popc(m & ((1u << lane) - 1u));
        before += __popc(m);
    }
    if (on) {
        if ((pos < nl ? nl : nr) < 4) {
            final_id[seg.start + pos] = p.id;
            leaf_parent[seg.start + pos] = node;
        } else {
            pout[seg.start + pos] = p;
        }
    }
}

// One level: a CTA per node of the list, then CTAs of kWarps small nodes each
// (one launch: a second one per level cost a 10k-triangle scene 0.15 ms).
__global__ void __launch_bounds__(kThreads) k_level(const SegG* __restrict__ segs, int n_seg,
                                                    const SegG* __restrict__ small, int n_small,
                                                    const PrimG* __restrict__ pin, PrimG* __restrict__ pout,
                                                    NodeG* __restrict__ nodes, LevelOut L,
                                                    int32_t* __restrict__ final_id, int32_t* __restrict__ leaf_parent) {
    __shared__ unsigned long long s_red[kWarps][12];
    __shared__ float s_bounds[12];  // lo xyz, hi xyz, centroid lo xyz, centroid hi xyz
    __shared__ unsigned long long s_bin[3][kBins][6];
    __shared__ int s_cnt[3][kBins], s_best[3];
    __shared__ float s_cost[3];
    __shared__ int s_axis, s_leaf;
    __shared__ float s_thr[3][kBins - 1];
    __shared__ int s_wbin[kWarps][kBins];
    if ((int)blockIdx.x >= n_seg) {
        level_warp(small, n_small, (int)blockIdx.x - n_seg, pin, pout, nodes, L, final_id, leaf_parent);
        return;
    }
    const SegG seg = segs[blockIdx.x];
    if (seg.count > kBigSeg) return;  // k_big_*
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const PrimG* P = pin + seg.start;
    const int n = seg.count;

    auto emit_leaf = [&]() {
        for (int i = tid; i < n; i += kThreads) {
            final_id[seg.start + i] = P[i].id;
            leaf_parent[seg.start + i] = seg.parent;
        }
    };
    // 1. bounds and centroid bounds
    {
        unsigned long long k[12];
        bounds_keys(P, 0, n, k);
        if (lane == 0)
#pragma unroll
            for (int j = 0; j < 12; j++) s_red[warp][j] = k[j];
        for (int j = tid; j < 3 * kBins * 6; j += kThreads) (&s_bin[0][0][0])[j] = comp_is_min(j % 6) ? ~0ull : 0ull;
        if (tid < 3 * kBins) (&s_cnt[0][0])[tid] = 0;
        __syncthreads();
        if (tid < 12) {
            const bool is_min = (tid % 6) < 3;
            unsigned long long r = s_red[0][tid];
            for (int w = 1; w < kWarps; w++) {
                const unsigned long long x = s_red[w][tid];
                r = is_min ? (x < r ? x : r) : (x > r ? x : r);
            }
            s_bounds[tid] = bounds_value(P, r, tid);
        }
        __syncthreads();
    }
    // 2. thresholds, then the bins
    if (tid < 3 * (kBins - 1)) {
        const int axis = tid / (kBins - 1), j = tid % (kBins - 1);
        s_thr[axis][j] = bin_threshold(s_bounds[6 + axis], s_bounds[9 + axis], j);
    }
    __syncthreads();
    fill_bins(P, 0, n, s_thr, s_bin, s_cnt);
    __syncthreads();
    // 3. split costs (one warp per axis, so that they overlap), axis
    if (lane == 0 && warp < 3) axis_split(P, s_bin[warp], s_cnt[warp], &s_cost[warp], &s_best[warp]);
    __syncthreads();
    if (tid == 0) {
        const int axis = pick_axis(s_cost);
        int nl = 0;
        for (int b = 0; b <= s_best[axis]; b++) nl += s_cnt[axis][b];
        s_axis = axis;
        s_leaf = (nl == 0 || nl == n) ? 1 : 0;
        if (!s_leaf) emit_node(seg, s_bounds, nl, nodes, L);
    }
    __syncthreads();
    if (s_leaf) {
        emit_leaf();
        return;
    }
    // 4. into pout
    const int axis = s_axis;
    int run[kBins];
    run[0] = 0;
#pragma unroll
    for (int b = 1; b < kBins; b++) run[b] = run[b - 1] + s_cnt[axis][b - 1];
    scatter_bins(P, pout + seg.start, 0, n, axis, s_thr[axis], run, s_wbin);
}

// ---------------------------------------------------------------------------
// The same steps for the large nodes of the top levels, a chunk of kBigChunk
// primitives per CTA: the chunks' bounds and bins meet in the node's BigG by
// atomic minima and maxima (of keys that make the result independent of the
// order), one CTA per node decides, and each chunk places its primitives after
// those of the chunks before it.  With one CTA of 128 threads per node the top
// levels were a serial pass over the scene each (18 ms for the root of 1M
// triangles).  Levels of the 192k-triangle room 19.9 -> 6.0 ms, of the
// 1M-triangle soup 104.8 -> 13.8 ms, with fill_bins' tests before its atomics.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kBigThreads) k_big_bounds(const ChunkG* __restrict__ chunks, BigG* __restrict__ big,
                                                            const PrimG* __restrict__ pin) {
    const ChunkG ch = chunks[blockIdx.x];
    BigG& B = big[ch.big];
    const int begin = ch.index * kBigChunk, end = min(begin + kBigChunk, B.seg.count);
    unsigned long long k[12];
    bounds_keys(pin + B.seg.start, begin, end, k);
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int j = 0; j < 12; j++) {
            if ((j % 6) < 3) atomicMin(&B.red[j], k[j]);
            else atomicMax(&B.red[j], k[j]);
        }
}

// The node's bounds (12 floats) and bin thresholds, for the CTA.
__device__ __forceinline__ void big_thresholds(const BigG& B, const PrimG* __restrict__ P, float* s_bounds,
                                               float (*s_thr)[kBins - 1]) {
    if (threadIdx.x < 12) s_bounds[threadIdx.x] = bounds_value(P, B.red[threadIdx.x], threadIdx.x);
    __syncthreads();
    if (threadIdx.x < 3 * (kBins - 1)) {
        const int axis = threadIdx.x / (kBins - 1), j = threadIdx.x % (kBins - 1);
        s_thr[axis][j] = bin_threshold(s_bounds[6 + axis], s_bounds[9 + axis], j);
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kBigThreads) k_big_bins(const ChunkG* __restrict__ chunks, BigG* __restrict__ big,
                                                          const PrimG* __restrict__ pin, int32_t* __restrict__ chunk_cnt) {
    __shared__ float s_bounds[12], s_thr[3][kBins - 1];
    __shared__ unsigned long long s_bin[3][kBins][6];
    __shared__ int s_cnt[3][kBins];
    const ChunkG ch = chunks[blockIdx.x];
    BigG& B = big[ch.big];
    const PrimG* P = pin + B.seg.start;
    const int begin = ch.index * kBigChunk, end = min(begin + kBigChunk, B.seg.count);
    for (int j = threadIdx.x; j < 3 * kBins * 6; j += blockDim.x) (&s_bin[0][0][0])[j] = comp_is_min(j % 6) ? ~0ull : 0ull;
    if (threadIdx.x < 3 * kBins) (&s_cnt[0][0])[threadIdx.x] = 0;
    big_thresholds(B, P, s_bounds, s_thr);
    fill_bins(P, begin, end, s_thr, s_bin, s_cnt);
    __syncthreads();
    for (int j = threadIdx.x; j < 3 * kBins * 6; j += blockDim.x) {
        const unsigned long long v = (&s_bin[0][0][0])[j];
        unsigned long long* g = &B.bin[0][0][0] + j;
        if (comp_is_min(j % 6)) atomicMin(g, v);
        else atomicMax(g, v);
    }
    if (threadIdx.x < 3 * kBins) {
        const int c = (&s_cnt[0][0])[threadIdx.x];
        chunk_cnt[(size_t)blockIdx.x * 3 * kBins + threadIdx.x] = c;
        if (c) atomicAdd(&B.cnt[0][0] + threadIdx.x, c);
    }
}

__global__ void __launch_bounds__(128) k_big_split(BigG* __restrict__ big, const PrimG* __restrict__ pin,
                                                   NodeG* __restrict__ nodes, LevelOut L) {
    __shared__ float s_cost[3], s_bounds[12];
    __shared__ int s_best[3];
    BigG& B = big[blockIdx.x];
    const PrimG* P = pin + B.seg.start;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x < 12) s_bounds[threadIdx.x] = bounds_value(P, B.red[threadIdx.x], threadIdx.x);
    if ((threadIdx.x & 31) == 0 && warp < 3) axis_split(P, B.bin[warp], B.cnt[warp], &s_cost[warp], &s_best[warp]);
    __syncthreads();
    if (threadIdx.x != 0) return;
    const int axis = pick_axis(s_cost);
    int nl = 0;
    for (int b = 0; b <= s_best[axis]; b++) nl += B.cnt[axis][b];
    B.axis = axis;
    B.leaf = (nl == 0 || nl == B.seg.count) ? 1 : 0;
    if (!B.leaf) emit_node(B.seg, s_bounds, nl, nodes, L);
}

__global__ void __launch_bounds__(kBigThreads) k_big_scatter(const ChunkG* __restrict__ chunks,
                                                             const BigG* __restrict__ big,
                                                             const PrimG* __restrict__ pin, PrimG* __restrict__ pout,
                                                             const int32_t* __restrict__ chunk_cnt,
                                                             int32_t* __restrict__ final_id,
                                                             int32_t* __restrict__ leaf_parent) {
    __shared__ float s_bounds[12], s_thr[3][kBins - 1];
    __shared__ int s_before[kBins];
    __shared__ int s_wbin[kBigThreads / 32][kBins];
    const ChunkG ch = chunks[blockIdx.x];
    const BigG& B = big[ch.big];
    const SegG seg = B.seg;
    const PrimG* P = pin + seg.start;
    const int begin = ch.index * kBigChunk, end = min(begin + kBigChunk, seg.count);
    if (B.leaf) {
        for (int i = begin + (int)threadIdx.x; i < end; i += blockDim.x) {
            final_id[seg.start + i] = P[i].id;
            leaf_parent[seg.start + i] = seg.parent;
        }
        return;
    }
    if (threadIdx.x < kBins) s_before[threadIdx.x] = 0;
    big_thresholds(B, P, s_bounds, s_thr);
    const int axis = B.axis;
    // each bin's primitives in the node's earlier chunks
    for (int e = threadIdx.x; e < ch.index * kBins; e += blockDim.x) {
        const int c = chunk_cnt[(size_t)(B.first + e / kBins) * 3 * kBins + axis * kBins + e % kBins];
        if (c) atomicAdd(&s_before[e % kBins], c);
    }
    __syncthreads();
    int run[kBins], base = 0;
#pragma unroll
    for (int b = 0; b < kBins; b++) {
        run[b] = base + s_before[b];
        base += B.cnt[axis][b];
    }
    scatter_bins(P, pout + seg.start, begin, end, axis, s_thr[axis], run, s_wbin);
}

// Subtree sizes (internal nodes), bottom-up: a thread starts at each node
// without internal children and climbs; the last of a node's arrivals
// (counted in `seen`, zeroed) finds its children's sizes and goes on (as
// k_collapse_cost in gpu_sah.cu, after Karras 2012).  One
// launch bound by the depth's chain of loads.  With a launch per level here and
// in k_preorder (92 for the 192k-triangle room) scene creation took 10.45 ms
// there, now 10.3; a 10k-triangle scene 3.72, now 3.56.
__global__ void k_sizes(const NodeG* __restrict__ nodes, int n, int32_t* __restrict__ seen, int32_t* __restrict__ size) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || nodes[i].child[0] >= 0 || nodes[i].child[1] >= 0) return;
    __stcg(size + i, 1);
    for (i = nodes[i].parent; i >= 0; i = nodes[i].parent) {
        const int a = nodes[i].child[0], b = nodes[i].child[1];
        __threadfence();
        if (atomicAdd(seen + i, 1) + 1 < (a >= 0) + (b >= 0)) return;
        __threadfence();
        __stcg(size + i, 1 + (a >= 0 ? __ldcg(size + a) : 0) + (b >= 0 ? __ldcg(size + b) : 0));
    }
}

// Pre-order numbers: the parent, then the first partition's subtree, then the
// second's, summed on the way to the root.
__global__ void k_preorder(const NodeG* __restrict__ nodes, int n, const int32_t* __restrict__ size,
                           int32_t* __restrict__ pre) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int number = 0;
    for (int k = i, p = nodes[i].parent; p >= 0; k = p, p = nodes[p].parent) {
        const int first = nodes[p].child[0];
        number += 1 + (nodes[k].side == 1 && first >= 0 ? size[first] : 0);
    }
    pre[i] = number;
}

__global__ void k_node_out(const NodeG* __restrict__ nodes, int n_nodes, const int32_t* __restrict__ pre,
                           float4* __restrict__ box, int32_t* __restrict__ parent) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_nodes) return;
    const NodeG& nd = nodes[i];
    const int p = pre[i];
    box[2 * (size_t)p] = make_float4(nd.lo[0], nd.lo[1], nd.lo[2], 0.f);
    box[2 * (size_t)p + 1] = make_float4(nd.hi[0], nd.hi[1], nd.hi[2], 0.f);
    parent[p] = nd.parent >= 0 ? pre[nd.parent] : -1;
}

__global__ void k_prim_out(const int32_t* __restrict__ final_id, const int32_t* __restrict__ leaf_parent, int n,
                           const int32_t* __restrict__ pre, int32_t* __restrict__ rank,
                           int32_t* __restrict__ prim_parent) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int id = final_id[i];
    rank[id] = i;
    const int lp = leaf_parent[i];
    prim_parent[id] = lp >= 0 ? pre[lp] : -1;
}

void ck(cudaError_t e, const char* what) {
    if (e != cudaSuccess) {
        cudaGetLastError();
        throw std::runtime_error(std::string("device BVH build: ") + what + ": " + cudaGetErrorString(e));
    }
}

template <class T>
T* dmalloc(std::vector<void*>& owned, size_t n) {
    void* p = nullptr;
    ck(cudaMalloc(&p, sizeof(T) * (n ? n : 1)), "cudaMalloc");
    owned.push_back(p);
    return static_cast<T*>(p);
}

}  // namespace

RefTree build_ref_tree(const float* d_tv, int n, cudaStream_t st, DeviceBufs& scratch, DeviceBufs& keep,
                       RefBuildStats* stats) {
    std::vector<void*>& owned = scratch.v;
    int* h_cnt = nullptr;  // pinned: LevelOut::counts
    ck(cudaMallocHost(&h_cnt, 5 * sizeof(int)), "cudaMallocHost");
    struct FreeHost {
        int* p;
        ~FreeHost() { cudaFreeHost(p); }
    } hguard{h_cnt};
    PrimG* buf[2] = {dmalloc<PrimG>(owned, n), dmalloc<PrimG>(owned, n)};
    // a split leaves at least one primitive on each side, so there are fewer
    // internal nodes than primitives, and at most n segments on a level
    const int max_nodes = n;
    NodeG* nodes = dmalloc<NodeG>(owned, max_nodes);
    SegG* segs[2] = {dmalloc<SegG>(owned, n + 2), dmalloc<SegG>(owned, n + 2)};
    SegG* small[2] = {dmalloc<SegG>(owned, n + 2), dmalloc<SegG>(owned, n + 2)};
    int* d_cnt = dmalloc<int>(owned, 5);  // LevelOut::counts
    const int max_big = n / kBigSeg + 1, max_chunks = n / kBigChunk + max_big + 1;
    BigG* big[2] = {dmalloc<BigG>(owned, max_big), dmalloc<BigG>(owned, max_big)};
    ChunkG* chunks[2] = {dmalloc<ChunkG>(owned, max_chunks), dmalloc<ChunkG>(owned, max_chunks)};
    int32_t* chunk_cnt = dmalloc<int32_t>(owned, (size_t)max_chunks * 3 * kBins);
    int32_t* final_id = dmalloc<int32_t>(owned, n);
    int32_t* leaf_parent = dmalloc<int32_t>(owned, n);
    k_prims<<<(n + 255) / 256, 256, 0, st>>>(d_tv, n, buf[0]);
    ck(cudaMemsetAsync(d_cnt, 0, 5 * sizeof(int), st), "memset");
    k_root<<<1, 1, 0, st>>>(LevelOut{segs[0], small[0], big[0], chunks[0], d_cnt}, n);
    int n_nodes = 0;
    int n_seg = n > 32 ? 1 : 0, n_small = n > 32 ? 0 : 1, cur = 0, levels = 0;
    int n_big = n > kBigSeg ? 1 : 0, n_chunks = n_big ? (n + kBigChunk - 1) / kBigChunk : 0;
    while (n_seg > 0 || n_small > 0) {
        const LevelOut L{segs[1 - cur], small[1 - cur], big[1 - cur], chunks[1 - cur], d_cnt};
        // all but the node count
        ck(cudaMemsetAsync(d_cnt, 0, sizeof(int), st), "memset");
        ck(cudaMemsetAsync(d_cnt + 2, 0, 3 * sizeof(int), st), "memset");
        k_level<<<n_seg + (n_small + kWarps - 1) / kWarps, kThreads, 0, st>>>(
            segs[cur], n_seg, small[cur], n_small, buf[cur], buf[1 - cur], nodes, L, final_id, leaf_parent);
        if (n_big > 0) {
            k_big_bounds<<<n_chunks, kBigThreads, 0, st>>>(chunks[cur], big[cur], buf[cur]);
            k_big_bins<<<n_chunks, kBigThreads, 0, st>>>(chunks[cur], big[cur], buf[cur], chunk_cnt);
            k_big_split<<<n_big, 128, 0, st>>>(big[cur], buf[cur], nodes, L);
            k_big_scatter<<<n_chunks, kBigThreads, 0, st>>>(chunks[cur], big[cur], buf[cur], buf[1 - cur], chunk_cnt,
                                                            final_id, leaf_parent);
        }
        ck(cudaGetLastError(), "level kernels");
        ck(cudaMemcpyAsync(h_cnt, d_cnt, 5 * sizeof(int), cudaMemcpyDeviceToHost, st), "counts");
        ck(cudaStreamSynchronize(st), "level");
        n_seg = h_cnt[0];
        n_big = h_cnt[2];
        n_chunks = h_cnt[3];
        n_small = h_cnt[4];
        n_nodes = h_cnt[1];
        if (h_cnt[1] > max_nodes || n_seg > n + 2 || n_small > n + 2 || n_big > max_big || n_chunks > max_chunks)
            throw std::runtime_error("device BVH build overflow");
        cur = 1 - cur;
        levels++;
    }
    int32_t* size = dmalloc<int32_t>(owned, n_nodes);
    int32_t* pre = dmalloc<int32_t>(owned, n_nodes);
    if (n_nodes > 0) {
        ck(cudaMemsetAsync(pre, 0, sizeof(int32_t) * (size_t)n_nodes, st), "memset");  // arrivals, until the numbers
        k_sizes<<<(n_nodes + 255) / 256, 256, 0, st>>>(nodes, n_nodes, pre, size);
        k_preorder<<<(n_nodes + 255) / 256, 256, 0, st>>>(nodes, n_nodes, size, pre);
    }
    float4* d_box = dmalloc<float4>(keep.v, 2 * (size_t)n_nodes);
    int32_t* d_parent = dmalloc<int32_t>(owned, n_nodes);
    int32_t* d_rank = dmalloc<int32_t>(owned, n);
    int32_t* d_pp = dmalloc<int32_t>(owned, n);
    if (n_nodes > 0) k_node_out<<<(n_nodes + 255) / 256, 256, 0, st>>>(nodes, n_nodes, pre, d_box, d_parent);
    k_prim_out<<<(n + 255) / 256, 256, 0, st>>>(final_id, leaf_parent, n, pre, d_rank, d_pp);
    ck(cudaGetLastError(), "outputs");
    ck(cudaStreamSynchronize(st), "outputs");
    if (stats) {
        stats->levels = levels;
        stats->nodes = n_nodes;
    }
    return RefTree{final_id, d_rank, d_pp, d_parent, d_box, n_nodes};
}

RefTopology build_ref_topology_device(const float* tri_v, int n, cudaStream_t st, RefBuildStats* stats) {
    RefTopology t;
    t.rank.assign(n, 0);
    t.prim_parent.assign(n, -1);
    if (n <= 0) return t;
    DeviceBufs scratch;
    float* d_tv = dmalloc<float>(scratch.v, 9 * (size_t)n);
    ck(cudaMemcpyAsync(d_tv, tri_v, sizeof(float) * 9 * (size_t)n, cudaMemcpyHostToDevice, st), "upload");
    const RefTree d = build_ref_tree(d_tv, n, st, scratch, scratch, stats);
    t.leaf_order.resize(n);
    t.node_box.resize(d.n_nodes);
    t.node_parent.resize(d.n_nodes);
    std::vector<float4> box(2 * (size_t)d.n_nodes);
    auto copy = [&](void* dst, const void* src, size_t bytes) {
        if (bytes) ck(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st), "copy");
    };
    copy(t.leaf_order.data(), d.leaf_order, sizeof(int32_t) * n);
    copy(t.rank.data(), d.rank, sizeof(int32_t) * n);
    copy(t.prim_parent.data(), d.prim_parent, sizeof(int32_t) * n);
    copy(box.data(), d.node_box, sizeof(float4) * box.size());
    copy(t.node_parent.data(), d.node_parent, sizeof(int32_t) * d.n_nodes);
    ck(cudaStreamSynchronize(st), "copies");
    for (int i = 0; i < d.n_nodes; i++) {
        std::memcpy(t.node_box[i].lo, &box[2 * (size_t)i], 12);
        std::memcpy(t.node_box[i].hi, &box[2 * (size_t)i + 1], 12);
    }
    return t;
}

}  // namespace cpppt_gb300
