// Device traversal of the compressed 4-wide BVH with the reference's exact
// closest-hit semantics (see bvh.h for why this reproduces BVH::intersect).
#pragma once
#include "dev_types.h"
#include "ray_range.h"

namespace cpppt_gb300 {

// Figures in this file: the two or more sides of a choice, measured together on
// the build of their time, on boxes whose clocks differ by several per cent.
// They compare with each other, not with those of another comment.  The whole
// now, in one session: 1.8M closest-hit rays 676 us, shadow rays 561 us, 1080p
// at 16 spp 68.8 ms (1M-triangle soup).
//
// Launch shape of the traversal kernels: threads per CTA and resident CTAs
// per SM (the grid is the latter times the SM count); 64 registers.  1024 x 1:
// 1.8M closest-hit rays on the 1M-triangle soup 967 us, 512 x 2 981 us; more
// threads (48 or 40 registers, spilling) were slower.
constexpr int kTraceThreads = 1024;
constexpr int kTraceBlocksPerSM = 1;
constexpr int kStackSize = kTraversalStackSize;
// Nodes whose entry distance exceeds best_t * (1 + 2^-8) are skipped.  The
// margin covers the rounding of the reference's Cramer-rule t (triangle.h:41-57)
// for every hit that is not within ~1e-4 rad of grazing the triangle.
constexpr float kCullScale = 1.00390625f;

// float(t) < 1e-4 (double) <=> t < kTriEps (triangle.h:55 compares with the double EPS)
__device__ __forceinline__ float tri_eps() { return __int_as_float(0x38d1b718); }  // nextafterf(1e-4f, inf)

struct HitRec {
    float t;
    int32_t prim;
    float beta, gamma;
    int32_t rank;
};

// Packed pairs of floats (two children per instruction on sm_100 and later:
// add.f32x2 / fma.f32x2 round each half exactly as add.f32 / fma.rn.f32).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk2(float a, float b) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ void upk2(f32x2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

__device__ __forceinline__ float m3r(float a, float b, float c) { return __fmul_rn(__fmul_rn(a, b), c); }

// Triangle::intersect up to acceptance (triangle.h:18-80): Cramer's rule with
// the reference's product and sum order, no fused multiply-add, IEEE
// reciprocal for 1.0/den (1.0 / float in double rounded to float is the
// correctly rounded float reciprocal).
__device__ __forceinline__ bool tri_exact(float4 A, float4 E1, float4 E2, float3 o, float3 d, float max_t,
                                          float& t, float& beta, float& gamma) {
    const float v1x = E1.x, v1y = E1.y, v1z = E1.z;
    const float v2x = E2.x, v2y = E2.y, v2z = E2.z;
    const float v3x = -d.x, v3y = -d.y, v3z = -d.z;
    const float vsx = __fsub_rn(o.x, A.x), vsy = __fsub_rn(o.y, A.y), vsz = __fsub_rn(o.z, A.z);
    float den = m3r(v1x, v2y, v3z);
    den = __fadd_rn(den, m3r(v2x, v3y, v1z));
    den = __fadd_rn(den, m3r(v3x, v1y, v2z));
    den = __fsub_rn(den, m3r(v3x, v2y, v1z));
    den = __fsub_rn(den, m3r(v3y, v2z, v1x));
    den = __fsub_rn(den, m3r(v3z, v2x, v1y));
    const float inv = __frcp_rn(den);
    float nt = m3r(v1x, v2y, vsz);
    nt = __fadd_rn(nt, m3r(v2x, vsy, v1z));
    nt = __fadd_rn(nt, m3r(vsx, v1y, v2z));
    nt = __fsub_rn(nt, m3r(vsx, v2y, v1z));
    nt = __fsub_rn(nt, m3r(vsy, v2z, v1x));
    nt = __fsub_rn(nt, m3r(vsz, v2x, v1y));
    t = __fmul_rn(nt, inv);
    if (t < tri_eps() || t > max_t) return false;
    float nb = m3r(vsx, v2y, v3z);
    nb = __fadd_rn(nb, m3r(v2x, v3y, vsz));
    nb = __fadd_rn(nb, m3r(v3x, vsy, v2z));
    nb = __fsub_rn(nb, m3r(v3x, v2y, vsz));
    nb = __fsub_rn(nb, m3r(v3y, v2z, vsx));
    nb = __fsub_rn(nb, m3r(v3z, v2x, vsy));
    beta = __fmul_rn(nb, inv);
    float ng = m3r(v1x, vsy, v3z);
    ng = __fadd_rn(ng, m3r(vsx, v3y, v1z));
    ng = __fadd_rn(ng, m3r(v3x, v1y, vsz));
    ng = __fsub_rn(ng, m3r(v3x, vsy, v1z));
    ng = __fsub_rn(ng, m3r(v3y, vsz, v1x));
    ng = __fsub_rn(ng, m3r(v3z, vsx, v1y));
    gamma = __fmul_rn(ng, inv);
    const float alpha = __fsub_rn(1.0f, __fadd_rn(gamma, beta));
    if (alpha < 0.f || alpha > 1.f || beta < 0.f || beta > 1.f || gamma < 0.f || gamma > 1.f) return false;
    // NaN t passes the reference's checks (it then accepts a NaN hit); such
    // rays lie exactly in the triangle's plane.  They are rejected here.
    return t == t;
}

// AABB::intersect_any (aabb.h:19-61) with the reference's division, order2
// swaps and comparison sequence.  `cand_t` stands in for the ray's running
// max_t, which only matters when tmax is NaN (a -0.0 direction component
// with the origin on the box's lower x plane).
__device__ __forceinline__ bool ref_box_exact(float4 lo, float4 hi, float3 o, float3 d, float cand_t) {
    float nminx = __fdiv_rn(__fsub_rn(lo.x, o.x), d.x);
    float nminy = __fdiv_rn(__fsub_rn(lo.y, o.y), d.y);
    float nminz = __fdiv_rn(__fsub_rn(lo.z, o.z), d.z);
    float nmaxx = __fdiv_rn(__fsub_rn(hi.x, o.x), d.x);
    float nmaxy = __fdiv_rn(__fsub_rn(hi.y, o.y), d.y);
    float nmaxz = __fdiv_rn(__fsub_rn(hi.z, o.z), d.z);
    float s;
    if (!(nmaxx >= nminx)) { s = nminx; nminx = nmaxx; nmaxx = s; }
    if (!(nmaxy >= nminy)) { s = nminy; nminy = nmaxy; nmaxy = s; }
    if (!(nmaxz >= nminz)) { s = nminz; nminz = nmaxz; nmaxz = s; }
    float tmin = nminx;
    if (tmin < nminy) tmin = nminy;
    if (tmin < nminz && nminz > nminy) tmin = nminz;
    float tmax = nmaxx;
    if (tmax > nmaxy) tmax = nmaxy;
    if (tmax > nmaxz && nmaxz < nmaxy) tmax = nmaxz;
    if (tmax < tmin) return false;
    if (tmin > 0.f && (double)tmin < (double)cand_t + 1e-4) return true;
    return tmax > 0.f;
}

// slab distances of byte children c and c + 1 of w: q B + A.  A byte permute
// builds 2^23 + q, an exact subtraction removes 2^23 (the integer pipe stays
// free for the min / max).
__device__ __forceinline__ void slab2(uint32_t w, int c, f32x2 B2, f32x2 A2, float& t0, float& t1) {
    const f32x2 q = pk2(__uint_as_float(__byte_perm(w, 0x4b000000u, 0x7540u | (uint32_t)c)),
                        __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7540u | (uint32_t)(c + 1))));
    upk2(fma2(add2(q, pk2(-8388608.0f, -8388608.0f)), B2, A2), t0, t1);
}

// three-operand min / max (one instruction on sm_100 and later)
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float fmin3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Per-lane traversal state (one ray in flight).  ANY=false: closest hit in
// `best` (best.t starts at the ray's max_t).  ANY=true: finishes at the first
// hit the reference would also report.
struct TraceCount {
    uint32_t nodes, tris;  // visited wide nodes, tested triangles (counting build only)
};

constexpr uint32_t kTravDone = 0xffffffffu;  // never a valid node or leaf reference
constexpr uint32_t kTravPop = 0x7fffffffu;   // take the next entry off the stack (never a valid node either)
constexpr uint32_t kLeafRef = 0x80000000u;

// kTravDone is the only reference with the leaf bit that is no leaf, and
// kTravPop the only one without it that is no node
__device__ __forceinline__ bool is_inner(uint32_t r) { return r < kTravPop; }
__device__ __forceinline__ bool is_leaf(uint32_t r) { return (int32_t)r < -1; }
__device__ __forceinline__ bool can_go(uint32_t r) { return (int32_t)r >= 0; }  // a node, or an entry to take

struct Trav {
    float3 o, d;
    float idx, idy, idz, oix, oiy, oiz;
    uint32_t neg;   // bit k: direction component k is negative
    uint32_t cur;   // next node or leaf to visit (kTravDone: nothing left on the stack)
    float cur_t;    // entry distance of cur
    uint32_t leaf;  // leaf postponed to the warp's next leaf phase (kTravDone: none)
    uint32_t sp;    // stack top (TravStack)
    int steps;
    HitRec best;
};

// Traversal stack of one lane: node references, and for closest-hit queries
// their entry distances.  The first entries lie in shared memory
// ([entry][thread], no bank conflicts whatever the lanes' depths), the rare
// rest in local memory.  Wholly in local memory the lanes' different depths
// made every access a scatter over lines that compete with the tree for L1:
// the any-hit kernel wrote 14 sectors per store and more to L2 than it read.
// The top is kept as the shared-memory address of the next entry, so a push is
// a store and an add; addresses past the region stand for the entries in local
// memory, and pushes go the short way while three more entries fit the region.
// Measured (1M-triangle soup, 1.8M closest-hit / shadow rays): all in local
// memory 1070 / 797 us, seven entries by index 1042 / 775 us; with addresses
// and 6, 8, 10, 12, 13 or 16 closest-hit entries 988, 948, 898, 862, 854, 852
// us, and 6, 8, 10, 12, 14 or 18 any-hit entries 693, 666, 637, 609, 604, 603
// us; 13 and 14 are 160 KB of an SM.
constexpr int kShortStack = 13;  // shared entries of a closest-hit lane (8 bytes each)
constexpr int kShortAny = 14;    // of an any-hit lane (4 bytes: an occlusion query culls nothing but by its own max_t)
// Bytes of the region of one kind of query.  A kernel that traces both has two
// regions: a warp may be at the second queue while another is at the first.
constexpr size_t stack_bytes(bool any, int threads) { return (size_t)(any ? 4 * kShortAny : 8 * kShortStack) * threads; }
constexpr size_t trace_smem(bool closest, bool any, int threads) {
    return (closest ? stack_bytes(false, threads) : 0) + (any ? stack_bytes(true, threads) : 0);
}
template <bool ANY, int THREADS>
struct TravStack {
    static constexpr int kShared = ANY ? kShortAny : kShortStack;
    static constexpr uint32_t kEntry = ANY ? 4u : 8u, kStep = kEntry * THREADS;
    uint32_t base;       // the thread's column
    uint32_t end;        // end of the region, the same for all threads: entries at or above it are local
    uint32_t fast;       // below it three more entries fit the region and the stack limit
    uint32_t ref[kStackSize - kShared];
    uint32_t t[ANY ? 1 : kStackSize - kShared];
    __device__ __forceinline__ TravStack(uint32_t* smem, int stack_limit) {
        const uint32_t s0 = (uint32_t)__cvta_generic_to_shared(smem);
        base = s0 + kEntry * threadIdx.x;
        end = s0 + kShared * kStep;
        const int f = min(kShared, stack_limit) - 2;
        fast = s0 + (f > 0 ? (uint32_t)f * kStep : 0u);
    }
    // entries on the stack
    __device__ __forceinline__ int depth(uint32_t sp) const { return (int)((sp - base) / kStep); }
    __device__ __forceinline__ void put_shared(uint32_t& sp, uint32_t r, uint32_t tb) const {
        if (ANY) asm volatile("st.shared.b32 [%0], %1;" ::"r"(sp), "r"(r));
        else asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(sp), "r"(r), "r"(tb));
        sp += kStep;
    }
    __device__ __forceinline__ void put(uint32_t& sp, uint32_t r, uint32_t tb) {
        if (sp < end) {
            put_shared(sp, r, tb);
            return;
        }
        const uint32_t k = (sp - end) / kStep;
        ref[k] = r;
        if (!ANY) t[k] = tb;
        sp += kStep;
    }
    __device__ __forceinline__ uint2 take(uint32_t& sp) const {
        sp -= kStep;
        uint2 e = make_uint2(0u, 0u);
        if (sp < end) {
            if (ANY) asm volatile("ld.shared.b32 %0, [%1];" : "=r"(e.x) : "r"(sp));
            else asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(e.x), "=r"(e.y) : "r"(sp));
        } else {
            const uint32_t k = (sp - end) / kStep;
            e.x = ref[k];
            if (!ANY) e.y = t[k];
        }
        return e;
    }
};

// root: wide-node index where the traversal starts (0 for a scene of its own;
// the scene's first node inside a merged multi-scene arena; kTravDone for a
// scene without triangles).
__device__ __forceinline__ void trav_init(Trav& T, uint32_t stack_base, float3 o, float3 d, float tmax0, uint32_t root) {
    T.o = o;
    T.d = d;
    T.best.t = tmax0;
    T.best.prim = -1;
    T.best.rank = -1;
    T.best.beta = T.best.gamma = 0.f;
    const float tiny = 7.888609052210118e-31f;  // 2^-100 stands in for a zero component
    const float dx = d.x == 0.f ? copysignf(tiny, d.x) : d.x;
    const float dy = d.y == 0.f ? copysignf(tiny, d.y) : d.y;
    const float dz = d.z == 0.f ? copysignf(tiny, d.z) : d.z;
    T.idx = 1.0f / dx;
    T.idy = 1.0f / dy;
    T.idz = 1.0f / dz;
    T.oix = o.x * T.idx;
    T.oiy = o.y * T.idy;
    T.oiz = o.z * T.idz;
    T.neg = (T.idx < 0.f ? 1u : 0u) | (T.idy < 0.f ? 2u : 0u) | (T.idz < 0.f ? 4u : 0u);
    T.cur = root;
    T.cur_t = 0.f;
    T.leaf = kTravDone;
    T.sp = stack_base;
    T.steps = 0;
}

__device__ __forceinline__ float cull_dist(const Trav& T) { return T.best.t * kCullScale + 1e-6f; }

// Next stacked node that is still in front of the best hit.
template <class Stack>
__device__ __forceinline__ void trav_pop(Trav& T, const Stack& K) {
    const float cull = cull_dist(T);
    while (T.sp != K.base) {
        const uint2 e = K.take(T.sp);
        if (__uint_as_float(e.y) <= cull) {
            T.cur = e.x;
            T.cur_t = __uint_as_float(e.y);
            return;
        }
    }
    T.cur = kTravDone;
}

__device__ __forceinline__ void trav_abort(Trav& T, uint32_t* status, uint32_t bit) {
    atomicOr(status, bit);
    T.cur = kTravDone;
    T.leaf = kTravDone;
}

// 32 bytes of a node in one load (sm_100 and later).
__device__ __forceinline__ void ld256(const uint4* p, uint4& a, uint4& b) {
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
        : "l"(p));
}

// One inner node (T.cur): a child that the ray enters in front of the best
// hit is next -- the nearest for a closest-hit query, the first in slot order
// for an any-hit query -- and the other entered children are pushed, for a
// closest-hit query with the second nearest on top.  (Culling compares each
// popped entry with the best hit, so the order changes the work, never the
// answer.)  kTravPop when no child is entered.  The nearest two come from two
// ordered pairs of children, with the references selected along: as many
// instructions as finding the nearest alone by keys that carry the slot.
// Against pushing in slot order: 1M rays in the 192k-triangle room 263 -> 207
// us, 1.8M on the 1M-triangle soup 753 -> 731, 1080p at 16 spp there 75.1 ->
// 74.0 ms, guided 720p in the room 10.8 -> 10.1 ms.  An any-hit query that
// takes the nearest first: room 124 -> 132 us, the farthest first: soup 578
// -> 715 us.  Two 256-bit loads instead of four of 128 bits: 1080p, 16 spp on
// the 1M-triangle soup 89.6 -> 88.3 ms.
template <bool ANY, bool COUNT, class Stack>
__device__ __forceinline__ void trav_node(Trav& T, Stack& K, const DevScene& S, uint32_t* status, TraceCount& cnt) {
    if (COUNT) cnt.nodes++;
    const uint4* np = S.nodes + 4 * (size_t)T.cur;
    uint4 w0, w1, w2, w3;
    ld256(np, w0, w1);
    ld256(np + 2, w2, w3);
    const float cull = cull_dist(T);
    // slab distance of quantised coordinate q on axis k:
    //   (p + q s - o) / d = q (s/d) + (p - o)/d = q B + A
    const float ax = fmaf(__uint_as_float(w0.x), T.idx, -T.oix);
    const float ay = fmaf(__uint_as_float(w0.y), T.idy, -T.oiy);
    const float az = fmaf(__uint_as_float(w0.z), T.idz, -T.oiz);
    const float bx = __uint_as_float((w0.w & 0xffu) << 23) * T.idx;
    const float by = __uint_as_float(((w0.w >> 8) & 0xffu) << 23) * T.idy;
    const float bz = __uint_as_float(((w0.w >> 16) & 0xffu) << 23) * T.idz;
    // words: lo_x lo_y lo_z hi_x | hi_y hi_z ref0 ref1 | ref2 ref3
    const bool nxs = T.neg & 1u, nys = T.neg & 2u, nzs = T.neg & 4u;
    const uint32_t nx = nxs ? w1.w : w1.x, fx = nxs ? w1.x : w1.w;
    const uint32_t ny = nys ? w2.x : w1.y, fy = nys ? w1.y : w2.x;
    const uint32_t nz = nzs ? w2.y : w1.z, fz = nzs ? w1.z : w2.y;
    uint32_t key[4];
    // children in pairs (packed adds and FMAs, the roundings of scalar ones)
    const f32x2 BX = pk2(bx, bx), BY = pk2(by, by), BZ = pk2(bz, bz);
    const f32x2 AX = pk2(ax, ax), AY = pk2(ay, ay), AZ = pk2(az, az);
#pragma unroll
    for (int c = 0; c < 4; c += 2) {
        float tnx[2], tny[2], tnz[2], tfx[2], tfy[2], tfz[2];
        slab2(nx, c, BX, AX, tnx[0], tnx[1]);
        slab2(ny, c, BY, AY, tny[0], tny[1]);
        slab2(nz, c, BZ, AZ, tnz[0], tnz[1]);
        slab2(fx, c, BX, AX, tfx[0], tfx[1]);
        slab2(fy, c, BY, AY, tfy[0], tfy[1]);
        slab2(fz, c, BZ, AZ, tfz[0], tfz[1]);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float tn = fmax3(tnx[h], tny[h], fmaxf(tnz[h], 0.0f));
            const float tf = fmin3(tfx[h], tfy[h], fminf(tfz[h], cull));
            const bool hit = tn <= tf * 1.0000005f;
            if (ANY) key[c + h] = hit ? 0u : 0xffffffffu;
            else key[c + h] = hit ? __float_as_uint(tn) : 0xffffffffu;  // tn >= 0: ordered as its bits
        }
    }
    // Indexed by constants only: with a run-time index (the nearest child's) the
    // array lives in local memory, a 16-byte store and a load per node visit
    // (closest hits of 1.8M rays on the 1M-triangle soup 1057 us, with selects
    // 1026 us; 1M rays in the 192k-triangle room 325 -> 318 us).
    const uint32_t refs[4] = {w2.z, w2.w, w3.x, w3.y};
    if (ANY) {
        const bool v0 = key[0] == 0u, v1 = key[1] == 0u, v2 = key[2] == 0u, v3 = key[3] == 0u;
        const bool p1 = v1 && v0, p2 = v2 && (v0 || v1), p3 = v3 && (v0 || v1 || v2);
        const uint32_t nxt = v0 ? refs[0] : (v1 ? refs[1] : (v2 ? refs[2] : (v3 ? refs[3] : kTravPop)));
        if (T.sp < K.fast) {
            if (p3) K.put_shared(T.sp, refs[3], 0u);
            if (p2) K.put_shared(T.sp, refs[2], 0u);
            if (p1) K.put_shared(T.sp, refs[1], 0u);
        } else {
            if (K.depth(T.sp) + 3 > S.stack_limit) {
                trav_abort(T, status, kStatusStackOverflow);
                return;
            }
            if (p3) K.put(T.sp, refs[3], 0u);
            if (p2) K.put(T.sp, refs[2], 0u);
            if (p1) K.put(T.sp, refs[1], 0u);
        }
        T.cur = nxt;
        T.cur_t = 0.f;
        return;
    }
    // the pairs (0, 1) and (2, 3), the nearer child first
    const bool p = key[1] < key[0], q = key[3] < key[2];
    const uint32_t ka = min(key[0], key[1]), kb = max(key[0], key[1]);
    const uint32_t kc = min(key[2], key[3]), kd = max(key[2], key[3]);
    const uint32_t ra = p ? refs[1] : refs[0], rb = p ? refs[0] : refs[1];
    const uint32_t rc = q ? refs[3] : refs[2], rd = q ? refs[2] : refs[3];
    const uint32_t k0 = min(ka, kc);
    if (k0 == 0xffffffffu) {
        T.cur = kTravPop;
        return;
    }
    // the pair with the nearest child, and the two children between it and the farthest
    const bool f = kc < ka;
    const uint32_t kn = f ? kd : kb, rn = f ? rd : rb;  // the nearest's neighbour
    const uint32_t kf = max(ka, kc), rf = f ? ra : rc;  // the nearer child of the other pair
    const uint32_t kl = f ? kb : kd, rl = f ? rb : rd;  // its farther one
    const bool g = kn < kf;
    const uint32_t k1 = min(kn, kf), r1 = g ? rn : rf;
    const uint32_t k2 = max(kn, kf), r2 = g ? rf : rn;
    if (T.sp < K.fast) {
        if (kl != 0xffffffffu) K.put_shared(T.sp, rl, kl);
        if (k2 != 0xffffffffu) K.put_shared(T.sp, r2, k2);
        if (k1 != 0xffffffffu) K.put_shared(T.sp, r1, k1);
    } else {
        if (K.depth(T.sp) + 3 > S.stack_limit) {
            trav_abort(T, status, kStatusStackOverflow);
            return;
        }
        if (kl != 0xffffffffu) K.put(T.sp, rl, kl);
        if (k2 != 0xffffffffu) K.put(T.sp, r2, k2);
        if (k1 != 0xffffffffu) K.put(T.sp, r1, k1);
    }
    T.cur = f ? rc : ra;
    T.cur_t = __uint_as_float(k0);
}

// The postponed leaf T.leaf.  Returns true when an any-hit query is answered.
template <bool ANY, bool COUNT>
__device__ __forceinline__ bool trav_leaf(Trav& T, const DevScene& S, TraceCount& cnt) {
    const uint32_t start = T.leaf & 0x7ffffffu;
    const uint32_t count = ((T.leaf >> 27) & 15u) + 1u;
    T.leaf = kTravDone;
    if (COUNT) cnt.tris += count;
    for (uint32_t k = 0; k < count; k++) {
        const float4* tp = S.tris + 3 * (size_t)(start + k);
        const float4 A = __ldg(tp), E1 = __ldg(tp + 1), E2 = __ldg(tp + 2);
        float t, beta, gamma;
        // ANY: best.t is the ray's own max_t until the first hit
        if (!tri_exact(A, E1, E2, T.o, T.d, T.best.t, t, beta, gamma)) continue;
        const int32_t rank = __float_as_int(A.w);
        if (!ANY && !(t < T.best.t || rank > T.best.rank)) continue;  // equal t: the later-visited wins
        const int32_t parent = __float_as_int(E1.w);
        if (parent >= 0) {
            const float4 lo = __ldg(S.ref_box + 2 * parent), hi = __ldg(S.ref_box + 2 * parent + 1);
            if (!ref_box_exact(lo, hi, T.o, T.d, t)) continue;
        }
        T.best.t = t;
        T.best.rank = rank;
        T.best.prim = __float_as_int(E2.w);
        T.best.beta = beta;
        T.best.gamma = gamma;
        if (ANY) {
            T.cur = kTravDone;
            return true;
        }
    }
    return false;
}

// One node phase and one leaf phase of a warp, n_act of whose lanes have rays
// (the others' cur and leaf are kTravDone).  Leaves are postponed as in Aila
// and Laine 2009, "Understanding the efficiency of ray traversal on GPUs": a
// lane that reaches a leaf parks it and keeps descending inner nodes; the node
// phase goes on while more than two thirds of the lanes with rays can (have a
// node, or a stacked entry to take), then the lanes with a parked leaf test its
// triangles together.  The result does not depend on the visiting order: the
// closest hit is the minimum over the tested triangles of (t, -rank), and a
// node is culled only when its entry distance lies behind the best hit.
//
// There is one place for each kind of work -- taking an entry off the stack,
// visiting a node, parking a leaf -- and the warp reconverges before the node:
// with the pops inlined where they arise (no child entered, leaf parked, entry
// culled), lanes went through the same code one group after another.  Finished
// lanes count as unable to go on, so they get a new ray soon.  Measured
// (1M-triangle soup, with the stack above) 1.8M closest-hit rays 1042 -> 967
// us, shadow rays 774 -> 739 us, 1M rays in the 192k-triangle room 324 -> 297
// us, 1080p at 16 spp 94.8 -> 88.2 ms.  Phase end at a half of the lanes 91.5
// ms, three fifths 89.5, three quarters 89.6; counting only lanes that wait on
// a leaf (a third of them) 90.5.
//
// The step limit is tested at every node visit, inside the phase, so the phase
// ends whatever the nodes hold: it goes on only while some lane has a node to
// visit, which takes one of that lane's steps, or an entry to take, of which
// its visits pushed at most three each.  (Tested once after the phase instead:
// closest hit 1 % faster, any hit 0.9 %, 1080p 0.5 %, but then a walk that
// pushes nothing is not bounded, and a ray whose last step was a leaf counts
// as over the limit.)
template <bool ANY, bool COUNT, class Stack>
__device__ __forceinline__ void trav_round(const DevScene& S, Trav& T, Stack& K, int n_act, uint32_t* status,
                                           TraceCount& cnt) {
    unsigned go;
    do {
        if (T.cur == kTravPop) trav_pop(T, K);
        __syncwarp();
        if (is_inner(T.cur)) {
            if (++T.steps > S.step_limit) trav_abort(T, status, kStatusIterLimit);
            else trav_node<ANY, COUNT>(T, K, S, status, cnt);
        }
        if (is_leaf(T.cur) && T.leaf == kTravDone) {
            T.leaf = T.cur;
            T.cur = kTravPop;
        }
        if (T.cur == kTravPop && T.sp == K.base) T.cur = kTravDone;
        go = __ballot_sync(0xffffffffu, can_go(T.cur));
    } while (3 * __popc(go) > 2 * n_act);
    if (T.leaf != kTravDone) {
        ++T.steps;
        if (!trav_leaf<ANY, COUNT>(T, S, cnt)) {
            if (!ANY && T.cur != kTravDone && T.cur_t > cull_dist(T)) T.cur = kTravPop;
            if (is_leaf(T.cur)) {
                T.leaf = T.cur;
                T.cur = kTravPop;
            }
        }
    }
}

// smem: the stacks' shared region (stack_bytes(ANY, THREADS)).
// Persistent ray loop.  Each warp takes chunks of up to kChunk consecutive
// rays (ray_chunk) into a warp-private range, the first one by its number and
// the next ones from a global counter; between rounds every lane whose ray
// has finished takes the next one, across the end of the range if need be (a
// lane left idle until the next fetch cost 4 % at 1080p).
// own_first = false: the first chunk comes from the counter too (a kernel's
// second queue, which warps reach at different times).
// load(i, o, d, tmax, root) fetches ray i; root arrives set to the scene's
// own root and may be replaced (rays of a merged multi-scene arena).
template <bool ANY, bool COUNT, int THREADS = kTraceThreads, class Load, class Store>
__device__ __forceinline__ void persistent_trace(const DevScene& S, uint32_t* __restrict__ smem, int n, int* counter,
                                                 uint32_t* status, TraceCount& cnt, Load load, Store store,
                                                 bool own_first = true) {
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lt_mask = (1u << lane) - 1u;
    Trav T;
    TravStack<ANY, THREADS> K(smem, S.stack_limit);
    T.cur = T.leaf = kTravDone;
    T.steps = 0;
    int ray = -1;
    // warp-uniform ray range; the first one is the warp's own (warps numbered
    // across the CTAs, so a small batch spreads over every SM), later ones
    // come from the counter
    const int nwarps = (int)(gridDim.x * (blockDim.x >> 5));
    const int c0 = own_first ? ray_chunk(n, nwarps, 1) : 0;
    RayRange pool = fetched_range(0, (int)((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * c0, c0, n);
    bool exhausted = nwarps * c0 >= n;
    while (true) {
        const unsigned idle = __ballot_sync(0xffffffffu, ray < 0);
        if (idle) {
            const uint32_t want = __popc(idle);
            RayRange after{pool.end, pool.end};  // the range after the present one
            if (pool.end - pool.next < want && !exhausted) {
                const int chunk = ray_chunk(n - (int)pool.end, nwarps, 2);
                int taken = 0;
                if (lane == 0) taken = atomicAdd(counter, chunk);
                after = fetched_range(__shfl_sync(0xffffffffu, taken, 0), nwarps * c0, chunk, n);
                exhausted = after.end == (uint32_t)n;
            }
            uint32_t i;
            const bool more = ray_of(__popc(idle & lt_mask), pool, after, i);
            if (ray < 0 && more) {
                ray = (int)i;
                float3 o, d;
                float tmax;
                uint32_t root = S.n_tris > 0 ? 0u : kTravDone;
                load(ray, o, d, tmax, root);
                trav_init(T, K.base, o, d, tmax, root);
            }
            pool = left_of(want, pool, after);
        }
        const unsigned act = __ballot_sync(0xffffffffu, ray >= 0);
        if (act == 0) break;
        trav_round<ANY, COUNT>(S, T, K, __popc(act), status, cnt);
        if (ray >= 0 && T.cur == kTravDone && T.leaf == kTravDone) {
            store(ray, T.best);
            ray = -1;
        }
    }
}

// Traces one ray per lane (active lanes' T, set up by trav_init) to the end:
// the closest hit, or with `any` until the first hit (the same test against
// the ray's own max_t, which best.t holds until then).  All 32 lanes call it.
template <class Stack>
__device__ __forceinline__ void warp_trace(const DevScene& S, Trav& T, Stack& K, bool active, bool any,
                                           uint32_t* status) {
    TraceCount cnt{0u, 0u};
    if (!active) T.cur = T.leaf = kTravDone;
    while (true) {
        const unsigned act = __ballot_sync(0xffffffffu, T.cur != kTravDone || T.leaf != kTravDone);
        if (act == 0) break;
        trav_round<false, false>(S, T, K, __popc(act), status, cnt);
        if (any && T.best.prim >= 0) {
            T.cur = T.leaf = kTravDone;
        }
    }
}

}  // namespace cpppt_gb300
