// SD-tree guided path tracing on the GPU: PPG::integrate
// (src/renderer/ppg.h:41-144) in the wavefront.  The SD-tree is built and
// updated on the host (sdtree.cpp); here it is looked up, sampled and
// splatted into.
//
// PPG keeps every path's vertices until the path ends (the splat needs the
// product of the factors that follow each vertex, ppg.h:131-141), so a path
// owns a slot of max_depth vertex records for its lifetime.  Slots come from
// a free list: k_generate_ppg pops, terminating paths push.
#include <cuda_runtime.h>

#include "launch.cuh"
#include "guide.h"
#include "shade.cuh"

namespace cpppt_gb300 {

constexpr float kPiPPG = 3.14159265358979323846f;

// SDTree::get_leaf(pt) (sdtree.h:354-406): midpoint splits, axis = depth % 3,
// right iff coordinate > mid.
__device__ __forceinline__ int sd_dtree(const DevSDTree& T, f3 p) {
    float lo[3] = {T.lo[0], T.lo[1], T.lo[2]}, hi[3] = {T.hi[0], T.hi[1], T.hi[2]};
    const float pc[3] = {p.x, p.y, p.z};
    int node = 0;
    for (int depth = 0; depth < 64; depth++) {
        const int2 n = __ldg(T.snode + node);
        if (n.x < 0) return -1 - n.x;
        const int k = depth % 3;
        const float mid = (lo[k] + hi[k]) * 0.5f;
        if (pc[k] > mid) { lo[k] = mid; node = n.y; }
        else { hi[k] = mid; node = n.x; }
    }
    return -1;
}

// DTree leaf lookup (SDTree::get_leaf / get_area, sdtree.h:277-352).
// Returns the value slot; *area = size_phi * size_cos of the leaf cell.
__device__ __forceinline__ int sd_dleaf(const DevSDTree& T, int dtree, float x, float y, float* area) {
    float lx = -kPiPPG, ly = -1.0f, hx = kPiPPG, hy = 1.0f;
    int node = __ldg(T.dtree_root + dtree);
    for (int depth = 0; depth < 48; depth++) {
        const int c = __ldg(T.dnode + node);
        if (c < 0) {
            *area = (hx - lx) * (hy - ly);
            return -1 - c;
        }
        const float mx = (lx + hx) * 0.5f, my = (ly + hy) * 0.5f;
        int child;
        if (x < mx) {
            if (y < my) { child = 0; hx = mx; hy = my; }
            else { child = 2; hx = mx; ly = my; }
        } else {
            if (y < my) { child = 1; lx = mx; hy = my; }
            else { child = 3; lx = mx; ly = my; }
        }
        node = c + child;
    }
    *area = 1.0f;
    return -1;
}

// SDTree::pdf (sdtree.h:525-537)
__device__ __forceinline__ float sd_pdf(const DevSDTree& T, f3 p, f3 dir) {
    const int t = sd_dtree(T, p);
    if (t < 0) return 0.f;
    float area;
    sd_dleaf(T, t, atan2f(dir.y, dir.x), dir.z, &area);
    return (1.0f / (float)__ldg(T.leaf_cnt + t)) * (1.0f / area);
}

// SDTree::sample -> sample_direction (sdtree.h:408-430,445-451): uniform over
// the quadtree's leaves, uniform in (phi, cos theta) inside the leaf.
__device__ __forceinline__ BSample sd_sample(const DevSDTree& T, f3 p, float u0, float u1, float u2) {
    BSample s;
    const int t = sd_dtree(T, p);
    const int sz = t >= 0 ? __ldg(T.leaf_cnt + t) : 1;
    const int i = ((int)(u0 * (float)sz)) % sz;
    const float4 L = t >= 0 ? __ldg(T.leaves + __ldg(T.leaf_off + t) + i) : make_float4(-kPiPPG, -1.f, 2.f * kPiPPG, 2.f);
    const float phi = L.x + u1 * L.z;
    const float ct = L.y + u2 * L.w;
    const float st = sqrtf(fmaxf(0.f, 1.0f - ct * ct));
    float sp, cp;
    sincosf(phi, &sp, &cp);
    s.wi = mk(cp * st, sp * st, ct);
    s.pdf = 1.0f / ((float)sz * (L.z * L.w));
    s.delta = false;
    return s;
}

// SDTree::splat (sdtree.h:514-524), by the lanes that have one (`on`; the
// whole warp calls).  The count and sum of a spatial leaf are added once per
// warp for each leaf its lanes hit: few leaves take all of a pass's splats,
// and additions to one address follow one another.
__device__ __forceinline__ void sd_splat_warp(const DevSDTree& T, bool on, float rad, f3 p, f3 dir) {
    const unsigned lane = threadIdx.x & 31u;
    const int t = on ? sd_dtree(T, p) : -1;
    if (t >= 0) {
        float area;
        const int slot = sd_dleaf(T, t, atan2f(dir.y, dir.x), dir.z, &area);
        if (slot >= 0) atomicAdd(T.slot_value + slot, rad);
    }
    // the sum over the lanes of one leaf: in each step a lane takes in the next
    // one of those that remain, and every second one leaves
    const unsigned group = __match_any_sync(0xffffffffu, t);
    const int rank = __popc(group & ((1u << lane) - 1u));
    unsigned rest = group & (0xfffffffeu << lane);  // remaining lanes above this one
    unsigned kept = group;
    float sum = t >= 0 ? rad : 0.f;
    for (int bit = 0; __any_sync(0xffffffffu, rest != 0); bit++) {
        const int next = __ffs(rest);
        const float x = __shfl_sync(0xffffffffu, sum, next ? next - 1 : (int)lane);
        if (next) sum += x;
        kept = __ballot_sync(0xffffffffu, (rank >> bit & 1) == 0) & kept;
        rest &= kept;
    }
    if (t >= 0 && rank == 0) {
        atomicAdd(T.dtree_count + t, __popc(group));
        atomicAdd(T.dtree_rad + t, sum);
    }
}

constexpr int kShadePPGThreads = 256;
// Backward products and splats of the finished paths (ppg.h:131-141): vertex k
// receives the largest channel of the product of the factors of vertices
// k..n-1, taken from the last one down.  The path's thread puts the running
// products in the place of the factors, four loads ahead; then a thread per
// vertex of the CTA's finished paths, found in the running total of their
// vertices, splats: the tree walks are chains of dependent loads, and one thread
// walking for vertex after vertex left the SM at 6 % of its issue slots (Cornell
// box 128x128, 64 spp: render 4.35 -> 3.60 ms with the sums per warp).  With the
// products multiplied anew by each vertex's thread a path of n vertices cost
// n^2 / 2 loads: that render 3.19 ms, now 3.10; the splats of 64 paths of 8000
// vertices 218 ms, now 7.
// slot: the thread's path, n_splat: its vertices (0: none to splat), last: the
// last one's factor.  All threads of the CTA call it.
__device__ __forceinline__ void splat_paths(const DevSDTree& T, const PPGVerts& V, int max_depth, int slot, int n_splat,
                                            f3 last) {
    constexpr int kWarps = kShadePPGThreads / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (n_splat > 1) {
        constexpr int kAhead = 4;  // factors read at a time
        const size_t base = (size_t)slot * max_depth;
        f3 acc = last;
        for (int v = n_splat - 2; v >= 0; v -= kAhead) {
            float2 b[kAhead];
            float c[kAhead];
#pragma unroll
            for (int j = 0; j < kAhead; j++)
                if (v >= j) {
                    b[j] = reinterpret_cast<const float2*>(V.vd + base + v - j)[1];
                    c[j] = V.vr[base + v - j];
                }
#pragma unroll
            for (int j = 0; j < kAhead; j++)
                if (v >= j) {
                    acc = acc * mk(b[j].x, b[j].y, c[j]);
                    reinterpret_cast<float2*>(V.vd + base + v - j)[1] = make_float2(acc.x, acc.y);
                    V.vr[base + v - j] = acc.z;
                }
        }
    }
    __shared__ int s_first[kShadePPGThreads], s_slot[kShadePPGThreads], s_total[kWarps];
    int incl = n_splat;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_total[warp] = incl;
    __syncthreads();
    int before = 0, n_verts = 0;
    for (int w = 0; w < kWarps; w++) {
        if (w < warp) before += s_total[w];
        n_verts += s_total[w];
    }
    s_first[threadIdx.x] = before + incl - n_splat;
    s_slot[threadIdx.x] = slot;
    __syncthreads();
    for (int j0 = 0; j0 < n_verts; j0 += kShadePPGThreads) {
        const int j = j0 + (int)threadIdx.x;
        const bool on = j < n_verts;
        float rad = 0.f;
        f3 vp = mk(0.f, 0.f, 0.f), vd = vp;
        if (on) {
            int path = 0;  // the last one that starts at or before j; those without vertices start with their successor
            for (int step = kShadePPGThreads / 2; step > 0; step >>= 1)
                if (s_first[path + step] <= j) path += step;
            const int k = j - s_first[path];
            const size_t vi = (size_t)s_slot[path] * max_depth + k;
            const float4 a = V.vp[vi], b = V.vd[vi];
            rad = fmaxf(b.z, fmaxf(b.w, V.vr[vi]));
            vp = mk(a.x, a.y, a.z);
            vd = mk(a.w, b.x, b.y);
        }
        sd_splat_warp(T, on, rad, vp, vd);
    }
}

__global__ void __launch_bounds__(kShadePPGThreads)
    k_shade_ppg(DevScene S, PathIO in, PathIO nxt, const float4* hit, RenderParams P, WaveCounters* ctr,
                unsigned long long* __restrict__ film, DevSDTree T, PPGVerts V, int* slot_stack) {
    after_previous();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = ctr->n_cur;
    if ((int)(blockIdx.x * blockDim.x) >= n) return;  // an empty CTA of the capacity's grid
    bool push_cont = false, release = false;
    float4 no, nd, nt;
    int4 ninfo;
    int slot = -1, n_splat = 0;  // vertices that take a splat (all of them, one per bounce, or none)
    f3 last = mk(0.f, 0.f, 0.f);  // the last one's factor
    if (i < n) {
        const float4 O = in.o[i], D = in.d[i], Tp = in.thr[i];
        const int4 I = in.info[i];
        const float4 H = hit[i];
        const int prim = __float_as_int(H.y);
        const int pixel = I.x, sample = I.y, bounce = I.z & 0xffff;
        slot = I.w;
        const int D_ = P.max_depth;
        f3 mul = mk(Tp.x, Tp.y, Tp.z);
        const f3 ro = mk(O.x, O.y, O.z), rd = mk(D.x, D.y, D.z);
        f3 vrad = mk(1.f, 1.f, 1.f);  // ppg.h:51-56: a vertex at the ray's origin with radiance 1
        bool done = true;
        if (prim < 0) {  // sky = 0 (ppg.h:57-63)
            vrad = mk(0.f, 0.f, 0.f);
        } else {
            int kind;
            DevMaterial m;
            const Surf s = make_surf(S, prim, ro, rd, H.x, H.z, H.w, bounce == 0, &kind, &m);
            const f3 wo = -rd;
            if (kind == PT_MAT_EMISSIVE_) {  // ppg.h:66-73
                const f3 rad = mk(m.r, m.g, m.b);
                vrad = rad;
                const f3 c = mul * rad;
                film_add_rgb(film, pixel, c.x, c.y, c.z, ctr);
            } else {
                const Rng4 r0 = rng4(P.seed, sample, pixel, bounce, 0);
                const Rng4 r1 = rng4(P.seed, sample, pixel, bounce, 1);
                BSample smp;
                float weight = 1.0f;
                bool ok = true;
                if (r0.v[0] > 0.5f) {  // ppg.h:76-81: BSDF sample
                    smp = bsdf_sample(m, s, wo, r0.v[1], r0.v[2]);
                    weight = smp.pdf / (smp.pdf + sd_pdf(T, s.p, smp.wi));
                } else {  // ppg.h:83-95: SD-tree sample
                    smp = sd_sample(T, s.p, r0.v[3], r1.v[0], r1.v[1]);
                    if (!same_hemisphere(s, wo, smp.wi)) ok = false;
                    else {
                        const float pb = bsdf_pdf(m, s, wo, smp.wi);
                        weight = smp.pdf / (smp.pdf + pb);
                    }
                }
                if (ok) {
                    float p = smp.pdf * 0.5f;
                    if (same_hemisphere(s, wo, smp.wi)) {  // ppg.h:105-107
                        const f3 f = bsdf_eval(m, s, wo, smp.wi);
                        bool alive = true;
                        if (bounce >= P.rr_start) {  // ppg.h:111-117
                            const float rr = russian_roulette(f);
                            if (r1.v[2] > rr) alive = false;
                            else p = p * rr;
                        }
                        if (alive) {
                            const f3 nm = f * (weight / p);
                            vrad = nm;
                            mul = mul * nm;
                            if (bounce + 1 < P.max_depth) {
                                done = false;
                                const f3 oo = s.p + smp.wi * kEps;
                                push_cont = true;
                                no = make_float4(oo.x, oo.y, oo.z, 1.f);
                                nd = make_float4(smp.wi.x, smp.wi.y, smp.wi.z, 0.f);
                                nt = make_float4(mul.x, mul.y, mul.z, 0.f);
                                ninfo = make_int4(pixel, sample, bounce + 1, slot);
                            }
                        }
                    }
                }
            }
        }
        if (bounce > 0) {
            const size_t vi = (size_t)slot * D_ + (bounce - 1);
            V.vp[vi] = make_float4(ro.x, ro.y, ro.z, rd.x);
            V.vd[vi] = make_float4(rd.y, rd.z, vrad.x, vrad.y);
            V.vr[vi] = vrad.z;
        }
        release = done;
        // ppg.h:131-141: splats only when the last vertex carries radiance
        if (done && (vrad.x > 0.f || vrad.y > 0.f || vrad.z > 0.f)) {
            n_splat = bounce;
            last = vrad;
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kWarps = kShadePPGThreads / 32;
    splat_paths(T, V, P.max_depth, slot, n_splat, last);
    // one addition to each queue's counter per CTA (as k_shade)
    __shared__ int s_count[2][kWarps], s_base[2];
    const unsigned m_free = __ballot_sync(0xffffffffu, release), m_cont = __ballot_sync(0xffffffffu, push_cont);
    if (lane == 0) {
        s_count[0][warp] = __popc(m_free);
        s_count[1][warp] = __popc(m_cont);
    }
    __syncthreads();
    if (lane == 0 && warp < 2) {
        int total = 0;
        for (int w = 0; w < kWarps; w++) {
            const int q = s_count[warp][w];
            s_count[warp][w] = total;
            total += q;
        }
        if (total) s_base[warp] = atomicAdd(warp == 0 ? &ctr->free_top : &ctr->n_next, total);
    }
    __syncthreads();
    const unsigned below = (1u << lane) - 1u;
    if (release) slot_stack[s_base[0] + s_count[0][warp] + __popc(m_free & below)] = slot;
    if (push_cont) {
        const int jc = s_base[1] + s_count[1][warp] + __popc(m_cont & below);
        nxt.o[jc] = no;
        nxt.d[jc] = nd;
        nxt.thr[jc] = nt;
        nxt.info[jc] = ninfo;
    }
}

// The splats of paths that finished elsewhere: path i in slot i with n_verts[i]
// vertices recorded (checks of splat_paths).
__global__ void __launch_bounds__(kShadePPGThreads) k_debug_splat(DevSDTree T, PPGVerts V, const int* n_verts, int n,
                                                                  int max_depth) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    int n_splat = i < n ? n_verts[i] : 0;
    f3 last = mk(0.f, 0.f, 0.f);
    if (n_splat > 0) {
        const size_t vi = (size_t)i * max_depth + n_splat - 1;
        last = mk(V.vd[vi].z, V.vd[vi].w, V.vr[vi]);
        if (!(last.x > 0.f || last.y > 0.f || last.z > 0.f)) n_splat = 0;
    }
    splat_paths(T, V, max_depth, i, n_splat, last);
}

// Camera paths for PPG (ppg.h:174-186: one jittered sample per pixel per
// pass, no strata), each with a vertex slot from the free list.
__global__ void __launch_bounds__(256) k_generate_ppg(DevScene S, PathIO nxt, int capacity, RenderParams P,
                                                      WaveCounters* ctr, const int* slot_stack) {
    after_previous();
    const int n_next = ctr->n_next, free_top = ctr->free_top;
    const unsigned long long first = ctr->work_next, left = ctr->work_total - first;
    const int avail = min(capacity - n_next, free_top);
    const int count = left < (unsigned long long)avail ? (int)left : avail;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < count; t += gridDim.x * blockDim.x) {
        const unsigned long long w = first + (unsigned long long)t;
        const unsigned long long npix = (unsigned long long)P.width * P.height;
        const int sample = (int)(w / npix);
        const int pixel = (int)(w - (unsigned long long)sample * npix);
        const int px = pixel % P.width, py = pixel / P.width;
        const Rng4 r = rng4(P.seed, sample, pixel, 0xffffu, 2);
        const float cx = (((float)px + r.v[0]) / (float)P.width) * 2.0f - 1.0f;
        const float cy = -((((float)py + r.v[1]) / (float)P.height) * 2.0f - 1.0f);
        const DevCamera& C = S.cam;
        const float dx = cx * C.tan_fovy * C.aspect, dy = cy * C.tan_fovy, dz = -1.0f;
        const f3 d = normalized(mk(C.m[0] * dx + C.m[1] * dy + C.m[2] * dz, C.m[3] * dx + C.m[4] * dy + C.m[5] * dz,
                                   C.m[6] * dx + C.m[7] * dy + C.m[8] * dz));
        const int j = n_next + t;
        const int slot = slot_stack[free_top - 1 - t];
        nxt.o[j] = make_float4(C.o[0], C.o[1], C.o[2], 1.0f);
        nxt.d[j] = make_float4(d.x, d.y, d.z, 0.f);
        nxt.thr[j] = make_float4(1.f, 1.f, 1.f, 0.f);
        nxt.info[j] = make_int4(pixel, sample, 0, slot);
    }
}

__global__ void k_advance_ppg(WaveCounters* ctr, int capacity) {
    after_previous();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const int n_next = ctr->n_next;
    const unsigned long long left = ctr->work_total - ctr->work_next;
    unsigned long long room = (unsigned long long)(capacity - n_next);
    if ((unsigned long long)ctr->free_top < room) room = (unsigned long long)ctr->free_top;
    const unsigned long long added = left < room ? left : room;
    ctr->work_next += added;
    ctr->stat_paths += added;
    ctr->free_top -= (int)added;
    ctr->n_cur = n_next + (int)added;
    ctr->stat_closest += (unsigned long long)ctr->n_cur;
    ctr->n_next = 0;
    ctr->n_shadow = 0;
    ctr->fetch_ext = 0;
    ctr->fetch_sh = 0;
    ctr->stat_iters += 1;
}

__global__ void k_init_slots(int* slot_stack, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) slot_stack[i] = i;
}

void launch_init_slots(int* slot_stack, int n, cudaStream_t st) {
    k_init_slots<<<min((n + 255) / 256, 2048), 256, 0, st>>>(slot_stack, n);
}
void launch_shade_ppg(const DevScene& S, const PathBuffers& B, int cur, const RenderParams& P, WaveCounters* ctr,
                      unsigned long long* film, const DevSDTree& T, const PPGVerts& V, int* slot_stack,
                      cudaStream_t st) {
    launch_after(k_shade_ppg, (B.capacity + kShadePPGThreads - 1) / kShadePPGThreads, kShadePPGThreads, 0, st,
        S, path_io(B, cur), path_io(B, 1 - cur), B.hit, P, ctr, film, T, V, slot_stack);
}
void launch_debug_splat(const DevSDTree& T, const PPGVerts& V, const int* n_verts, int n, int max_depth,
                        cudaStream_t st) {
    k_debug_splat<<<(n + kShadePPGThreads - 1) / kShadePPGThreads, kShadePPGThreads, 0, st>>>(T, V, n_verts, n,
                                                                                             max_depth);
}
void launch_generate_ppg(const DevScene& S, const PathBuffers& B, int cur, const RenderParams& P, WaveCounters* ctr,
                         const int* slot_stack, int num_sms, cudaStream_t st) {
    // a resident grid over the free slots (as the plain wavefront's)
    launch_after(k_generate_ppg, max(1, min((B.capacity + 255) / 256, num_sms * 8)), 256, 0, st, S, path_io(B, 1 - cur),
                 B.capacity, P, ctr, slot_stack);
    launch_after(k_advance_ppg, 1, 32, 0, st, ctr, B.capacity);
}

}  // namespace cpppt_gb300
