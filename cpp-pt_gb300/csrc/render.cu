// CUDA kernels: ray-batch traversal and the wavefront PT+NEE+MIS integrator
// (PathtracerMIS::integrate/render, src/renderer/pathtracerMIS.h:29-167).
//
// Wavefront layout: path state lives in HBM as structure-of-arrays, two
// copies (current / next).  One iteration = trace (closest hit for every live
// path, then any hit for the shadow rays the iteration before queued, whose
// unoccluded NEE contributions go to the film) -> shade (emission + MIS, BSDF
// sample, NEE shadow ray, Russian roulette; survivors are appended compactly
// to the next buffer, one counter addition per CTA) -> generate (new camera
// paths fill the next buffer up to capacity from a global work counter) ->
// advance (one thread swaps counts).
// All sizes are read from device counters, so an iteration needs no host
// round trip and a chain of iterations is captured once in a CUDA graph.
#include <cuda_runtime.h>

#include <mutex>

#include "launch.cuh"
#include "kernels.h"
#include "shade.cuh"
#include "trace.cuh"

namespace cpppt_gb300 {

constexpr size_t kClosestSmem = trace_smem(true, false, kTraceThreads);
constexpr size_t kAnySmem = trace_smem(false, true, kTraceThreads);
constexpr size_t kBothSmem = trace_smem(true, true, kTraceThreads);
constexpr size_t kBothAnyWord = kClosestSmem / 4;  // the any-hit region of a kernel with both

__device__ __forceinline__ float4 shfl4(float4 v, int src) {
    return make_float4(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src),
                       __shfl_sync(0xffffffffu, v.z, src), __shfl_sync(0xffffffffu, v.w, src));
}

// ---------------------------------------------------------------------------
// Ray batches (BVH::intersect / intersect_any on arrays of rays)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kTraceThreads, kTraceBlocksPerSM)
    k_trace_closest(DevScene S, const float* __restrict__ rays, int n, float4* __restrict__ hits, int* counter,
                    uint32_t* status) {
    extern __shared__ __align__(16) uint32_t s_stack[];
    TraceCount cnt{0u, 0u};
    persistent_trace<false, false>(
        S, s_stack, n, counter, status, cnt,
        [&](int i, float3& o, float3& d, float& tmax, uint32_t& root) {
            const float* r = rays + 7 * (size_t)i;
            o = make_float3(r[0], r[1], r[2]);
            d = make_float3(r[3], r[4], r[5]);
            tmax = r[6];
        },
        [&](int i, const HitRec& h) { hits[i] = make_float4(h.t, __int_as_float(h.prim), h.beta, h.gamma); });
}

__global__ void __launch_bounds__(kTraceThreads, kTraceBlocksPerSM)
    k_trace_any(DevScene S, const float* __restrict__ rays, int n, uint8_t* __restrict__ occ, int* counter,
                uint32_t* status) {
    extern __shared__ __align__(16) uint32_t s_stack[];
    TraceCount cnt{0u, 0u};
    persistent_trace<true, false>(
        S, s_stack, n, counter, status, cnt,
        [&](int i, float3& o, float3& d, float& tmax, uint32_t& root) {
            const float* r = rays + 7 * (size_t)i;
            o = make_float3(r[0], r[1], r[2]);
            d = make_float3(r[3], r[4], r[5]);
            tmax = r[6];
        },
        [&](int i, const HitRec& h) { occ[i] = h.prim >= 0 ? 1 : 0; });
}

bool trace_needs_counter(int n, int num_sms) {
    return n > min(num_sms * kTraceBlocksPerSM, n) * (kTraceThreads / 32);
}

void launch_trace_closest(const DevScene& S, const float* rays, int n, float4* hits, int* counter, uint32_t* status,
                          int num_sms, cudaStream_t st) {
    if (n <= 0) return;
    const int blocks = min(num_sms * kTraceBlocksPerSM, n);
    k_trace_closest<<<blocks, kTraceThreads, kClosestSmem, st>>>(S, rays, n, hits, counter, status);
}

void launch_trace_any(const DevScene& S, const float* rays, int n, uint8_t* occ, int* counter, uint32_t* status,
                      int num_sms, cudaStream_t st) {
    if (n <= 0) return;
    const int blocks = min(num_sms * kTraceBlocksPerSM, n);
    k_trace_any<<<blocks, kTraceThreads, kAnySmem, st>>>(S, rays, n, occ, counter, status);
}

// ---------------------------------------------------------------------------
// Wavefront integrator
// ---------------------------------------------------------------------------
// Film (film_add_rgb, shade.cuh): the image does not depend on the order in
// which contributions arrive (bit-identical across schedules, batch sizes and
// launch shapes).  The final division by spp happens in FP64.
__device__ __forceinline__ void film_add(unsigned long long* film, size_t pix, float r, float g, float b,
                                         WaveCounters* ctr) {
    film_add_rgb(film, pix, r, g, b, ctr);
}

// The extension rays of a path buffer.
template <bool COUNT>
__device__ __forceinline__ void extend_queue(const DevScene& S, uint32_t* s_stack, const PathIO& in,
                                             float4* __restrict__ Hout, int n, WaveCounters* ctr, TraceCount& cnt) {
    const float4* O = in.o;
    const float4* D = in.d;
    persistent_trace<false, COUNT>(
        S, s_stack, n, &ctr->fetch_ext, &ctr->status, cnt,
        [&](int i, float3& o, float3& d, float& tmax, uint32_t& root) {
            const float4 a = O[i], b = D[i];
            o = make_float3(a.x, a.y, a.z);
            d = make_float3(b.x, b.y, b.z);
            tmax = __int_as_float(0x7f800000);
            if (root != kTravDone) root = __float_as_uint(b.w);  // the path's scene root (0 unbatched)
        },
        [&](int i, const HitRec& h) { Hout[i] = make_float4(h.t, __int_as_float(h.prim), h.beta, h.gamma); });
}

// The shadow rays of a queue; the unoccluded ones' contributions go to the film.
template <int THREADS>
__device__ __forceinline__ void shadow_queue(const DevScene& S, uint32_t* s_stack, const ShadowIO& Q, int n,
                                             WaveCounters* ctr, unsigned long long* __restrict__ film, bool own_first) {
    TraceCount cnt{0u, 0u};
    persistent_trace<true, false, THREADS>(
        S, s_stack, n, &ctr->fetch_sh, &ctr->status, cnt,
        [&](int i, float3& o, float3& d, float& tmax, uint32_t& root) {
            const float4 a = Q.o[i], b = Q.d[i];
            o = make_float3(a.x, a.y, a.z);
            d = make_float3(b.x, b.y, b.z);
            tmax = a.w;
            if (root != kTravDone) root = __float_as_uint(Q.c[i].w);
        },
        [&](int i, const HitRec& h) {
            if (h.prim < 0) {  // unoccluded: the NEE contribution reaches the film
                const float4 c = Q.c[i];
                film_add(film, (uint32_t)__float_as_int(Q.d[i].w), c.x, c.y, c.z, ctr);
            }
        },
        own_first);
}

template <bool COUNT>
__global__ void __launch_bounds__(kTraceThreads, kTraceBlocksPerSM)
    k_extend(DevScene S, PathIO in, float4* __restrict__ Hout, WaveCounters* ctr) {
    after_previous();
    extern __shared__ __align__(16) uint32_t s_stack[];
    const int n = ctr->n_cur;
    if (n == 0) return;  // drained wavefront
    TraceCount cnt{0u, 0u};
    extend_queue<COUNT>(S, s_stack, in, Hout, n, ctr, cnt);
    if (COUNT) {
        const unsigned nodes = __reduce_add_sync(0xffffffffu, cnt.nodes);
        const unsigned tris = __reduce_add_sync(0xffffffffu, cnt.tris);
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(&ctr->stat_nodes, (unsigned long long)nodes);
            atomicAdd(&ctr->stat_tris, (unsigned long long)tris);
        }
    }
}

__global__ void __launch_bounds__(kTraceThreads, kTraceBlocksPerSM)
    k_shadow(DevScene S, ShadowIO Q, int cur, WaveCounters* ctr, unsigned long long* __restrict__ film) {
    extern __shared__ __align__(16) uint32_t s_stack[];
    const int n = cur ? ctr->n_shadow1 : ctr->n_shadow;
    if (n == 0) return;
    shadow_queue<kTraceThreads>(S, s_stack, Q, n, ctr, film, true);
}

// One wavefront iteration's rays: the extension rays of path buffer `in`,
// then the shadow rays that the iteration before queued (those of the other
// buffer; film additions are exact integers, so the image does not depend on
// when they arrive).  A warp that finds no extension ray left goes on with
// the shadow rays, so the launch has one tail of long rays instead of two:
// measured (1M-triangle soup) 640x360 at 1 spp 2.9 -> 2.4
// ms, 1920x1080 at 16 spp 106.3 -> 98.8 ms together with k_generate's grid;
// the Cornell box at 256x256, 64 spp 6.1 -> 4.75 ms (same images).
__global__ void __launch_bounds__(kTraceThreads, kTraceBlocksPerSM)
    k_trace_wave(DevScene S, PathIO in, float4* __restrict__ Hout, ShadowIO Q, int cur, WaveCounters* ctr,
                 unsigned long long* __restrict__ film) {
    after_previous();
    extern __shared__ __align__(16) uint32_t s_stack[];
    const int n = ctr->n_cur, m = cur ? ctr->n_shadow : ctr->n_shadow1;
    if (n == 0 && m == 0) return;
    TraceCount cnt{0u, 0u};
    if (n > 0) extend_queue<false>(S, s_stack, in, Hout, n, ctr, cnt);
    if (m > 0) shadow_queue<kTraceThreads>(S, s_stack + kBothAnyWord, Q, m, ctr, film, n == 0);
}

// info.w is the path's job: its table entry holds the render parameters,
// the scene's light list inside the arena and the job's film offset.  A
// single-scene render is a table of one job (so batched and single renders
// run the same instructions and give bit-identical images).
// Resident CTAs of 256 threads per SM for the shading kernel.  Measured on
// the 1M-triangle soup at 1080p, 64 spp, 2^24 paths in flight: 2 (128
// registers) 333.4 Mpaths/s, 3 (80 registers) 341.5, 4 (64 registers, some
// spilling) 345.1.
#ifndef CPPPT_SHADE_BLOCKS
#define CPPPT_SHADE_BLOCKS 4
#endif
// What shading a path's vertex leaves: a shadow ray, the continued path.
struct ShadeOut {
    bool push_sh, push_cont;
    float4 sh_o, sh_d, sh_c;
    float4 o, d, thr;
    int4 info;
};

// One vertex of a path (PathtracerMIS::integrate's loop body): emission with
// its MIS weight, BSDF sample, next-event estimation, Russian roulette.
__device__ __forceinline__ void shade_vertex(DevScene S, const DevBatchJob* __restrict__ jobs, float4 O, float4 D,
                                             float4 T, int4 I, float4 H, WaveCounters* ctr,
                                             unsigned long long* __restrict__ film, ShadeOut& out) {
    out.push_sh = out.push_cont = false;
    const int prim = __float_as_int(H.y);
    const int pixel = I.x, sample = I.y, bounce = I.z & 0xffff;
    const bool sdelta = (I.z >> 16) & 1;
    const DevBatchJob* J = jobs + I.w;
    const int integrator = J->integrator;
    const uint32_t seed = J->seed;
    const int rr_start = J->rr_start, max_depth = J->max_depth;
    const size_t fpix = (size_t)(uint32_t)pixel + J->film_off;
    S.light_prim += J->light_off;
    S.light_area += J->light_off;
    S.n_lights = J->n_lights;
    float p = O.w;
    f3 mul = mk(T.x, T.y, T.z);
    const f3 ro = mk(O.x, O.y, O.z), rd = mk(D.x, D.y, D.z);
    if (prim >= 0) {  // a miss adds render_sky = 0 (pathtracerMIS.h:38-41)
        int kind;
        DevMaterial m;
        const Surf s = make_surf(S, prim, ro, rd, H.x, H.z, H.w, bounce == 0, &kind, &m);
        const f3 wo = -rd;
        if (kind == PT_MAT_EMISSIVE_) {  // pathtracerMIS.h:43-67: emitters end the path
            float w = 1.0f;
            if (!sdelta && integrator == kIntegratorNEE) {
                w = 0.0f;  // pathtracer.h:41-46: NEE already counted this emitter
            } else if (!sdelta && integrator == kIntegratorMIS) {
                const int4 vi = __ldg(S.tri_vidx + prim);
                const f3 a = f3of(__ldg(S.v_pos + vi.x)), b = f3of(__ldg(S.v_pos + vi.y)),
                         c = f3of(__ldg(S.v_pos + vi.z));
                const float area = length(cross(b - a, c - a)) * 0.5f;
                const float pdf_l = (1.0f / (float)S.n_lights) * (1.0f / area);
                const float r = H.x;
                const float cos_theta = fabsf(dot(s.n, rd)) + kEps;
                const float p_nee = pdf_l * r * r / cos_theta;
                w = p / (p + p_nee);
            }
            film_add(film, fpix, mul.x * m.r * w, mul.y * m.g * w, mul.z * m.b * w, ctr);
        } else {
            const Rng4 r0 = rng4(seed, sample, pixel, bounce, 0);
            const Rng4 r1 = rng4(seed, sample, pixel, bounce, 1);
            const BSample bs = bsdf_sample(m, s, wo, r0.v[0], r0.v[1]);
            p = bs.pdf;
            if (!bs.delta && S.n_lights > 0 && integrator != kIntegratorPT) {  // NEE, pathtracerMIS.h:79-106
                const LSample ls = sample_light(S, s.p, r0.v[2], r0.v[3], r1.v[0]);
                f3 sd = ls.pos - s.p;
                const float len = length(sd);
                sd = sd * (1.0f / len);
                if (same_hemisphere(s, wo, sd)) {
                    const float pb = bsdf_pdf(m, s, wo, sd);
                    const float cosl = fabsf(dot(ls.n, sd)) + kEps;
                    const float pn = ls.pdf * len * len / cosl;
                    const float w = integrator == kIntegratorMIS ? pn / (pb + pn) : 1.0f;
                    const f3 f = bsdf_eval(m, s, wo, sd);
                    const f3 c = mul * f * ls.le * (1.0f / (ls.pdf * len * len)) * w;
                    if (c.x != 0.f || c.y != 0.f || c.z != 0.f) {
                        out.push_sh = true;
                        const f3 so = s.p + sd * kEps;
                        out.sh_o = make_float4(so.x, so.y, so.z, len - 2.0f * kEps);
                        out.sh_d = make_float4(sd.x, sd.y, sd.z, __int_as_float((int)(uint32_t)fpix));
                        out.sh_c = make_float4(c.x, c.y, c.z, D.w);  // w: the scene root
                    }
                }
            }
            if (same_hemisphere(s, wo, bs.wi)) {  // pathtracerMIS.h:112-126
                const f3 f = bsdf_eval(m, s, wo, bs.wi);
                bool alive = true;
                if (bounce >= rr_start) {
                    const float rr = russian_roulette(f);
                    if (r1.v[1] > rr) alive = false;
                    else p = p * rr;
                }
                if (alive && bounce + 1 < max_depth) {
                    mul = mul * f * (1.0f / p);
                    const f3 oo = s.p + bs.wi * kEps;
                    out.push_cont = true;
                    out.o = make_float4(oo.x, oo.y, oo.z, p);
                    out.d = make_float4(bs.wi.x, bs.wi.y, bs.wi.z, D.w);
                    out.thr = make_float4(mul.x, mul.y, mul.z, 0.f);
                    out.info = make_int4(pixel, sample, (bounce + 1) | ((bs.delta ? 1 : 0) << 16), I.w);
                }
            }
        }
    }
}

constexpr int kShadeThreads = 256;
__global__ void __launch_bounds__(kShadeThreads, CPPPT_SHADE_BLOCKS)
    k_shade(DevScene S, PathIO in, PathIO nxt, ShadowIO Q, const float4* hit, int cur, WaveCounters* ctr,
            unsigned long long* __restrict__ film, const DevBatchJob* __restrict__ jobs) {
    after_previous();
    const int n = ctr->n_cur;
    // an empty CTA of the capacity's grid: nothing to shade, no barriers to
    // wait at (Cornell box, 256x256, 64 spp, 3.65 -> 3.57 ms)
    if ((int)(blockIdx.x * blockDim.x) >= n) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    ShadeOut out;
    out.push_sh = out.push_cont = false;
    if (i < n) shade_vertex(S, jobs, in.o[i], in.d[i], in.thr[i], in.info[i], hit[i], ctr, film, out);
    // One addition to each queue's counter per CTA (a warp's position comes
    // from the counts of the warps before it): with one per warp every warp
    // waited on two contended atomics.  Cornell box, 256x256, 64 spp, 4.03 ->
    // 3.64 ms; the soups, whose shading waits on scattered loads, unchanged
    // (CTAs of 128: 3.66 ms and 1080p 1 % slower; of 512: 3.73 ms).
    __shared__ int s_count[2][kShadeThreads / 32], s_base[2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned m_sh = __ballot_sync(0xffffffffu, out.push_sh), m_cont = __ballot_sync(0xffffffffu, out.push_cont);
    if (lane == 0) {
        s_count[0][warp] = __popc(m_sh);
        s_count[1][warp] = __popc(m_cont);
    }
    __syncthreads();
    if (lane == 0 && warp < 2) {
        int total = 0;
        for (int w = 0; w < kShadeThreads / 32; w++) {
            const int c = s_count[warp][w];
            s_count[warp][w] = total;
            total += c;
        }
        int* counter = warp == 1 ? &ctr->n_next : (cur ? &ctr->n_shadow1 : &ctr->n_shadow);
        if (total) s_base[warp] = atomicAdd(counter, total);
    }
    __syncthreads();
    const unsigned below = (1u << lane) - 1u;
    if (out.push_sh) {
        const int js = s_base[0] + s_count[0][warp] + __popc(m_sh & below);
        Q.o[js] = out.sh_o;
        Q.d[js] = out.sh_d;
        Q.c[js] = out.sh_c;
    }
    if (out.push_cont) {
        const int jc = s_base[1] + s_count[1][warp] + __popc(m_cont & below);
        nxt.o[jc] = out.o;
        nxt.d[jc] = out.d;
        nxt.thr[jc] = out.thr;
        nxt.info[jc] = out.info;
    }
}

// Index of the job whose work range holds w (job work ranges ascend).
__device__ __forceinline__ int find_job(const DevBatchJob* __restrict__ jobs, int n_jobs, unsigned long long w) {
    int lo = 0, hi = n_jobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&jobs[mid].work_begin) <= w) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// New camera paths for the free slots of the next buffer; work index w
// (global over the jobs' pixel x sample ranges) selects job, sample, pixel.
__global__ void __launch_bounds__(256) k_generate(PathIO nxt, int capacity, WaveCounters* ctr,
                                                  const DevBatchJob* __restrict__ jobs, int n_jobs) {
    after_previous();
    const int n_next = ctr->n_next;
    const unsigned long long first = ctr->work_next, left = ctr->work_total - first;
    const int room = capacity - n_next;
    const int count = left < (unsigned long long)room ? (int)left : room;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < count; t += gridDim.x * blockDim.x) {
        unsigned long long w = first + (unsigned long long)t;
        const int job = n_jobs > 1 ? find_job(jobs, n_jobs, w) : 0;
        const DevBatchJob* J = jobs + job;
        w -= J->work_begin;
        const DevCamera* C = &J->cam;
        const int width = C->width, height = C->height, spp_axis = J->spp_axis;
        const uint32_t seed = J->seed, root = J->root;
        const unsigned long long npix = (unsigned long long)width * height;
        const int sample = (int)(w / npix);
        int pixel = (int)(w - (unsigned long long)sample * npix);
        {  // visit the pass in tiles (a bijection of the pixels; the RNG is keyed by pixel, not by order)
            const int tw = J->tile_w, th = J->tile_h;
            if (tw * th > 1) {
                const int tile = pixel / (tw * th), r = pixel - tile * (tw * th);
                const int tiles_x = width / tw;
                const int ty = tile / tiles_x, tx = tile - ty * tiles_x;
                pixel = (ty * th + r / tw) * width + tx * tw + r % tw;
            }
        }
        const int px = pixel % width, py = pixel / width;
        const Rng4 r = rng4(seed, sample, pixel, 0xffffu, 2);
        float cx, cy;
        if (spp_axis > 0) {  // pathtracerMIS.h:148-153: spp x spp strata
            const int k = sample / spp_axis, l = sample - (sample / spp_axis) * spp_axis;
            cx = (((float)px + ((float)k + r.v[0]) / (float)spp_axis) / (float)width) * 2.0f - 1.0f;
            cy = -((((float)py + ((float)l + r.v[1]) / (float)spp_axis) / (float)height) * 2.0f - 1.0f);
        } else {
            cx = (((float)px + r.v[0]) / (float)width) * 2.0f - 1.0f;
            cy = -((((float)py + r.v[1]) / (float)height) * 2.0f - 1.0f);
        }
        // CameraPerspective::get_ray (camera_perspective.h:30-39)
        const float dx = cx * C->tan_fovy * C->aspect, dy = cy * C->tan_fovy, dz = -1.0f;
        const f3 d = normalized(mk(C->m[0] * dx + C->m[1] * dy + C->m[2] * dz, C->m[3] * dx + C->m[4] * dy + C->m[5] * dz,
                                   C->m[6] * dx + C->m[7] * dy + C->m[8] * dz));
        const int j = n_next + t;
        nxt.o[j] = make_float4(C->o[0], C->o[1], C->o[2], 1.0f);
        nxt.d[j] = make_float4(d.x, d.y, d.z, __uint_as_float(root));
        nxt.thr[j] = make_float4(1.f, 1.f, 1.f, 0.f);
        nxt.info[j] = make_int4(pixel, sample, 0 | (1 << 16), job);  // sampled_delta starts true (:34)
    }
}

// Counters at the end of an iteration that read path buffer `cur`.  traced: the
// buffer whose shadow rays have been traced by now (the other one in
// k_trace_wave's order).  Once no work is left, the last finish_max paths are
// handed to k_finish and the wavefront has none.
__global__ void k_advance(WaveCounters* ctr, int capacity, int cur, int traced, int finish_max) {
    after_previous();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const int n_next = ctr->n_next;
    const unsigned long long left = ctr->work_total - ctr->work_next;
    const unsigned long long room = (unsigned long long)(capacity - n_next);
    const unsigned long long added = left < room ? left : room;
    ctr->work_next += added;
    ctr->stat_paths += added;
    ctr->stat_shadow += (unsigned long long)(cur ? ctr->n_shadow1 : ctr->n_shadow);
    int n_cur = n_next + (int)added;
    if (n_cur > 0 && n_cur <= finish_max && added == left) {
        ctr->n_finish = n_cur;
        ctr->finish_buf = 1 - cur;
        n_cur = 0;
    }
    ctr->n_cur = n_cur;
    ctr->stat_closest += (unsigned long long)n_cur;
    ctr->n_next = 0;
    (traced ? ctr->n_shadow1 : ctr->n_shadow) = 0;
    ctr->fetch_ext = 0;
    ctr->fetch_sh = 0;
    ctr->stat_iters += 1;
}

// ---------------------------------------------------------------------------
// The last paths of a render, each to its end in one launch.
//
// With few paths left an iteration takes as long as its slowest ray (a chain
// of dependent node loads) plus the launches, whatever their number, and a
// render has up to max_depth such iterations.  Here a path does not wait for
// the others: each warp takes up to 16 paths, one per lane of its lower half,
// and steps them vertex by vertex; the upper half traces the shadow rays of
// the vertex before in the same traversal loop.  Same functions, same random
// numbers and integer film as the wavefront, so the image is the same.
// First the shadow rays of the wavefront's last iteration are traced.
// ---------------------------------------------------------------------------
// Bound by the latency of its rays' node loads.  Measured (1M-triangle soup,
// 640x360, 1 spp, 230,400 paths) for the last 16k, 32k, 64k and 128k paths:
// 2285, 2234, 2186 and 2231 us against 2441 us without it; the batch of eight
// soups 29.35 -> 29.09 ms; the Cornell box and 1080p renders unchanged (their
// last 64k paths are a small part).  512 threads per SM with 128 registers;
// 1024 with 64 (spilling) 2262 us, two CTAs of 256 2190 us.
constexpr int kFinishThreads = 512;
constexpr size_t kFinishSmem = trace_smem(true, true, kFinishThreads);
constexpr size_t kFinishAnyWord = trace_smem(true, false, kFinishThreads) / 4;
__global__ void __launch_bounds__(kFinishThreads, 1) k_finish(
    DevScene S, PathIO b0, PathIO b1, ShadowIO Q, WaveCounters* ctr, unsigned long long* __restrict__ film,
    const DevBatchJob* __restrict__ jobs) {
    after_previous();
    const unsigned full = 0xffffffffu;
    const int m = ctr->n_shadow + ctr->n_shadow1;  // at most one of them is non-zero
    extern __shared__ __align__(16) uint32_t s_stack[];
    if (m > 0) shadow_queue<kFinishThreads>(S, s_stack + kFinishAnyWord, Q, m, ctr, film, true);
    const int n = ctr->n_finish;
    if (n == 0) return;
    const PathIO in = ctr->finish_buf ? b1 : b0;
    const int lane = threadIdx.x & 31, low = lane & 15;
    const int nwarps = (int)(gridDim.x * (blockDim.x >> 5));
    const int c0 = ray_chunk(n, nwarps, 1);
    int pool_next = min((int)((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * c0, n);
    int pool_end = min(pool_next + c0, n);
    bool exhausted = nwarps * c0 >= n;
    // lower half: a path; upper half: the shadow ray of the path 16 lanes below
    bool alive = false, pending = false;
    float4 O, D, C;
    int4 I;
    O = D = C = make_float4(0.f, 0.f, 0.f, 0.f);
    I = make_int4(0, 0, 0, 0);
    unsigned n_closest = 0, n_shadow = 0;
    int passes = 0;
    TravStack<false, kFinishThreads> K(s_stack, S.stack_limit);
    while (true) {
        const unsigned idle = __ballot_sync(full, lane < 16 && !alive);
        if (idle) {
            if (pool_next >= pool_end && !exhausted) {
                const int chunk = ray_chunk(n - pool_end, nwarps, 2);
                int base = 0;
                if (lane == 0) base = atomicAdd(&ctr->fetch_ext, chunk);
                base = __shfl_sync(full, base, 0) + nwarps * c0;
                pool_next = base;
                pool_end = min(base + chunk, n);
                if (base + chunk >= n) exhausted = true;
            }
            const int avail = max(0, pool_end - pool_next);
            const int r = __popc(idle & ((1u << lane) - 1u));
            if (lane < 16 && !alive && r < avail) {
                const int i = pool_next + r;
                O = in.o[i];
                D = in.d[i];
                C = in.thr[i];
                I = in.info[i];
                alive = true;
            }
            pool_next += min(avail, __popc(idle));
        }
        const unsigned live = __ballot_sync(full, alive);
        if (__ballot_sync(full, alive || pending) == 0) break;
        passes++;
        n_closest += __popc(live);
        Trav T;
        trav_init(T, K.base, make_float3(O.x, O.y, O.z), make_float3(D.x, D.y, D.z),
                  pending ? O.w : __int_as_float(0x7f800000),
                  S.n_tris > 0 ? __float_as_uint(pending ? C.w : D.w) : kTravDone);
        warp_trace(S, T, K, alive || pending, pending, &ctr->status);
        if (pending && T.best.prim < 0)
            film_add(film, (uint32_t)__float_as_int(D.w), C.x, C.y, C.z, ctr);
        ShadeOut out;
        out.push_sh = out.push_cont = false;
        if (alive)
            shade_vertex(S, jobs, O, D, C, I,
                         make_float4(T.best.t, __int_as_float(T.best.prim), T.best.beta, T.best.gamma), ctr, film, out);
        const unsigned push = __ballot_sync(full, out.push_sh);
        n_shadow += __popc(push);
        alive = out.push_cont;
        pending = lane >= 16 && ((push >> low) & 1u);
        const float4 so = shfl4(out.sh_o, low), sd = shfl4(out.sh_d, low), sc = shfl4(out.sh_c, low);
        if (lane >= 16) {
            O = so;
            D = sd;
            C = sc;
        } else {
            O = out.o;
            D = out.d;
            C = out.thr;
            I = out.info;
        }
    }
    if (lane == 0 && passes > 0) {
        atomicAdd(&ctr->stat_closest, (unsigned long long)n_closest);
        atomicAdd(&ctr->stat_shadow, (unsigned long long)n_shadow);
        atomicMax(&ctr->n_next, passes);  // read by the host as iterations
    }
}

__global__ void k_resolve(const unsigned long long* __restrict__ film, float* __restrict__ out, int n, double scale) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = (float)((double)(long long)film[i] * scale);
}

void launch_extend(const DevScene& S, const PathBuffers& B, int cur, WaveCounters* ctr, int num_sms, cudaStream_t st,
                   bool count) {
    const int g = num_sms * kTraceBlocksPerSM;
    if (count) launch_after(k_extend<true>, g, kTraceThreads, kClosestSmem, st, S, path_io(B, cur), B.hit, ctr);
    else launch_after(k_extend<false>, g, kTraceThreads, kClosestSmem, st, S, path_io(B, cur), B.hit, ctr);
}
void launch_trace_wave(const DevScene& S, const PathBuffers& B, int cur, WaveCounters* ctr, unsigned long long* film,
                       int num_sms, cudaStream_t st) {
    launch_after(k_trace_wave, num_sms * kTraceBlocksPerSM, kTraceThreads, kBothSmem, st, S, path_io(B, cur), B.hit,
                 shadow_io(B), cur, ctr, film);
}
cudaError_t trace_kernels_setup() {
    const auto limit = [](const void* f, size_t bytes) {
        return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    cudaError_t e = limit((const void*)k_trace_closest, kClosestSmem);
    if (e == cudaSuccess) e = limit((const void*)k_trace_any, kAnySmem);
    if (e == cudaSuccess) e = limit((const void*)k_extend<true>, kClosestSmem);
    if (e == cudaSuccess) e = limit((const void*)k_extend<false>, kClosestSmem);
    if (e == cudaSuccess) e = limit((const void*)k_shadow, kAnySmem);
    if (e == cudaSuccess) e = limit((const void*)k_trace_wave, kBothSmem);
    if (e == cudaSuccess) e = limit((const void*)k_finish, kFinishSmem);
    return e;
}

void launch_shade(const DevScene& S, const PathBuffers& B, int cur, WaveCounters* ctr, unsigned long long* film,
                  const DevBatchJob* jobs, cudaStream_t st) {
    launch_after(k_shade, (B.capacity + kShadeThreads - 1) / kShadeThreads, kShadeThreads, 0, st, S, path_io(B, cur),
                 path_io(B, 1 - cur), shadow_io(B), B.hit, cur, ctr, film, jobs);
}
void launch_shadow(const DevScene& S, const PathBuffers& B, int cur, WaveCounters* ctr, unsigned long long* film,
                   int num_sms, cudaStream_t st) {
    k_shadow<<<num_sms * kTraceBlocksPerSM, kTraceThreads, kAnySmem, st>>>(S, shadow_io(B), cur, ctr, film);
}
void launch_generate(const PathBuffers& B, int cur, WaveCounters* ctr, const DevBatchJob* jobs, int n_jobs, int num_sms,
                     cudaStream_t st, bool shadows_traced) {
    // a resident grid that strides over the free slots: most iterations have
    // few of them or none, and a CTA per 256 slots of the capacity cost up to
    // 50 us a launch there (a quarter of the Cornell box's 64-spp render)
    const int g = max(1, min((B.capacity + 255) / 256, num_sms * 8));
    launch_after(k_generate, g, 256, 0, st, path_io(B, 1 - cur), B.capacity, ctr, jobs, n_jobs);
    launch_after(k_advance, 1, 32, 0, st, ctr, B.capacity, cur, shadows_traced ? cur : 1 - cur,
                 shadows_traced ? 0 : kFinishPaths);
}
void launch_advance(WaveCounters* ctr, int capacity, int cur, cudaStream_t st) {
    launch_after(k_advance, 1, 32, 0, st, ctr, capacity, cur, 1 - cur, 0);
}
void launch_wave_iteration(const DevScene& S, const PathBuffers& B, int cur, WaveCounters* ctr, unsigned long long* film,
                           const DevBatchJob* jobs, int n_jobs, int num_sms, cudaStream_t st) {
    launch_trace_wave(S, B, cur, ctr, film, num_sms, st);
    launch_shade(S, B, cur, ctr, film, jobs, st);
    launch_generate(B, cur, ctr, jobs, n_jobs, num_sms, st, false);
}

void launch_finish(const DevScene& S, const PathBuffers& B, WaveCounters* ctr, unsigned long long* film,
                   const DevBatchJob* jobs, int num_sms, cudaStream_t st) {
    launch_after(k_finish, num_sms, kFinishThreads, kFinishSmem, st, S, path_io(B, 0), path_io(B, 1), shadow_io(B),
                 ctr, film, jobs);
}

// Body end of a device-driven render loop (build_render_graph).  One thread.
__global__ void k_round_control(WaveCounters* ctr, cudaGraphConditionalHandle h) {
    const uint32_t r = ctr->rounds + 1u;
    ctr->rounds = r;
    bool more = !(ctr->n_cur == 0 && ctr->work_next >= ctr->work_total) && ctr->status == 0u;
    if (more && r >= ctr->max_rounds) {
        ctr->status |= kStatusRoundLimit;
        more = false;
    }
    cudaGraphSetConditional(h, more ? 1u : 0u);
}

cudaError_t build_render_graph(const DevScene& S, const PathBuffers& B, WaveCounters* ctr, unsigned long long* film,
                               const DevBatchJob* jobs, int n_jobs, int iters, int num_sms, cudaStream_t st,
                               cudaGraphExec_t* out) {
    *out = nullptr;
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaGraphCreate(&g, 0);
    if (e != cudaSuccess) return e;
    cudaGraphConditionalHandle h;
    e = cudaGraphConditionalHandleCreate(&h, g, 1u, cudaGraphCondAssignDefault);
    cudaGraphNodeParams cp = {};
    if (e == cudaSuccess) {
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = h;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        cudaGraphNode_t node;
        e = cudaGraphAddNode(&node, g, nullptr, nullptr, 0, &cp);
    }
    if (e == cudaSuccess) {
        cudaGraph_t body = cp.conditional.phGraph_out[0];
        e = cudaStreamBeginCaptureToGraph(st, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            for (int k = 0; k < iters; k++)
                launch_wave_iteration(S, B, k & 1, ctr, film, jobs, n_jobs, num_sms, st);
            k_round_control<<<1, 1, 0, st>>>(ctr, h);
            cudaGraph_t captured = nullptr;
            const cudaError_t e2 = cudaStreamEndCapture(st, &captured);
            e = e2 != cudaSuccess ? e2 : cudaGetLastError();
        }
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(out, g, 0);
    cudaGraphDestroy(g);
    return e;
}

DevBatchJob single_job(const DevScene& S, const RenderParams& P) {
    DevBatchJob j{};
    j.cam = S.cam;
    j.work_begin = 0;
    j.film_off = 0;
    j.root = S.n_tris > 0 ? 0u : kTravDone;
    j.light_off = 0;
    j.n_lights = S.n_lights;
    j.spp = P.spp;
    j.spp_axis = P.spp_axis;
    j.max_depth = P.max_depth;
    j.rr_start = P.rr_start;
    j.seed = P.seed;
    j.tile_w = 1;
    j.tile_h = 1;
    j.integrator = kIntegratorMIS;
    return j;
}
void launch_film_resolve(const unsigned long long* film, float* out, int n, double scale, cudaStream_t st) {
    k_resolve<<<min((n + 255) / 256, 4096), 256, 0, st>>>(film, out, n, scale * (1.0 / 4294967296.0));
}

// ---------------------------------------------------------------------------
// Unit-test kernels: the integrator's own BxDF and light-sampling functions
// (shade.cuh) on cases given by the host, one case per thread
// (pt_debug_bsdf, pt_debug_light_sample).
// ---------------------------------------------------------------------------
__global__ void k_debug_bsdf(const float* __restrict__ in, float* __restrict__ out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* c = in + (size_t)kDebugBsdfIn * i;
    DevMaterial m{};
    m.kind = (int32_t)c[0];
    m.r = c[1];
    m.g = c[2];
    m.b = c[3];
    m.alpha = fmaxf(c[4] * c[4], 0.01f);  // glossy_bxdf.h:77-79, as the scene upload sets it
    m.delta = (double)c[4] < 0.01 ? 1 : 0;
    m.ior = c[5];
    m.tex = kNoTextures;
    // The frame make_surf builds at a path's first hit on a flat triangle
    // whose vertices carry normal N and tangent T (bitangent N x T,
    // loader.h:237), then re-orthogonalised (standard_material.h:64-71).
    Surf s;
    s.p = mk(0.f, 0.f, 0.f);
    s.mat = 0;
    s.n = normalized(mk(c[6], c[7], c[8]));
    s.ng = s.n;
    s.b = normalized(cross(s.n, mk(c[9], c[10], c[11])));
    s.t = normalized(cross(s.b, s.n));
    if (m.kind == PT_MAT_DIFFUSE_ || m.kind == PT_MAT_GGX_) s.n = normalized(s.n);
    s.b = normalized(cross(s.n, s.t));
    s.t = normalized(cross(s.b, s.n));
    const f3 wo = mk(c[12], c[13], c[14]), wi = mk(c[15], c[16], c[17]);
    const f3 ev = bsdf_eval(m, s, wo, wi);
    const BSample b = bsdf_sample(m, s, wo, c[18], c[19]);
    float* o = out + (size_t)kDebugBsdfOut * i;
    o[0] = ev.x;
    o[1] = ev.y;
    o[2] = ev.z;
    o[3] = bsdf_pdf(m, s, wo, wi);
    o[4] = same_hemisphere(s, wo, wi) ? 1.f : 0.f;
    o[5] = b.wi.x;
    o[6] = b.wi.y;
    o[7] = b.wi.z;
    o[8] = b.pdf;
    o[9] = b.delta ? 1.f : 0.f;
}

__global__ void k_debug_light(DevScene S, const float* __restrict__ in, float* __restrict__ out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* c = in + (size_t)kDebugLightIn * i;
    const LSample l = sample_light(S, mk(c[0], c[1], c[2]), c[3], c[4], c[5]);
    float* o = out + (size_t)kDebugLightOut * i;
    o[0] = l.pos.x; o[1] = l.pos.y; o[2] = l.pos.z;
    o[3] = l.n.x; o[4] = l.n.y; o[5] = l.n.z;
    o[6] = l.le.x; o[7] = l.le.y; o[8] = l.le.z;
    o[9] = l.pdf;
}

void launch_debug_bsdf(const float* in, float* out, int n, cudaStream_t st) {
    if (n > 0) k_debug_bsdf<<<(n + 127) / 128, 128, 0, st>>>(in, out, n);
}
void launch_debug_light(const DevScene& S, const float* in, float* out, int n, cudaStream_t st) {
    if (n > 0) k_debug_light<<<(n + 127) / 128, 128, 0, st>>>(S, in, out, n);
}

// ---------------------------------------------------------------------------
// Allocation-free render (pt_render_device_noalloc)
//
// For callers that cannot allocate device memory at render time: a host
// whose device memory is reserved up front by another allocator (a caching
// allocator or an engine's memory budget), or a frame loop that must not
// enter the driver's allocation path.  The host still polls the wavefront's
// counters between rounds of iterations.  The wavefront's scratch --
// path state, queues, film and counters -- lives in one file-scope
// __device__ array instead of per-scene buffers.  The array is part of this
// module, so every GPU that loads the library holds it until the process
// exits.  Capacity: kNoAllocPaths paths in flight, at most kNoAllocMaxPixels
// pixels.  Every call shares the array and leaves its contents behind; each
// call clears the film and counters first, and calls that overlap on the GPU
// (concurrent streams or threads) race on it.
// ---------------------------------------------------------------------------
constexpr int kNoAllocPaths = 1 << 16;
constexpr int kNoAllocMaxPixels = 1 << 18;  // e.g. 512 x 512
constexpr size_t kNoAllocPathBytes = (size_t)kNoAllocPaths * 16;  // one float4 / int4 array
constexpr size_t kNoAllocFilmOffset = 12 * kNoAllocPathBytes;
constexpr size_t kNoAllocCtrOffset = kNoAllocFilmOffset + (size_t)3 * kNoAllocMaxPixels * 8;
constexpr size_t kNoAllocJobOffset = kNoAllocCtrOffset + 256;
constexpr size_t kNoAllocBytes = kNoAllocJobOffset + 256;
static_assert(kNoAllocPaths >= kFinishPaths, "the first generate holds every path of a render without a wavefront loop");
static_assert(sizeof(WaveCounters) <= 256 && sizeof(DevBatchJob) <= 256, "scratch slots");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

namespace {
std::mutex g_noalloc_mutex;
void* g_noalloc_addr[128] = {};  // per device ordinal
}  // namespace

size_t noalloc_scratch_bytes() { return kNoAllocBytes; }
int noalloc_max_pixels() { return kNoAllocMaxPixels; }
int noalloc_paths() { return kNoAllocPaths; }

// Device address of the scratch array on the current device, looked up once
// per device (the host-side symbol is not a device address).
static cudaError_t noalloc_scratch(void** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 128) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_addr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_noalloc_addr[dev] = p;
    }
    *out = g_noalloc_addr[dev];
    return cudaSuccess;
}

cudaError_t render_noalloc(const DevScene& S, const RenderParams& P, int num_sms, int max_depth, float* d_out,
                           cudaStream_t st, WaveCounters* final_counters, int* limit_hit) {
    *limit_hit = 0;
    void* base = nullptr;
    cudaError_t e = noalloc_scratch(&base);
    if (e != cudaSuccess) return e;
    unsigned char* b = static_cast<unsigned char*>(base);
    PathBuffers B;
    for (int k = 0; k < 2; k++) {
        B.o[k] = reinterpret_cast<float4*>(b + (0 + k) * kNoAllocPathBytes);
        B.d[k] = reinterpret_cast<float4*>(b + (2 + k) * kNoAllocPathBytes);
        B.thr[k] = reinterpret_cast<float4*>(b + (4 + k) * kNoAllocPathBytes);
        B.info[k] = reinterpret_cast<int4*>(b + (6 + k) * kNoAllocPathBytes);
    }
    B.hit = reinterpret_cast<float4*>(b + 8 * kNoAllocPathBytes);
    B.sh_o = reinterpret_cast<float4*>(b + 9 * kNoAllocPathBytes);
    B.sh_d = reinterpret_cast<float4*>(b + 10 * kNoAllocPathBytes);
    B.sh_c = reinterpret_cast<float4*>(b + 11 * kNoAllocPathBytes);
    B.capacity = kNoAllocPaths;
    unsigned long long* film = reinterpret_cast<unsigned long long*>(b + kNoAllocFilmOffset);
    WaveCounters* ctr = reinterpret_cast<WaveCounters*>(b + kNoAllocCtrOffset);
    DevBatchJob* job = reinterpret_cast<DevBatchJob*>(b + kNoAllocJobOffset);
    const int film_n = 3 * P.width * P.height;
    const unsigned long long total = (unsigned long long)P.width * P.height * (unsigned long long)P.spp;
    e = cudaMemsetAsync(film, 0, sizeof(unsigned long long) * film_n, st);
    if (e != cudaSuccess) return e;
    WaveCounters init{};
    init.work_total = total;
    init.film_safe = film_safe_bound((double)P.spp * (2.0 * max_depth + 2.0));
    e = cudaMemcpyAsync(ctr, &init, sizeof(init), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    const DevBatchJob hjob = single_job(S, P);
    e = cudaMemcpyAsync(job, &hjob, sizeof(hjob), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    launch_generate(B, 1, ctr, job, 1, num_sms, st, false);
    const int iters = 16;
    const unsigned long long max_rounds =
        64 + (total / (unsigned long long)kNoAllocPaths + 2) * (unsigned long long)(max_depth + 2) * 4 / iters;
    WaveCounters h{};
    for (unsigned long long round = 0;; round++) {
        // a render of at most kFinishPaths paths goes straight to k_finish
        for (int k = 0; k < iters && total > (unsigned long long)kFinishPaths; k++)
            launch_wave_iteration(S, B, k & 1, ctr, film, job, 1, num_sms, st);
        e = cudaMemcpyAsync(&h, ctr, sizeof(h), cudaMemcpyDeviceToHost, st);
        if (e != cudaSuccess) return e;
        e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return e;
        if (h.status) break;
        if (h.n_cur == 0 && h.work_next >= h.work_total) {
            launch_finish(S, B, ctr, film, job, num_sms, st);
            e = cudaMemcpyAsync(&h, ctr, sizeof(h), cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            if (e != cudaSuccess) return e;
            break;
        }
        if (round > max_rounds) {
            *limit_hit = 1;
            break;
        }
    }
    *final_counters = h;
    if (h.status || *limit_hit) return cudaSuccess;
    launch_film_resolve(film, d_out, film_n, 1.0 / (double)P.spp, st);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(st);
}

}  // namespace cpppt_gb300
