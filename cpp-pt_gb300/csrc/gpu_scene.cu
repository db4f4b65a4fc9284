// A scene's device arrays, assembled on the device from the caller's arrays
// and the two trees.  One thread per triangle or vertex, a streaming pass
// each, bound by memory (130 MB for a million triangles).  As host loops, with
// the trees read back and the wider arrays sent, the same work took half of
// the scene creation: 192k-triangle room 16.5 -> 11.0 ms, 1M-triangle soup 53
// -> 22.8, Cornell box 2.1 -> 1.8.  The arithmetic has no fused multiply-adds.
#include <cmath>
#include <cstring>

#include "gpu_bvh.h"

namespace cpppt_gb300 {
namespace {

constexpr int kThreads = 256;

// Order-preserving key of a float; 0 is below every key of a number.
__device__ __forceinline__ uint32_t fkey(float v) {
    const uint32_t u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Vertex positions by triangle, the shading index {a, b, c, material}, and
// the bounds: key6 = maxima of ~key (lower) and key (upper) per axis, NaN
// coordinates left out.
__global__ void __launch_bounds__(kThreads) k_triangle_positions(const float* __restrict__ verts,
                                                                 const int32_t* __restrict__ tri,
                                                                 const int32_t* __restrict__ material, int n,
                                                                 float* __restrict__ tv, int4* __restrict__ vidx,
                                                                 uint32_t* __restrict__ key6) {
    __shared__ uint32_t skey[6];
    if (threadIdx.x < 6) skey[threadIdx.x] = 0;
    __syncthreads();
    uint32_t key[6] = {0, 0, 0, 0, 0, 0};
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        int id[3];
        for (int k = 0; k < 3; k++) {
            id[k] = tri[3 * (size_t)t + k];
            for (int a = 0; a < 3; a++) {
                const float x = verts[3 * (size_t)id[k] + a];
                tv[9 * (size_t)t + 3 * k + a] = x;
                if (x == x) {
                    key[a] = max(key[a], ~fkey(x));
                    key[3 + a] = max(key[3 + a], fkey(x));
                }
            }
        }
        vidx[t] = make_int4(id[0], id[1], id[2], material[t]);
    }
    for (int f = 0; f < 6; f++) {
        const uint32_t v = __reduce_max_sync(0xffffffffu, key[f]);
        if ((threadIdx.x & 31) == 0) atomicMax(skey + f, v);
    }
    __syncthreads();
    if (threadIdx.x < 6) atomicMax(key6 + threadIdx.x, skey[threadIdx.x]);
}

// Traversal triangles in leaf order: {a, rank}, {b - a, parent}, {c - a, prim}
// (edges: triangle.h:40-41).
__global__ void __launch_bounds__(kThreads) k_leaf_triangles(const float* __restrict__ tv,
                                                             const int32_t* __restrict__ order,
                                                             const int32_t* __restrict__ rank,
                                                             const int32_t* __restrict__ parent, int n,
                                                             float4* __restrict__ tris) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int p = order[k];
    float v[9];
    for (int j = 0; j < 9; j++) v[j] = tv[9 * (size_t)p + j];
    float4* o = tris + 3 * (size_t)k;
    o[0] = make_float4(v[0], v[1], v[2], __int_as_float(rank[p]));
    o[1] = make_float4(__fsub_rn(v[3], v[0]), __fsub_rn(v[4], v[1]), __fsub_rn(v[5], v[2]), __int_as_float(parent[p]));
    o[2] = make_float4(__fsub_rn(v[6], v[0]), __fsub_rn(v[7], v[1]), __fsub_rn(v[8], v[2]), __int_as_float(p));
}

__device__ __forceinline__ void cross_rn(const float* a, const float* b, float* o) {
    o[0] = __fsub_rn(__fmul_rn(a[1], b[2]), __fmul_rn(a[2], b[1]));
    o[1] = __fsub_rn(__fmul_rn(a[2], b[0]), __fmul_rn(a[0], b[2]));
    o[2] = __fsub_rn(__fmul_rn(a[0], b[1]), __fmul_rn(a[1], b[0]));
}

// Positions, normals and bitangents cross(normal, tangent) (loader.h:237); a
// vertex without a tangent takes some vector perpendicular to its normal.
__global__ void __launch_bounds__(kThreads) k_vertices(const float* __restrict__ verts, const float* __restrict__ nrms,
                                                       const float* __restrict__ tans, int n,
                                                       float4* __restrict__ vpos, float4* __restrict__ vnrm,
                                                       float4* __restrict__ vbt) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    const float* p = verts + 3 * (size_t)v;
    const float nr[3] = {nrms[3 * (size_t)v], nrms[3 * (size_t)v + 1], nrms[3 * (size_t)v + 2]};
    float tg[3], bt[3];
    if (tans) {
        for (int a = 0; a < 3; a++) tg[a] = tans[3 * (size_t)v + a];
    } else {
        const bool x = fabsf(nr[1]) < 0.9f;
        const float ax[3] = {x ? 0.f : 1.f, x ? 1.f : 0.f, 0.f};
        cross_rn(ax, nr, tg);
        const float l = __fsqrt_rn(
            __fadd_rn(__fadd_rn(__fmul_rn(tg[0], tg[0]), __fmul_rn(tg[1], tg[1])), __fmul_rn(tg[2], tg[2])));
        const float inv = __fdiv_rn(1.0f, l);
        for (int a = 0; a < 3; a++) tg[a] = __fmul_rn(tg[a], inv);
    }
    cross_rn(nr, tg, bt);
    vpos[v] = make_float4(p[0], p[1], p[2], 0.f);
    vnrm[v] = make_float4(nr[0], nr[1], nr[2], 0.f);
    vbt[v] = make_float4(bt[0], bt[1], bt[2], 0.f);
}

}  // namespace

void launch_triangle_positions(const float* verts, const int32_t* tri, const int32_t* material, int n, float* tv,
                               int4* vidx, uint32_t* key6, int num_sms, cudaStream_t st) {
    if (n <= 0) return;
    const int blocks = (n + kThreads - 1) / kThreads;
    k_triangle_positions<<<blocks < 8 * num_sms ? blocks : 8 * num_sms, kThreads, 0, st>>>(verts, tri, material, n, tv,
                                                                                          vidx, key6);
}

void launch_leaf_triangles(const float* tv, const int32_t* order, const int32_t* rank, const int32_t* parent, int n,
                           float4* tris, cudaStream_t st) {
    if (n > 0) k_leaf_triangles<<<(n + kThreads - 1) / kThreads, kThreads, 0, st>>>(tv, order, rank, parent, n, tris);
}

void launch_vertices(const float* verts, const float* nrms, const float* tans, int n, float4* vpos, float4* vnrm,
                     float4* vbt, cudaStream_t st) {
    if (n > 0) k_vertices<<<(n + kThreads - 1) / kThreads, kThreads, 0, st>>>(verts, nrms, tans, n, vpos, vnrm, vbt);
}

void triangle_bounds(const uint32_t key6[6], float lo[3], float hi[3]) {
    auto value = [](uint32_t k) {
        const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
        float f;
        std::memcpy(&f, &u, 4);
        return f;
    };
    for (int a = 0; a < 3; a++) {
        lo[a] = key6[a] ? value(~key6[a]) : INFINITY;
        hi[a] = key6[3 + a] ? value(key6[3 + a]) : -INFINITY;
    }
}

}  // namespace cpppt_gb300
