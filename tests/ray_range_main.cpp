// Deals the rays of a batch to the warps of a traversal launch with the
// kernels' own arithmetic (ray_range.h) and checks that every ray is taken
// once and none outside the batch.  argv: rays, warps, 1 for a first range
// without the counter, rays that the counter starts with.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../cpp-pt_gb300/csrc/ray_range.h"

using namespace cpppt_gb300;

struct Warp {
    RayRange pool;
    bool exhausted, done = false;
};

int main(int, char** argv) {
    const int n = std::atoi(argv[1]), nwarps = std::atoi(argv[2]);
    const bool own_first = std::atoi(argv[3]) != 0;
    uint32_t counter = (uint32_t)std::strtoul(argv[4], nullptr, 10);
    const int c0 = own_first ? ray_chunk(n, nwarps, 1) : 0;
    const long long skipped = counter;  // as if taken before
    const int first_seen = (int)(nwarps * (long long)c0 + skipped);
    std::vector<unsigned char> seen(n - first_seen > 0 ? n - first_seen : 0, 0);
    std::vector<unsigned char> own(nwarps * (size_t)c0, 0);
    std::vector<Warp> w(nwarps);
    for (int i = 0; i < nwarps; i++) w[i] = Warp{fetched_range(0, i * c0, c0, n), nwarps * c0 >= n};
    for (int live = nwarps, step = 0; live > 0; step++)
        for (int i = 0; i < nwarps; i++) {
            Warp& v = w[i];
            if (v.done) continue;
            const uint32_t want = 1 + (i + step) % 32;
            RayRange after{v.pool.end, v.pool.end};
            if (v.pool.end - v.pool.next < want && !v.exhausted) {
                const int chunk = ray_chunk(n - (int)v.pool.end, nwarps, 2);
                const int taken = (int)counter;
                counter += chunk;
                after = fetched_range(taken, nwarps * c0, chunk, n);
                v.exhausted = after.end == (uint32_t)n;
            }
            bool any = false;
            for (uint32_t r = 0; r < want; r++) {
                uint32_t i32;
                if (!ray_of(r, v.pool, after, i32)) continue;
                any = true;
                const int ray = (int)i32;
                if (ray < 0 || ray >= n) return std::printf("ray %d of %d\n", ray, n), 1;
                unsigned char* s = ray < (int)own.size() ? &own[ray] : (ray >= first_seen ? &seen[ray - first_seen] : nullptr);
                if (!s || (*s)++) return std::printf("ray %d twice\n", ray), 1;
            }
            v.pool = left_of(want, v.pool, after);
            if (!any) {
                v.done = true;
                live--;
            }
        }
    for (size_t i = 0; i < own.size() && (int)i < n; i++)
        if (!own[i]) return std::printf("ray %zu not taken\n", i), 1;
    for (size_t i = 0; i < seen.size(); i++)
        if (!seen[i]) return std::printf("ray %zu not taken\n", i + first_seen), 1;
    return 0;
}
