// Pieces shared by the two precession kernels (homs_precess64.cu,
// homs_precess32.cu): the FP64 matrix instruction, 16- and 8-byte asynchronous
// copies, and the cut of a launch into sample tiles and spin parts.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

namespace homs {

// d (8 x 8) += a (8 x 4) b (4 x 8): lane l holds a[l / 4][l % 4], b[l % 4][l / 4]
// and d[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}
// Asynchronous copies into shared memory; zeros where !valid (src stays a valid address).
__device__ __forceinline__ void cp16(uint32_t dst, const void *src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
// The first n (0 .. 16) bytes, then zeros.
__device__ __forceinline__ void cp16_part(uint32_t dst, const void *src, int n) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp8(uint32_t dst, const void *src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(valid ? 8 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

constexpr int COIL_GROUP = 32;  // coils per launch slice
// 8-coil tiles of a slice for nc coils, and 8-sample tiles of a warp: the coil
// sums of 32 coils would not fit the registers beside those of 16 samples.
inline int coil_tiles(int32_t nc) { return nc <= 8 ? 1 : nc <= 16 ? 2 : 4; }
__host__ __device__ constexpr int sample_tiles(int coil_tiles) { return coil_tiles == 4 ? 1 : 2; }

// Cut of a launch of `nsamples` samples x `chunks` 32-spin chunks into sample
// tiles of 8 * sample_tiles * wj rows and `parts` ranges of chunks, for CTAs
// of 8 warps (`places` at a time; two per SM by default).
struct CoilCut {
    int wj = 8;           // warps along the samples; the 8 / wj groups of warps split the spins
    int parts = 1;
    int64_t round_tiles = 0;  // tiles per launch
    size_t partial_bytes = 0; // FP64 partial sums of a launch
    int tile(int32_t nc) const { return 8 * sample_tiles(coil_tiles(nc)) * wj; }
};
inline CoilCut coil_cut(int64_t chunks, int32_t nc, int64_t nsamples, size_t budget, int64_t places = 148 * 2) {
    CoilCut p;
    if (nsamples <= 0) return p;
    // 8 warps along the samples, or fewer where that tile would be mostly padding
    const int per_warp = 8 * sample_tiles(coil_tiles(nc));
    auto padded = [&](int wj) { return (nsamples + per_warp * wj - 1) / (per_warp * wj) * (per_warp * wj); };
    for (int wj : {4, 2})
        if (padded(wj) * 10 <= padded(p.wj) * 8) p.wj = wj;
    const int tile = p.tile(nc), ksplit = 8 / p.wj;
    const int64_t tiles = (nsamples + tile - 1) / tile, groups = (nc + COIL_GROUP - 1) / COIL_GROUP;
    // rounds whose partial sums fit the budget in one part
    const size_t tile_bytes = 16 * (size_t)ksplit * tile * nc;
    p.round_tiles = std::max<int64_t>(1, std::min<int64_t>(tiles, (int64_t)(budget / tile_bytes)));
    // parts: least waves of `places` CTAs x (chunks of a CTA + 2 for its start and its sums)
    const int64_t per_wave = p.round_tiles * groups;
    const int64_t most = std::max<int64_t>(
        1, std::min<int64_t>(std::min<int64_t>(chunks, 1024), (int64_t)(budget / (tile_bytes * p.round_tiles))));
    int64_t best = INT64_MAX;
    for (int64_t waves = 1; waves <= 8; ++waves) {
        const int64_t n = std::max<int64_t>(1, std::min<int64_t>(most, waves * places / per_wave));
        const int64_t cost = ((per_wave * n + places - 1) / places) * ((chunks + n - 1) / n + 2);
        if (cost < best) {
            best = cost;
            p.parts = (int)n;
        }
    }
    p.partial_bytes = tile_bytes * p.round_tiles * p.parts;
    return p;
}

}  // namespace homs
