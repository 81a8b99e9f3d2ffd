// Pieces shared by the two precession kernels (homs_precess64.cu,
// homs_precess32.cu): the FP64 matrix instruction, 16- and 8-byte asynchronous
// copies, and the cut of a launch into sample tiles and spin parts.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "homs_common.cuh"

namespace homs {

// d (8 x 8) += a (8 x 4) b (4 x 8): lane l holds a[l / 4][l % 4], b[l % 4][l / 4]
// and d[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}
// Re and Im of a complex sum from its three products k1, k2, k3, in k1 and k2;
// `top` collects the largest high word: from NOT_FINITE on, an infinity or a NaN
// is among them.  Infinite operands make inf - inf of the three products where the
// four of the plain form keep the infinity; the kernels then take their sums anew.
constexpr int NOT_FINITE = 0x7FF00000;
__device__ __forceinline__ void from_three(double &k1, double &k2, double k3, int &top) {
    k2 += k1;
    k1 -= k3;
    top = max(top, max(__double2hiint(k1) & 0x7FFFFFFF, __double2hiint(k2) & 0x7FFFFFFF));
}
// re += x w, im likewise, by four real products.
__device__ __forceinline__ void dmma4(double (&re)[2], double (&im)[2], double xr, double xi, double wr, double wi) {
    dmma(re, xr, wr);
    dmma(re, -xi, wi);
    dmma(im, xr, wi);
    dmma(im, xi, wr);
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

// A warp's coil sums into its block of the partial sums, in a kernel of 8 warps, WJ
// of them along the samples (blockIdx: sample tile, spin part, coil slice).
template <int NT, int WJ>
__device__ __forceinline__ void store_sums(cplx<double> *partial, int64_t round_samples, int32_t nc,
                                           const double (&re)[sample_tiles(NT)][NT][2],
                                           const double (&im)[sample_tiles(NT)][NT][2]) {
    constexpr int MT = sample_tiles(NT);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 3, r = lane >> 2;
    const int c0 = (int)blockIdx.z * COIL_GROUP, ncg = min(COIL_GROUP, nc - c0);
    cplx<double> *out = partial + (size_t)(blockIdx.y * (8 / WJ) + warp / WJ) * round_samples * nc + c0;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
        const int64_t j = (int64_t)blockIdx.x * (8 * MT * WJ) + warp % WJ * (8 * MT) + mt * 8 + r;
        if (j >= round_samples) continue;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int c = nt * 8 + 2 * q + e;
                if (c < ncg) out[j * nc + c] = cplx<double>{re[mt][nt][e], im[mt][nt][e]};
            }
    }
}

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

// No launch of at most `nsamples` samples has larger partial sums (coil_cut): a
// launch takes a tile at least, and beyond the budget no more; its parts fill at most
// 8 waves of `places` CTAs.
inline size_t coil_cut_bound(int64_t chunks, int32_t nc, int64_t nsamples, size_t budget, int64_t places = 148 * 2) {
    if (nsamples <= 0) return 0;
    const int64_t per_warp = 8 * sample_tiles(coil_tiles(nc)), groups = (nc + COIL_GROUP - 1) / COIL_GROUP;
    const double tile = 16.0 * 8 * per_warp * nc;  // of one part, whatever wj
    const int64_t tiles = (nsamples + 2 * per_warp - 1) / (2 * per_warp);
    const double most = tile * std::max(tiles, std::min(tiles * chunks, 8 * places / groups));
    return (size_t)std::max(tile, std::min((double)budget, most));
}

}  // namespace homs
