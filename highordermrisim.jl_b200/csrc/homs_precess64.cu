// Free precession in FP64, in parallel over time and spins.
//
// Within a segment (a run of precession blocks) the field is a sum of 16 terms
// per spin times one coefficient waveform each, so the phase at sample j is
//   theta(s, j) = kappa_0(j) + sum_k b_k(s) kappa_k(j)   (turns)
// with kappa_k the running trapezoid integral of waveform k from the segment
// start (the prefix table of homs_split.cu; trapezoid and decay as
// src/simulation/Bloch/BlochHighOrderSimulatitonMethod.jl:76-92), and
//   M(s, j) = m0(s) exp(-t_j / T2(s)) cis(2 pi theta),   S(j, c) = sum_s M csm.
// No sample depends on another one, so samples spread over CTAs; a walk node by
// node leaves a small phantom's few CTAs waiting on one dependent chain.  The
// blocks of a run only restart the same exponentials, so a run is one segment.
//
// What bounds it: the FP64 pipe (64 multiply-adds per SM and clock, the same
// for DFMA and for the FP64 matrix instruction; about 72% busy) and the latency
// of its chains: leaving out the matrix step of an unused third order gains
// nothing (9.20 against 9.22 ms at 8 coils), a shorter decay series does.
// Per spin and sample 16 multiply-adds of phase, 27 to 30 FP64 operations of
// sine, cosine, decay and the complex product, 3 per coil of contraction.
//
// Organisation: CTA = 8 warps, a tile of samples x a range of 32-spin chunks
// (cp.async, NSTAGE stages).  A warp owns 16 samples (8 for more than 16
// coils, whose sums would not fit beside them: 5.60 against 5.74 ms at 32
// coils) and keeps their kappa rows and coil sums in registers.  Both
// contractions are m8n8k4 FP64 matrix instructions: the phase as (samples x
// terms) (terms x spins), whose result fragment (sample lane / 4, spins
// 2 (lane % 4) + {0, 1}) is, taken one spin parity at a time, exactly the A
// fragment of the coil product (samples x spins) (spins x coils), so M never
// leaves its registers.  The complex product takes three real ones: k1 = (Re M + Im M) Re c, k2 = Re M (Im c - Re c),
// k3 = Im M (Re c + Im c); Re = k1 - k3, Im = k1 + k2 (10.87 -> 10.31 ms at 8
// coils, 6.15 -> 5.86 ms at 32); above 16 coils, where a warp's 8 samples share a
// coefficient less, the form with one sum of c and two of M (5.63 -> 5.53 ms).  wj < 8 (segments of few samples): the other
// warps take other spin groups of the chunk and write partial sums of their own.
// The decay is 2^(t_ref r2), once per spin, chunk and tile, times a series of
// 2^((t - t_ref) r2) of degree 8 where that argument stays within 1/16 for the
// whole warp (10.28 -> 9.35 ms, 5.84 -> 5.76 ms) and of degree 5 within 1/128;
// four spin groups per iteration let their chains overlap (1, 2, 4 groups: 9.09,
// 8.90, 8.82 ms at 8 coils, 5.57, 5.49, 5.48 ms at 32).  Sine and cosine take the
// nearest of 256 points of the circle in shared memory and three terms of either
// series, a shorter chain than two polynomials over a quarter turn (8.83 -> 8.20
// ms, 5.48 -> 5.30 ms).
//
// Measured (B200, prepared runs, against the sequential per-spin kernel that it
// replaces): 40,000 spins x 4 segments of 10,000 samples x 8 coils 44.6 ->
// 8.2 ms, 11,979 spins x 4 x 9,500 samples x 32 coils 48.9 -> 5.2 ms.  Three
// CTAs per SM (80 registers) run the 8-coil case no faster (10.5 ms).
#include <algorithm>

#include "homs_fp64math.cuh"
#include "homs_fp64mma.cuh"
#include "homs_precess64.cuh"
#include "homs_split.cuh"

namespace homs {

namespace precess64 {

constexpr int THREADS = 256;
constexpr int CHUNK = 32;    // spins per stage
constexpr int NSTAGE = 3;
constexpr size_t PARTIAL_BUDGET = size_t(256) << 20;
constexpr int TERMS = 16;    // phase slots: basis terms 1..15, dw/(2 pi)
constexpr int BROW = 144;    // bytes of a staged basis row (128 + 16: conflict-free fragment loads)
constexpr double TWO_PI = 2.0 * 3.141592653589793;

__host__ __device__ constexpr int csm_row(int nt) { return nt * 128 + 16; }  // bytes of a staged sensitivity row
__host__ __device__ constexpr int stage_bytes(int nt) { return CHUNK * (BROW + 16 + 8 + csm_row(nt)); }
__host__ __device__ constexpr int smem_bytes(int nt) { return NSTAGE * stage_bytes(nt) + 2 * CHUNK * 8 + CIS_POINTS * 16; }  // + decays, circle

__host__ __device__ inline int64_t pad_spins(int64_t ns) { return (ns + CHUNK - 1) / CHUNK * CHUNK; }

// Phase slots switched on by a method (slot k: basis term k + 1, slot 15: dw).
__host__ __device__ inline uint32_t slot_mask(uint32_t method) {
    uint32_t m = 0x7u;  // first order: the field coefficients or the nominal gradients
    if (method & HOMS_HO2) m |= 0xF8u;
    if (method & HOMS_HO3) m |= 0x7F00u;
    if (method & HOMS_DW_PRECESSION) m |= 0x8000u;
    return m;
}

__global__ void table_kernel(const double *x, const double *y, const double *z, const double *dw, const double *T2,
                             int64_t ns, int64_t ns_pad, double *basis, double *r2) {
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < ns_pad; s += (int64_t)gridDim.x * blockDim.x) {
        double b[TERMS] = {};
        double r = 0.0;
        if (s < ns) {
            const double X = x[s], Y = y[s], Z = z[s];
            const double x2 = X * X, y2 = Y * Y, z2 = Z * Z;
            const double q = (x2 + y2) + z2;
            b[0] = X;
            b[1] = Y;
            b[2] = Z;
            b[3] = X * Y;
            b[4] = Z * Y;
            b[5] = 3.0 * z2 - q;
            b[6] = X * Z;
            b[7] = x2 - y2;
            b[8] = (3.0 * Y) * x2 - (y2 * Y);
            b[9] = (X * Z) * Y;
            b[10] = (5.0 * z2 - q) * Y;
            b[11] = 5.0 * (z2 * Z) - (3.0 * Z) * q;
            b[12] = (5.0 * z2 - q) * X;
            b[13] = x2 * Z - y2 * Z;
            b[14] = (x2 * X) - (3.0 * X) * y2;
            b[15] = dw[s] / TWO_PI;
            r = -1.4426950408889634 / T2[s];
        }
        double2 *out = reinterpret_cast<double2 *>(basis + s * TERMS);
#pragma unroll
        for (int k = 0; k < TERMS / 2; ++k) out[k] = make_double2(b[2 * k], b[2 * k + 1]);
        r2[s] = r;
    }
}

struct KernelArgs {
    int64_t ns, sample0, nchunks;  // samples sample0 + [0, tiles of the round)
    int64_t round_samples;                   // samples of the round (rows of a partial block)
    int32_t nc, parts;
    uint32_t slots;
    const double *basis, *r2, *prefix;
    const cplx<double> *xy, *csm_rows;
    cplx<double> *partial;
};

// A warp's sums by four real products, straight from memory (infinite states or
// sensitivities, see from_three).
template <int NT, int WJ>
__device__ __forceinline__ void sums_of_four(const KernelArgs &a, const double2 *circle) {
    constexpr int KSPLIT = 8 / WJ, MT = sample_tiles(NT);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 3, r = lane >> 2;
    const int c0 = (int)blockIdx.z * COIL_GROUP, ncg = min(COIL_GROUP, a.nc - c0);
    const int64_t ch0 = a.nchunks * blockIdx.y / a.parts, ch1 = a.nchunks * (blockIdx.y + 1) / a.parts;
    const int64_t jw = (int64_t)blockIdx.x * (8 * MT * WJ) + warp % WJ * (8 * MT);
    double re[MT][NT][2] = {}, im[MT][NT][2] = {};
#pragma unroll 1
    for (int64_t g = (CHUNK / 8) * ch0 + warp / WJ; g < (CHUNK / 8) * ch1; g += KSPLIT)
#pragma unroll 1
        for (int e = 0; e < 2; ++e) {
            const int64_t s = g * 8 + 2 * q + e;
            const bool ok = s < a.ns;
            cplx<double> v[MT];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                v[mt] = cplx<double>{0.0, 0.0};
                if (!ok) continue;
                const int64_t j = imin64(jw + mt * 8 + r, a.round_samples - 1);
                const double *row = a.prefix + (a.sample0 + j) * SPLIT_PREFIX_STRIDE;
                double th = row[0], sn, cs;
                for (int k = 0; k < TERMS; ++k)
                    if ((a.slots >> k) & 1u) th = fma(row[1 + k], a.basis[s * TERMS + k], th);
                cis_table(circle, th, cs, sn);
                const double ex = pow2(row[SPLIT_PREFIX_T] * a.r2[s]), ec = ex * cs, es = ex * sn;
                const cplx<double> m0 = a.xy[s];
                v[mt] = cplx<double>{m0.re * ec - m0.im * es, m0.re * es + m0.im * ec};
            }
            __syncwarp();
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const int c = nt * 8 + r;
                const cplx<double> w = ok && c < ncg ? a.csm_rows[s * a.nc + c0 + c] : cplx<double>{0.0, 0.0};
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) dmma4(re[mt][nt], im[mt][nt], v[mt].re, v[mt].im, w.re, w.im);
            }
        }
    store_sums<NT, WJ>(a.partial, a.round_samples, a.nc, re, im);
}

// NT: 8-coil tiles (at most COIL_GROUP coils per z slice); WJ: warps along the samples.
template <int NT, int WJ>
__global__ void __launch_bounds__(THREADS, 2) main_kernel(const KernelArgs a) {
    constexpr int CS = csm_row(NT), STAGE = stage_bytes(NT), KSPLIT = 8 / WJ, MT = sample_tiles(NT);
    // Three-product form: two sums of M and one of c, or one and two; NT of the
    // latter per element and MT of the former per 8 coils.
    constexpr bool SUMS_OF_M = NT > MT;
    extern __shared__ __align__(16) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane & 3, r = lane >> 2;
    const int wj = warp % WJ, kw = warp / WJ;
    const int c0 = (int)blockIdx.z * COIL_GROUP;
    const int ncg = min(COIL_GROUP, a.nc - c0);
    const int64_t ch0 = a.nchunks * blockIdx.y / a.parts, ch1 = a.nchunks * (blockIdx.y + 1) / a.parts;
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);

    // Sensitivity columns past the last coil are zero in every stage.
    if (ncg < NT * 8) {
        const int extra = NT * 8 - ncg;
        for (int i = tid; i < NSTAGE * CHUNK * extra; i += THREADS) {
            const int row = i / extra, col = ncg + i % extra;
            *reinterpret_cast<double2 *>(smem + (row / CHUNK) * STAGE + CHUNK * (BROW + 24) + (row % CHUNK) * CS +
                                         col * 16) = make_double2(0.0, 0.0);
        }
    }
    auto issue = [&](int64_t ch, int stage) {
        const uint32_t st = sbase + (uint32_t)(stage * STAGE);
        const int64_t s0 = ch * CHUNK;
        {
            const int spin = tid >> 3, piece = tid & 7;
            cp16(st + spin * BROW + piece * 16, a.basis + (s0 + spin) * TERMS + piece * 2, true);
        }
        if (tid < CHUNK) {
            const bool ok = s0 + tid < a.ns;
            cp16(st + CHUNK * BROW + tid * 16, a.xy + (ok ? s0 + tid : 0), ok);
        } else if (tid < CHUNK + CHUNK / 2) {
            const int p = tid - CHUNK;
            cp16(st + CHUNK * (BROW + 16) + p * 16, a.r2 + s0 + 2 * p, true);
        }
#pragma unroll
        for (int i = 0; i < CHUNK * NT * 8 / THREADS; ++i) {
            const int p = tid + i * THREADS, spin = p / (NT * 8), coil = p % (NT * 8);
            if (coil < ncg) {
                const bool ok = s0 + spin < a.ns;
                cp16(st + CHUNK * (BROW + 24) + spin * CS + coil * 16,
                     a.csm_rows + (ok ? (s0 + spin) * a.nc + c0 + coil : 0), ok);
            }
        }
    };

    // This warp's samples: rows 8 mt + r of its 16.  Phase slot of lane q in
    // step i: 4 q + i (the term order of a sum is free, and this one makes a
    // spin's fragment contiguous).
    double kap[MT][4], k0[MT], tj[MT], dmax = 0.0;
    const double t_ref =
        a.prefix[(a.sample0 + imin64((int64_t)blockIdx.x * (8 * MT * WJ) + 4 * MT * WJ, a.round_samples - 1)) *
                     SPLIT_PREFIX_STRIDE +
                 SPLIT_PREFIX_T];
    const int64_t jw = (int64_t)blockIdx.x * (8 * MT * WJ) + wj * (8 * MT);
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
        const int64_t j = jw + mt * 8 + r;
        const bool ok = j < a.round_samples;
        const double *row = a.prefix + (a.sample0 + (ok ? j : 0)) * SPLIT_PREFIX_STRIDE;
        k0[mt] = ok ? row[0] : 0.0;
        tj[mt] = ok ? row[SPLIT_PREFIX_T] : t_ref;
        dmax = fmax(dmax, fabs(tj[mt] - t_ref));
#pragma unroll
        for (int i = 0; i < 4; ++i) kap[mt][i] = ok ? row[1 + 4 * q + i] : 0.0;
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
    // Decay of the tile: E = 2^(t_ref r2) once per spin and chunk, by one warp a
    // chunk ahead, and a short series for the rest.
    double *decay = reinterpret_cast<double *>(smem + NSTAGE * STAGE);
    double2 *circle = reinterpret_cast<double2 *>(decay + 2 * CHUNK);
    if (tid < CIS_POINTS) cis_turns(tid * (1.0 / CIS_POINTS), circle[tid].x, circle[tid].y);
    auto load_r2 = [&](int64_t ch) { return a.r2[ch * CHUNK + lane]; };
    const uint32_t on = (a.slots >> (4 * q)) & 15u;
    double k1[MT][NT][2], k2[MT][NT][2], k3[MT][NT][2];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) k1[mt][nt][e] = k2[mt][nt][e] = k3[mt][nt][e] = 0.0;

#pragma unroll
    for (int s = 0; s < NSTAGE - 1; ++s) {
        if (ch0 + s < ch1) issue(ch0 + s, s);
        cp_commit();
    }
    if (warp == 0 && ch0 < ch1) decay[(ch0 & 1) * CHUNK + lane] = pow2(t_ref * load_r2(ch0));
    int stage = 0;
    for (int64_t ch = ch0; ch < ch1; ++ch) {
        cp_wait<NSTAGE - 2>();
        __syncthreads();
        const int fill = stage == 0 ? NSTAGE - 1 : stage - 1;  // the stage consumed last
        if (ch + NSTAGE - 1 < ch1) issue(ch + NSTAGE - 1, fill);
        cp_commit();
        const bool next_decay = ch + 1 < ch1 && warp == (int)(ch & 7);
        double next_r2 = 0.0;
        if (next_decay) next_r2 = load_r2(ch + 1);
        const double *dec = decay + (ch & 1) * CHUNK;
        const uint8_t *st = smem + stage * STAGE;
        if (++stage == NSTAGE) stage = 0;
#pragma unroll 4
        for (int g = kw; g < CHUNK / 8; g += KSPLIT) {
            const double2 *brow = reinterpret_cast<const double2 *>(st + (g * 8 + r) * BROW + q * 32);
            const double2 b01 = brow[0], b23 = brow[1];
            const double b[4] = {(on & 1u) ? b01.x : 0.0, (on & 2u) ? b01.y : 0.0, (on & 4u) ? b23.x : 0.0,
                                 (on & 8u) ? b23.y : 0.0};
            const double2 *m0p = reinterpret_cast<const double2 *>(st + CHUNK * BROW + (g * 8 + 2 * q) * 16);
            const double2 m0[2] = {m0p[0], m0p[1]};
            const double2 rr = *reinterpret_cast<const double2 *>(st + CHUNK * (BROW + 16) + (g * 8 + 2 * q) * 8);
            double th[MT][2];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) th[mt][0] = th[mt][1] = k0[mt];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) dmma(th[mt], kap[mt][i], b[i]);
            double mr[MT][2], mi[MT][2], ms[MT][2], md[MT][2];
            // m0 and the decay of each element: m0 E and a series of 2^(dt r2), of degree
            // 5 or 8 by the range of dt r2 in the warp; else m0 and 2^(t r2).
            const double most = dmax * fmax(fabs(rr.x), fabs(rr.y));
            double2 m[2] = {m0[0], m0[1]};
            double ex[MT][2];
            if (__all_sync(0xffffffffu, most <= POW2_SMALL)) {
                const double2 E = *reinterpret_cast<const double2 *>(dec + g * 8 + 2 * q);
                m[0] = make_double2(m0[0].x * E.x, m0[0].y * E.x);
                m[1] = make_double2(m0[1].x * E.y, m0[1].y * E.y);
                if (__all_sync(0xffffffffu, most <= POW2_TINY)) {
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                        for (int e = 0; e < 2; ++e) ex[mt][e] = pow2_tiny((tj[mt] - t_ref) * (e ? rr.y : rr.x));
                } else {
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                        for (int e = 0; e < 2; ++e) ex[mt][e] = pow2_small((tj[mt] - t_ref) * (e ? rr.y : rr.x));
                }
            } else {
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                    for (int e = 0; e < 2; ++e) ex[mt][e] = pow2(tj[mt] * (e ? rr.y : rr.x));
            }
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    double sn, cs;
                    cis_table(circle, th[mt][e], cs, sn);
                    const double ec = ex[mt][e] * cs, es = ex[mt][e] * sn;
                    mr[mt][e] = m[e].x * ec - m[e].y * es;
                    mi[mt][e] = m[e].x * es + m[e].y * ec;
                    ms[mt][e] = mr[mt][e] + mi[mt][e];
                    if (SUMS_OF_M) md[mt][e] = mi[mt][e] - mr[mt][e];
                }
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const double2 w = *reinterpret_cast<const double2 *>(st + CHUNK * (BROW + 24) +
                                                                         (g * 8 + 2 * q + e) * CS + (nt * 8 + r) * 16);
                    const double ws = w.x + w.y, wd = SUMS_OF_M ? 0.0 : w.y - w.x;
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt) {
                        if (SUMS_OF_M) {
                            dmma(k1[mt][nt], mr[mt][e], ws);
                            dmma(k2[mt][nt], md[mt][e], w.x);
                            dmma(k3[mt][nt], ms[mt][e], w.y);
                        } else {
                            dmma(k1[mt][nt], ms[mt][e], w.x);
                            dmma(k2[mt][nt], mr[mt][e], wd);
                            dmma(k3[mt][nt], mi[mt][e], ws);
                        }
                    }
                }
        }
        if (next_decay) decay[((ch + 1) & 1) * CHUNK + lane] = pow2(t_ref * next_r2);
    }
    cp_wait<0>();
    int top = 0;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) from_three(k1[mt][nt][e], k2[mt][nt][e], k3[mt][nt][e], top);
    store_sums<NT, WJ>(a.partial, a.round_samples, a.nc, k1, k2);
    if (__any_sync(0xffffffffu, top >= NOT_FINITE)) sums_of_four<NT, WJ>(a, circle);
}

// State at the segment's end: the same formula at the end row of the prefix
// table, and Mz = Mz e^{-T/T1} + rho (1 - e^{-T/T1}).
__global__ void __launch_bounds__(256) state_kernel(const double *basis, const double *endrow, uint32_t slots,
                                                    const double *T1, const double *T2, const double *rho, int64_t ns,
                                                    cplx<double> *xy, double *mz) {
    double kap[TERMS];
#pragma unroll
    for (int k = 0; k < TERMS; ++k) kap[k] = endrow[1 + k];
    const double k0 = endrow[0], T = endrow[SPLIT_PREFIX_T];
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < ns; s += (int64_t)gridDim.x * blockDim.x) {
        double th = k0;
#pragma unroll
        for (int k = 0; k < TERMS; ++k)
            if ((slots >> k) & 1u) th = fma(basis[s * TERMS + k], kap[k], th);
        double sn, cs;
        sincospi(2.0 * (th - rint(th)), &sn, &cs);
        const double e2 = exp(0.0 - T / T2[s]);
        const cplx<double> m0 = xy[s];
        const double ec = e2 * cs, es = e2 * sn;
        xy[s] = cplx<double>{m0.re * ec - m0.im * es, m0.re * es + m0.im * ec};
        const double e1 = exp(0.0 - T / T1[s]);
        mz[s] = mz[s] * e1 + rho[s] * (1.0 - e1);
    }
}

inline int grid_for(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 8)); }

template <int NT, int WJ>
cudaError_t launch(const KernelArgs &ka, int64_t tiles, int groups, cudaStream_t stream) {
    cudaError_t e = allow_max_dynamic_smem((const void *)main_kernel<NT, WJ>);
    if (e != cudaSuccess) return e;
    const dim3 grid((unsigned)tiles, (unsigned)ka.parts, (unsigned)groups);
    main_kernel<NT, WJ><<<grid, THREADS, smem_bytes(NT), stream>>>(ka);
    return cudaGetLastError();
}
template <int NT>
cudaError_t launch(int wj, const KernelArgs &ka, int64_t tiles, int groups, cudaStream_t stream) {
    return wj == 8 ? launch<NT, 8>(ka, tiles, groups, stream)
                   : wj == 4 ? launch<NT, 4>(ka, tiles, groups, stream) : launch<NT, 2>(ka, tiles, groups, stream);
}

}  // namespace precess64

using namespace precess64;

size_t precess64_table_bytes(int64_t ns) { return sizeof(double) * (TERMS + 1) * (size_t)pad_spins(ns); }

cudaError_t precess64_table(const double *x, const double *y, const double *z, const double *dw, const double *T2,
                            int64_t ns, void *table, cudaStream_t stream) {
    const int64_t np = pad_spins(ns);
    double *basis = static_cast<double *>(table);
    table_kernel<<<grid_for(np), 256, 0, stream>>>(x, y, z, dw, T2, ns, np, basis, basis + TERMS * np);
    return cudaGetLastError();
}

CoilCut precess64_cut(int64_t ns, int32_t nc, int64_t nsamples) {
    return coil_cut(pad_spins(ns) / CHUNK, nc, nsamples, PARTIAL_BUDGET);
}

size_t precess64_run_bytes(int64_t ns, int32_t nc, int64_t nadc) {
    return sizeof(double) * SPLIT_PREFIX_STRIDE * split_prefix_rows(nadc) +
           coil_cut_bound(pad_spins(ns) / CHUNK, nc, nadc, PARTIAL_BUDGET);
}

cudaError_t precess64_run(const Precess64Args &a, const CoilCut &cut, cudaEvent_t ev_start,
                          cudaEvent_t ev_stop, unsigned ev_flags, int64_t *launches, cudaStream_t stream) {
    const int64_t np = pad_spins(a.ns);
    const double *basis = static_cast<const double *>(a.table);
    const uint32_t slots = slot_mask(a.method);
    cudaError_t e;
    if (a.nsamples > 0) {
        const int tile = cut.tile(a.nc), groups = (a.nc + COIL_GROUP - 1) / COIL_GROUP, ksplit = 8 / cut.wj;
        const int64_t tiles = (a.nsamples + tile - 1) / tile;
        if (ev_start) cudaEventRecordWithFlags(ev_start, stream, ev_flags);
        for (int64_t t0 = 0; t0 < tiles; t0 += cut.round_tiles) {
            const int64_t nt = std::min(cut.round_tiles, tiles - t0);
            KernelArgs ka;
            ka.ns = a.ns;
            ka.sample0 = t0 * tile;
            ka.round_samples = std::min<int64_t>(nt * tile, a.nsamples - ka.sample0);
            ka.nchunks = np / CHUNK;
            ka.nc = a.nc;
            ka.parts = cut.parts;
            ka.slots = slots;
            ka.basis = basis;
            ka.r2 = basis + TERMS * np;
            ka.prefix = a.prefix;
            ka.xy = a.xy;
            ka.csm_rows = a.csm_rows;
            ka.partial = a.partial;
            switch (coil_tiles(a.nc)) {
                case 1: e = launch<1>(cut.wj, ka, nt, groups, stream); break;
                case 2: e = launch<2>(cut.wj, ka, nt, groups, stream); break;
                default: e = launch<4>(cut.wj, ka, nt, groups, stream); break;
            }
            if (e != cudaSuccess) return e;
            if (ev_stop && t0 + cut.round_tiles >= tiles) cudaEventRecordWithFlags(ev_stop, stream, ev_flags);
            e = launch_partial_finalize(a.partial, (int64_t)cut.parts * ksplit, ka.round_samples, a.nc,
                                                a.sig + ka.sample0, a.ldsig, stream);
            if (e != cudaSuccess) return e;
            if (launches) *launches += 2;
        }
    }
    state_kernel<<<grid_for(a.ns), 256, 0, stream>>>(basis, a.prefix + (size_t)a.nsamples * SPLIT_PREFIX_STRIDE, slots,
                                                     a.T1, a.T2, a.rho, a.ns, a.xy, a.mz);
    if (launches) *launches += 1;
    return cudaGetLastError();
}

}  // namespace homs
