// Free precession in FP32: the phases by a walk over the nodes, the signal in
// parallel over samples and spins.
//
// A spin's phase in FP32 is the running sum of its trapezoid terms, rounded
// node by node in the reference's order (src/simulation/Bloch/
// BlochHighOrderSimulatitonMethod.jl:54-92; this unit is compiled with
// -fmad=false): another order of that sum moves the signal by 1e-5 to 1e-4 of
// itself on readouts of 10,000 nodes.  The sum is therefore walked node by node
// as before, but alone: walk_kernel evaluates the field and writes one phase per
// spin and sample; coil_kernel turns phases into magnetisation (sine, cosine,
// decay, the initial state) and contracts it with the sensitivities, every
// sample on its own.  The single kernel that did both kept sine, cosine, decay
// and the coil sum of each sample in the walk's dependent chain and, for small
// phantoms, on the few SMs that the spins filled.
//
// walk_kernel is bound by instruction issue and latency (27 instructions per
// spin and node: the field of two nodes at a time in packed FP32 operations, then
// the sum through 8 of them in order; 41 with scalar operations, 214 -> 175 us
// for 40,000 spins x 2,516 nodes).  Up to SMALL_NS spins a spin takes 8 lanes,
// each evaluating two of 16 nodes, and only the sum itself runs through the
// lanes in order (4,096 spins x 2,058 nodes: 147 -> 67 us).
// coil_kernel waits on latency for few coils (no pipe above 45%, issue 58% with
// two CTAs per SM; per spin and sample 68 instructions with scalar sine, cosine
// and decay, 96 with sincosf, expf and a division per element: 457 -> 337 us for
// 40,000 spins x 2,516 samples x 8 coils), so up to 8 coils take packed FP32
// operations on two spins at a time and 74 registers for three CTAs per SM (a
// one-shot run of 4 x 10,000 such samples 10.45 -> 9.93 ms; packed alone 10.35).
// For many coils it is bound by the FP64 pipe: the coil sums are FP64 matrix
// instructions (homs_precess64.cu has the fragment layouts and the three-product
// complex form), which leaves the FP32 pipe to the magnetisation and sums the
// FP32 products without rounding them.  Phases cross
// through memory, 4 bytes per spin and sample each way.  A tile of one block takes
// the packed functions; tiles across blocks (a small max_block_length) take expf,
// sincosf and the initial state of each sample's own block: 40,000 spins x 4,000
// samples x 8 coils whole 1.24 ms, in blocks of 16, 4 and 1 nodes 1.36, 1.80 and 3.19
// (the sequential kernel 3.37 to 3.65).
//
// Measured (B200, against the single kernel): one-shot calls, 4,096 spins x
// 2,048 samples x 1 coil 1,754 -> 285 us, 40,000 spins x 4 x 10,000 samples x 8
// coils 33.3 -> 9.9 ms (0.1 and 1.4 ms of it by leaner calls); a prepared run of 48
// repetitions of 64 pulse nodes and 128 samples, 29,929 spins x 8 coils, 6.9 -> 3.9 ms.
#include <algorithm>

#include "homs_fp32math.cuh"
#include "homs_fp64mma.cuh"
#include "homs_precess32.cuh"

namespace homs {

namespace precess32 {

// Node table: COLS columns of node_stride(nnodes) words.
constexpr int COLS = 19;  // h[16], dt of the interval that ends at the node, block time, flags
constexpr int C_DT = 16, C_TP = 17, C_FLAGS = 18;
constexpr int F_ADC = 1, F_BLOCK = 2;
constexpr int WCHUNK = 64;  // nodes per shared-memory stage of the walk (aligned to their index)
constexpr int SMALL_NS = 16384;
inline int64_t node_stride(int64_t nnodes) { return (nnodes + WCHUNK - 1) / WCHUNK * WCHUNK; }
// Memory of a round: 384 MB of phases, or up to 4 GB for rounds of 128 samples (from
// 786,000 spins on; 4,000,000 spins x 300 samples x 8 coils: rounds of 128, 64 and 32
// samples 6.4, 7.2 and 9.5 ms), and never fewer than 32 samples.
constexpr size_t PHASE_BUDGET = size_t(384) << 20, PHASE_MOST = size_t(4) << 30, BLOCK_BUDGET = size_t(64) << 20, PARTIAL_BUDGET = size_t(128) << 20;

__host__ __device__ inline int64_t pad_spins(int64_t ns) { return (ns + 31) / 32 * 32; }

// Work area of a round: phases [nsamples][ns_pad], initial magnetisation
// [nblocks][ns_pad], and (block time, block) per sample.
struct RowInfo {
    float tp;
    int blk;
};
struct Work {
    float *phi;
    cplx<float> *xyb;
    RowInfo *rows;
};
inline size_t align256(size_t b) { return (b + 255) & ~size_t(255); }
inline Work carve(void *w, int64_t ns, int64_t nsamples, int32_t nblocks) {
    uint8_t *p = static_cast<uint8_t *>(w);
    Work out;
    out.phi = reinterpret_cast<float *>(p);
    p += align256(sizeof(float) * (size_t)pad_spins(ns) * (size_t)nsamples);
    out.xyb = reinterpret_cast<cplx<float> *>(p);
    p += align256(sizeof(cplx<float>) * (size_t)pad_spins(ns) * (size_t)nblocks);
    out.rows = reinterpret_cast<RowInfo *>(p);
    return out;
}

__global__ void nodes_kernel(SeqDev<float> q, uint32_t m, const float *tp, int64_t stride, float *nodes) {
    const int k = blockIdx.y;
    for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < stride; n += (int64_t)gridDim.x * blockDim.x) {
        float v = 0.0f;
        if (n < q.nnodes) {
            if (k == 0) {
                if (m & HOMS_HO0) v = q.h[0][n];
            } else if (k <= 3) {
                v = (m & HOMS_HO1) ? q.h[k][n] : (k == 1 ? q.gx : k == 2 ? q.gy : q.gz)[n];
            } else if (k <= 8) {
                if (m & HOMS_HO2) v = q.h[k][n];
            } else if (k <= 15) {
                if (m & HOMS_HO3) v = q.h[k][n];
            } else if (k == C_DT) {
                if (n > 0) v = q.dt[n - 1];
            } else if (k == C_TP) {
                v = tp[n];
            } else {
                v = __int_as_float((q.adc[n] ? F_ADC : 0) | (q.boundary[n] ? F_BLOCK : 0));
            }
        }
        nodes[k * stride + n] = v;
    }
}

struct WalkArgs {
    PhantomDev<float> p;
    StateDev<float> st;
    const float *nodes;
    int64_t node_stride, n_lo, n_hi, ns_pad;
    int block_start;
    uint32_t method;
    float c_twopig, c_neg;  // FP32 of 2 pi gamma and -2 pi gamma
    float neg_zero;         // -0 (mul2)
    Work w;
};

__device__ __forceinline__ cplx<float> cmul(cplx<float> a, cplx<float> b) {
    return cplx<float>{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
__device__ __forceinline__ cplx<float> magnetisation(cplx<float> xy, float phi, float tp, float T2) {
    const float e = expf(0.0f - tp / T2);
    float sn, cs;
    sincosf(phi, &sn, &cs);
    return cmul(xy, cplx<float>{e * cs, e * sn});
}

// Two FP32 operations in one instruction, each half rounded as the scalar one.
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 z, x, y;\n\t"
        "mov.b64 {%0, %1}, z;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
// The product as a multiply-add of `nz` = (-0, -0), a value that the compiler does
// not know: ptxas contracts mul.rn.f32x2 followed by add.rn.f32x2 into one
// multiply-add, whatever the rounding modifiers and -fmad say.
__device__ __forceinline__ float2 mul2(float s, float2 b, float nz) {
    float2 d;
    asm("{\n\t.reg .b64 x, y, z, w;\n\tmov.b64 x, {%2, %2};\n\tmov.b64 y, {%3, %4};\n\tmov.b64 w, {%5, %5};\n\t"
        "fma.rn.f32x2 z, x, y, w;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(s), "f"(b.x), "f"(b.y), "f"(nz));
    return d;
}

// Bz of two consecutive nodes, in the reference's order.  h(k): coefficient k
// of the two.  ORD: highest order of the method (a lower order that is off
// holds zero coefficients and zero basis terms).
template <int ORD, typename H>
__device__ __forceinline__ float2 field2(const H &h, const float (&b)[16], float dwterm, float nz) {
    float2 bz = add2(h(0), add2(add2(mul2(b[1], h(1), nz), mul2(b[2], h(2), nz)), mul2(b[3], h(3), nz)));
    if (ORD >= 2) {
        float2 t = add2(mul2(b[4], h(4), nz), mul2(b[5], h(5), nz));
#pragma unroll
        for (int k = 6; k <= 8; ++k) t = add2(t, mul2(b[k], h(k), nz));
        bz = add2(bz, t);
    }
    if (ORD >= 3) {
        float2 t = add2(mul2(b[9], h(9), nz), mul2(b[10], h(10), nz));
#pragma unroll
        for (int k = 11; k <= 15; ++k) t = add2(t, mul2(b[k], h(k), nz));
        bz = add2(bz, t);
    }
    return add2(bz, make_float2(dwterm, dwterm));
}

// G lanes per spin (1 or 8).
template <int ORD, int G>
__global__ void __launch_bounds__(128) walk_kernel(const WalkArgs a) {
    // Columns used: the coefficients up to the order, then dt, block time and flags.
    constexpr int NH = ORD >= 3 ? 16 : ORD == 2 ? 9 : 4, NCOL = NH + 3;
    constexpr int S_DT = NH, S_TP = NH + 1, S_FLAGS = NH + 2;
    __shared__ __align__(16) float stage[2][NCOL][WCHUNK];
    const int tid = threadIdx.x, lane = tid & 31, g = tid % G;
    const int64_t s = ((int64_t)blockIdx.x * blockDim.x + tid) / G;
    const bool active = s < a.p.ns;
    const int64_t si = active ? s : 0;
    const uint32_t m = a.method;
    const float px = a.p.x[si], py = a.p.y[si], pz = a.p.z[si];
    const float T1 = a.p.T1[si], T2 = a.p.T2[si], rho = a.p.rho[si];
    cplx<float> xy = active ? a.st.xy[si] : cplx<float>{0.0f, 0.0f};
    float mz = active ? a.st.z[si] : 0.0f;
    float acc = a.block_start ? 0.0f : (active ? a.st.acc[si] : 0.0f);
    const float dwterm = (m & HOMS_DW_PRECESSION) ? a.p.dw[si] / a.c_twopig : 0.0f;
    float b[16];
    {
        const float x2 = px * px, y2 = py * py, z2 = pz * pz;
        const float r2 = (x2 + y2) + z2;
        b[0] = 1.0f;
        b[1] = px;
        b[2] = py;
        b[3] = pz;
        b[4] = px * py;
        b[5] = pz * py;
        b[6] = 3.0f * z2 - r2;
        b[7] = px * pz;
        b[8] = x2 - y2;
        b[9] = (3.0f * py) * x2 - (y2 * py);
        b[10] = (px * pz) * py;
        b[11] = (5.0f * z2 - r2) * py;
        b[12] = 5.0f * (z2 * pz) - (3.0f * pz) * r2;
        b[13] = (5.0f * z2 - r2) * px;
        b[14] = x2 * pz - y2 * pz;
        b[15] = (x2 * px) - (3.0f * px) * y2;
        if (!(m & HOMS_HO2))
#pragma unroll
            for (int k = 4; k <= 8; ++k) b[k] = 0.0f;
    }
    // Stage c holds nodes 64 c .. 64 c + 63; the walk takes nodes n_lo + 1 .. n_hi.
    const int64_t c_lo = (a.n_lo + 1) / WCHUNK, c_hi = a.n_hi / WCHUNK;
    auto issue = [&](int64_t c, int buf) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&stage[buf][0][0]);
        for (int i = tid; i < NCOL * (WCHUNK / 4); i += blockDim.x) {
            const int col = i / (WCHUNK / 4), piece = i % (WCHUNK / 4);
            const int src = col < NH ? col : col - NH + C_DT;
            cp16(dst + i * 16, a.nodes + src * a.node_stride + c * WCHUNK + piece * 4, true);
        }
        cp_commit();
    };
    issue(c_lo, 0);
    // the field at node n_lo
    float prev;
    {
        const float *nd = a.nodes + a.n_lo;
        auto h = [&](int k) { return make_float2(nd[k * a.node_stride], 0.0f); };
        prev = field2<ORD>(h, b, dwterm, a.neg_zero).x;
    }
    float *phi = a.w.phi + s;
    cplx<float> *xyb = a.w.xyb + s;
    int blk = 0, sample = 0;
    if (active && g == 0) *xyb = xy;
    // Block end: Mxy of the last node, Mz relaxed over the block, the phase sum restarts.
    auto end_block = [&](float tp, bool more) {
        xy = magnetisation(xy, a.c_neg * (0.5f * acc), tp, T2);
        const float e1 = expf((0.0f - tp) / T1);
        mz = mz * e1 + rho * (1.0f - e1);
        acc = 0.0f;
        xyb += a.ns_pad;
        if (active && g == 0 && more) *xyb = xy;
    };
    int buf = 0;
    for (int64_t c = c_lo; c <= c_hi; ++c, buf ^= 1) {
        if (c < c_hi) issue(c + 1, buf ^ 1);
        else cp_commit();
        cp_wait<1>();
        __syncthreads();
        const float(&st)[NCOL][WCHUNK] = stage[buf];
        const int64_t n0 = c * WCHUNK;
        // Rows [lo, hi) of the stage belong to the walk; their flags as bit masks (bit i: row i).
        const int lo = (int)imax64(a.n_lo + 1 - n0, 0), hi = (int)imin64(a.n_hi + 1 - n0, WCHUNK);
        const uint64_t valid = (hi == 64 ? ~0ull : (1ull << hi) - 1ull) & ~((1ull << lo) - 1ull);
        uint64_t adc, ends;
        {
            const int f0 = __float_as_int(st[S_FLAGS][lane]), f1 = __float_as_int(st[S_FLAGS][lane + 32]);
            adc = (__ballot_sync(0xffffffffu, f0 & F_ADC) | (uint64_t)__ballot_sync(0xffffffffu, f1 & F_ADC) << 32) &
                  valid;
            ends = (__ballot_sync(0xffffffffu, f0 & F_BLOCK) |
                    (uint64_t)__ballot_sync(0xffffffffu, f1 & F_BLOCK) << 32) &
                   valid;
        }
        // The block time and block of the stage's samples.
        if (blockIdx.x == 0 && tid < 32) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = lane + 32 * h;
                const uint64_t below = (1ull << i) - 1ull;
                if ((adc >> i) & 1u)
                    a.w.rows[sample + __popcll(adc & below)] = RowInfo{st[S_TP][i], blk + __popcll(ends & below)};
            }
        }
        if (G == 1) {
            // 8 rows at a time: their fields first, then the sum through them in order.
#pragma unroll 1
            for (int i = lo & ~7; i < hi; i += 8) {
                float y[8];
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    const int at = i + 4 * v;
                    float2 f[2];
#pragma unroll
                    for (int w = 0; w < 2; ++w) {
                        auto h = [&](int k) { return *reinterpret_cast<const float2 *>(&st[k][at + 2 * w]); };
                        f[w] = field2<ORD>(h, b, dwterm, a.neg_zero);
                    }
                    const float4 dt = *reinterpret_cast<const float4 *>(&st[S_DT][at]);
                    y[4 * v] = (f[0].x + prev) * dt.x;
                    y[4 * v + 1] = (f[0].y + f[0].x) * dt.y;
                    y[4 * v + 2] = (f[1].x + f[0].y) * dt.z;
                    y[4 * v + 3] = (f[1].y + f[1].x) * dt.w;
                    prev = f[1].y;
                }
                const unsigned au = (unsigned)(adc >> i) & 0xFFu, eu = (unsigned)(ends >> i) & 0xFFu;
                const unsigned vu = (unsigned)(valid >> i) & 0xFFu;
                if (eu == 0u && vu == 0xFFu && au == 0xFFu) {
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        acc = acc + y[u];
                        if (active) phi[u * a.ns_pad] = a.c_neg * (0.5f * acc);
                    }
                    phi += 8 * a.ns_pad;
                } else {
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        if ((vu >> u) & 1u) acc = acc + y[u];
                        if ((au >> u) & 1u) {
                            if (active) *phi = a.c_neg * (0.5f * acc);
                            phi += a.ns_pad;
                        }
                        if ((eu >> u) & 1u) end_block(st[S_TP][i + u], n0 + i + u < a.n_hi);
                    }
                }
            }
        } else {
            // Lane g takes rows 2 g, 2 g + 1 of every 2 G; the sum runs through all of
            // them in order in every lane, and lane g keeps its own rows' values.
            constexpr int P = WCHUNK / (2 * G);
            float2 y[P], mine[P];
#pragma unroll
            for (int j = 0; j < P; ++j) {
                const int at = j * 2 * G + 2 * g;
                auto h = [&](int k) { return *reinterpret_cast<const float2 *>(&st[k][at]); };
                const float2 f = field2<ORD>(h, b, dwterm, a.neg_zero);
                const float before = __shfl_up_sync(0xffffffffu, f.y, 1, G);
                const float2 dt = *reinterpret_cast<const float2 *>(&st[S_DT][at]);
                y[j].x = (f.x + (g == 0 ? prev : before)) * dt.x;
                y[j].y = (f.y + f.x) * dt.y;
                prev = __shfl_sync(0xffffffffu, f.y, G - 1, G);
            }
#pragma unroll
            for (int j = 0; j < P; ++j) {
                mine[j] = make_float2(0.0f, 0.0f);
                const int i = j * 2 * G;
                float2 yk[G];
#pragma unroll
                for (int k = 0; k < G; ++k) {
                    yk[k].x = __shfl_sync(0xffffffffu, y[j].x, k, G);
                    yk[k].y = __shfl_sync(0xffffffffu, y[j].y, k, G);
                }
                constexpr unsigned FULL = (1u << (2 * G)) - 1u;
                const unsigned eu = (unsigned)(ends >> i) & FULL, vu = (unsigned)(valid >> i) & FULL;
                if (eu == 0u && vu == FULL) {
#pragma unroll
                    for (int k = 0; k < G; ++k) {
                        const float a0 = acc + yk[k].x;
                        acc = a0 + yk[k].y;
                        if (g == k) mine[j] = make_float2(a0, acc);
                    }
                } else {
#pragma unroll 1
                    for (int u = 0; u < 2 * G; ++u) {
                        const float yu = __shfl_sync(0xffffffffu, (u & 1) ? y[j].y : y[j].x, u >> 1, G);
                        if ((vu >> u) & 1u) acc = acc + yu;
                        if (g == u >> 1) {
                            if (u & 1) mine[j].y = acc;
                            else mine[j].x = acc;
                        }
                        if ((eu >> u) & 1u) end_block(st[S_TP][i + u], n0 + i + u < a.n_hi);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < P; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int i = j * 2 * G + 2 * g + e;
                    if (active && ((adc >> i) & 1u))
                        phi[(int64_t)__popcll(adc & ((1ull << i) - 1ull)) * a.ns_pad] =
                            a.c_neg * (0.5f * (e ? mine[j].y : mine[j].x));
                }
            phi += (int64_t)__popcll(adc) * a.ns_pad;
        }
        blk += __popcll(ends);
        sample += __popcll(adc);
        __syncthreads();
    }
    cp_wait<0>();
    if (active && g == 0) {
        a.st.xy[s] = xy;
        a.st.z[s] = mz;
        a.st.acc[s] = acc;
    }
}

constexpr int THREADS = 256;
constexpr int CHUNK = 32;
constexpr int NSTAGE = 3;
constexpr int PROW = 160;  // bytes of a staged phase row (32 spins, padded: conflict-free pairs)

__host__ __device__ constexpr int csm_row(int nt) { return nt * 64 + 16; }
__host__ __device__ constexpr int stage_bytes(int nt, int tile) { return tile * PROW + CHUNK * (csm_row(nt) + 8); }
__host__ __device__ constexpr int coil_smem(int nt, int tile) {
    return NSTAGE * stage_bytes(nt, tile) + 2 * CHUNK * 12;  // stages, decay entries of two chunks
}
constexpr float SMALL_DECAY = 0.0625f;  // |dt / T2| up to which the decay series below is used

struct CoilArgs {
    int64_t ns, ns_pad, sample0, round_samples, nchunks;
    int32_t nc, parts;
    const float *T2;
    const cplx<float> *csm_rows;
    Work w;
    cplx<double> *partial;
};

// A warp's sums by four real products, straight from memory (infinite states or
// sensitivities, see from_three).
template <int NT, int WJ>
__device__ __forceinline__ void sums_of_four(const CoilArgs &a) {
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
            cplx<float> v[MT];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                v[mt] = cplx<float>{0.0f, 0.0f};
                if (!ok) continue;
                const int64_t j = a.sample0 + imin64(jw + mt * 8 + r, a.round_samples - 1);
                const RowInfo row = a.w.rows[j];
                v[mt] = magnetisation(a.w.xyb[(int64_t)row.blk * a.ns_pad + s], a.w.phi[j * a.ns_pad + s], row.tp, a.T2[s]);
            }
            __syncwarp();
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const int c = nt * 8 + r;
                const cplx<float> w = ok && c < ncg ? a.csm_rows[s * a.nc + c0 + c] : cplx<float>{0.0f, 0.0f};
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) dmma4(re[mt][nt], im[mt][nt], v[mt].re, v[mt].im, w.re, w.im);
            }
        }
    store_sums<NT, WJ>(a.partial, a.round_samples, a.nc, re, im);
}

template <int NT, int WJ>
__global__ void __launch_bounds__(THREADS, NT == 1 ? 3 : 2) coil_kernel(const CoilArgs a) {
    constexpr int KSPLIT = 8 / WJ, MT = sample_tiles(NT), TILE = 8 * MT * WJ;
    constexpr int CS = csm_row(NT), STAGE = stage_bytes(NT, TILE);
    constexpr int O_CSM = TILE * PROW, O_XY = O_CSM + CHUNK * CS, O_DECAY = NSTAGE * STAGE;
    extern __shared__ __align__(16) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane & 3, r = lane >> 2;
    const int wj = warp % WJ, kw = warp / WJ;
    const int c0 = (int)blockIdx.z * COIL_GROUP;
    const int ncg = min(COIL_GROUP, a.nc - c0);
    const int64_t ch0 = a.nchunks * blockIdx.y / a.parts, ch1 = a.nchunks * (blockIdx.y + 1) / a.parts;
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
    const int64_t jt = (int64_t)blockIdx.x * TILE;  // first row of the tile in the round
    const int64_t rows_left = a.round_samples - jt;

    // Sensitivity columns past the last coil are zero in every stage.
    if (ncg < NT * 8) {
        const int extra = NT * 8 - ncg;
        for (int i = tid; i < NSTAGE * CHUNK * extra; i += THREADS) {
            const int row = i / extra, col = ncg + i % extra;
            *reinterpret_cast<float2 *>(smem + (row / CHUNK) * STAGE + O_CSM + (row % CHUNK) * CS + col * 8) =
                make_float2(0.0f, 0.0f);
        }
    }
    // This warp's samples: rows 8 mt + r of its 8 MT; the tile's rows mostly share one block.
    float tp[MT], dtp[MT], dmax = 0.0f;
    int blk[MT];
    const int blk0 = a.w.rows[a.sample0 + jt].blk;
    const bool one_block = a.w.rows[a.sample0 + jt + imin64(TILE, rows_left) - 1].blk == blk0;
    const float tp_ref = a.w.rows[a.sample0 + jt + imin64(TILE, rows_left) / 2].tp;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
        const int64_t j = imin64(wj * (8 * MT) + mt * 8 + r, rows_left - 1);
        const RowInfo info = a.w.rows[a.sample0 + jt + j];
        tp[mt] = info.tp;
        blk[mt] = info.blk;
        dtp[mt] = info.tp - tp_ref;
        dmax = fmaxf(dmax, fabsf(dtp[mt]));
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) dmax = fmaxf(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
    // Decay of the tile: exp(-t / T2) = E exp(-(t - tp_ref) / T2) with E = exp(-tp_ref
    // / T2) once per spin and chunk (by one warp, a chunk ahead) and a short
    // series for the rest.  Entries of spin i: E, -1/T2, T2.
    float *decay = reinterpret_cast<float *>(smem + O_DECAY);
    auto load_T2 = [&](int64_t ch) { return ch * CHUNK + lane < a.ns ? a.T2[ch * CHUNK + lane] : 1.0f; };
    auto fill_decay = [&](int64_t ch, float T2) {
        float *d = decay + (int)(ch & 1) * (3 * CHUNK);
        d[lane] = expf(0.0f - tp_ref / T2);
        d[CHUNK + lane] = -1.0f / T2;
        d[2 * CHUNK + lane] = T2;
    };
    auto issue = [&](int64_t ch, int stage) {
        const uint32_t st = sbase + (uint32_t)(stage * STAGE);
        const int64_t s0 = ch * CHUNK;
        // Bytes of this thread's pieces that hold a spin's phase: the walk writes none for
        // padding spins, whose phases are zero here (they vote on the path below).
        const int held = (int)imax64(0, imin64(16, (a.ns - s0 - (tid & 7) * 4) * 4));
#pragma unroll
        for (int i = 0; i < (TILE * 8 + THREADS - 1) / THREADS; ++i) {
            const int p = tid + i * THREADS, row = p >> 3, piece = p & 7;
            if (TILE * 8 < THREADS && p >= TILE * 8) break;
            const bool ok = row < rows_left;
            cp16_part(st + row * PROW + piece * 16,
                      a.w.phi + (a.sample0 + jt + (ok ? row : 0)) * a.ns_pad + s0 + piece * 4, ok ? held : 0);
        }
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const int p = tid + i * THREADS, spin = p / (NT * 8), coil = p % (NT * 8);
            if (coil < ncg) {
                const bool ok = s0 + spin < a.ns;
                cp8(st + O_CSM + spin * CS + coil * 8, a.csm_rows + (ok ? (s0 + spin) * a.nc + c0 + coil : 0), ok);
            }
        }
        if (tid < CHUNK) {
            const bool ok = s0 + tid < a.ns;
            cp8(st + O_XY + tid * 8, a.w.xyb + (int64_t)blk0 * a.ns_pad + (ok ? s0 + tid : 0), ok);
        }
    };
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
    if (warp == 0 && ch0 < ch1) fill_decay(ch0, load_T2(ch0));
    int stage = 0;
    for (int64_t ch = ch0; ch < ch1; ++ch) {
        cp_wait<NSTAGE - 2>();
        __syncthreads();
        const int fill = stage == 0 ? NSTAGE - 1 : stage - 1;  // the stage consumed last
        if (ch + NSTAGE - 1 < ch1) issue(ch + NSTAGE - 1, fill);
        cp_commit();
        const bool next_decay = ch + 1 < ch1 && warp == (int)(ch & 7);
        float next_T2 = 1.0f;
        if (next_decay) next_T2 = load_T2(ch + 1);
        const float *dec = decay + (int)(ch & 1) * (3 * CHUNK);
        const uint8_t *st = smem + stage * STAGE;
        if (++stage == NSTAGE) stage = 0;
#pragma unroll 1
        for (int g = kw; g < CHUNK / 8; g += KSPLIT) {
            const int sl = g * 8 + 2 * q;  // this lane's two spins
            const int64_t s = ch * CHUNK + sl;
            const float4 x4 = *reinterpret_cast<const float4 *>(st + O_XY + sl * 8);
            const float2 E = *reinterpret_cast<const float2 *>(dec + sl);
            const float2 r2 = *reinterpret_cast<const float2 *>(dec + CHUNK + sl);
            float2 ph[MT];
            float pmax = 0.0f;
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                ph[mt] = *reinterpret_cast<const float2 *>(st + (wj * (8 * MT) + mt * 8 + r) * PROW + sl * 4);
                pmax = fmaxf(pmax, fmaxf(fabsf(ph[mt].x), fabsf(ph[mt].y)));
            }
            cplx<float> v[MT][2];
            // One block, every |dt / T2| and phase of the warp within the series' and
            // the reduction's ranges; else the general functions (fmaxf drops a NaN
            // phase, which stays NaN in either form).
            if (one_block &&
                __all_sync(0xffffffffu,
                           dmax * fmaxf(fabsf(r2.x), fabsf(r2.y)) <= SMALL_DECAY && pmax < CIS32_RANGE)) {
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    // both spins at a time
                    const f32x2 x = pmul(pack2(dtp[mt], dtp[mt]), pack2(r2.x, r2.y)), E0 = pack2(E.x, E.y);
                    f32x2 p = pfma(x, pair(1.0f / 120.0f), pair(1.0f / 24.0f));
                    p = pfma(p, x, pair(1.0f / 6.0f));
                    p = pfma(p, x, pair(0.5f));
                    p = pfma(p, x, pair(1.0f));
                    const f32x2 ec = pfma(E0, pmul(x, p), E0);
                    f32x2 cs, sn;
                    cis32_pair(pack2(ph[mt].x, ph[mt].y), cs, sn);
                    cs = pmul(ec, cs);
                    sn = pmul(ec, sn);
                    const f32x2 xr = pack2(x4.x, x4.z), xi = pack2(x4.y, x4.w);
                    const float2 re = unpack2(pfma(xr, cs, pmul(pneg(xi), sn)));
                    const float2 im = unpack2(pfma(xr, sn, pmul(xi, cs)));
                    v[mt][0] = cplx<float>{re.x, im.x};
                    v[mt][1] = cplx<float>{re.y, im.y};
                }
            } else {
                const float2 t2 = *reinterpret_cast<const float2 *>(dec + 2 * CHUNK + sl);
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        cplx<float> xy = e ? cplx<float>{x4.z, x4.w} : cplx<float>{x4.x, x4.y};
                        if (!one_block && s + e < a.ns) xy = a.w.xyb[(int64_t)blk[mt] * a.ns_pad + s + e];
                        v[mt][e] = magnetisation(xy, e ? ph[mt].y : ph[mt].x, tp[mt], e ? t2.y : t2.x);
                    }
            }
            double mr[MT][2], mi[MT][2], ms[MT][2];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    mr[mt][e] = (double)v[mt][e].re;
                    mi[mt][e] = (double)v[mt][e].im;
                    ms[mt][e] = mr[mt][e] + mi[mt][e];
                }
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const float2 wf =
                        *reinterpret_cast<const float2 *>(st + O_CSM + (sl + e) * CS + (nt * 8 + r) * 8);
                    const double wx = wf.x, wy = wf.y, wd = wy - wx, ws = wx + wy;
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt) {
                        dmma(k1[mt][nt], ms[mt][e], wx);
                        dmma(k2[mt][nt], mr[mt][e], wd);
                        dmma(k3[mt][nt], mi[mt][e], ws);
                    }
                }
        }
        if (next_decay) fill_decay(ch + 1, next_T2);
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
    if (__any_sync(0xffffffffu, top >= NOT_FINITE)) sums_of_four<NT, WJ>(a);
}

template <int ORD>
cudaError_t launch_walk(const WalkArgs &a, cudaStream_t stream) {
    // Small phantoms: 8 lanes per spin; else one.  Prepared runs of 4 segments of 512
    // (2,048) samples x 8 coils, one lane and eight: 12,000 spins 0.41 and 0.41 ms (1.16
    // and 1.04), 16,000 0.42 and 0.45 (1.23 and 1.20), 20,000 0.48 and 0.54 (1.43 and
    // 1.51).  One lane in CTAs of 32, 64 and 128 threads, 75,000 x 2,048: 3.31, 3.27, 3.25.
    if (a.p.ns <= SMALL_NS) {
        walk_kernel<ORD, 8><<<(unsigned)((a.p.ns * 8 + 127) / 128), 128, 0, stream>>>(a);
    } else {
        walk_kernel<ORD, 1><<<(unsigned)((a.p.ns + 127) / 128), 128, 0, stream>>>(a);
    }
    return cudaGetLastError();
}
template <int NT, int WJ>
cudaError_t launch_coil(const CoilArgs &ca, int64_t tiles, int groups, cudaStream_t stream) {
    cudaError_t e = allow_max_dynamic_smem((const void *)coil_kernel<NT, WJ>);
    if (e != cudaSuccess) return e;
    const dim3 grid((unsigned)tiles, (unsigned)ca.parts, (unsigned)groups);
    coil_kernel<NT, WJ><<<grid, THREADS, coil_smem(NT, 8 * sample_tiles(NT) * WJ), stream>>>(ca);
    return cudaGetLastError();
}
template <int NT>
cudaError_t launch_coil(int wj, const CoilArgs &ca, int64_t tiles, int groups, cudaStream_t stream) {
    return wj == 8 ? launch_coil<NT, 8>(ca, tiles, groups, stream)
                   : wj == 4 ? launch_coil<NT, 4>(ca, tiles, groups, stream)
                             : launch_coil<NT, 2>(ca, tiles, groups, stream);
}

}  // namespace precess32

using namespace precess32;

size_t precess32_node_bytes(int64_t nnodes) { return sizeof(float) * COLS * (size_t)node_stride(nnodes); }

cudaError_t precess32_nodes(const SeqDev<float> &q, uint32_t method, const float *tp, void *nodes,
                            cudaStream_t stream) {
    const int64_t stride = node_stride(q.nnodes);
    const dim3 grid((unsigned)std::min<int64_t>((stride + 255) / 256, 1024), COLS);
    nodes_kernel<<<grid, 256, 0, stream>>>(q, method, tp, stride, static_cast<float *>(nodes));
    return cudaGetLastError();
}

int64_t precess32_max_samples(int64_t ns) {
    const size_t row = sizeof(float) * (size_t)pad_spins(ns);
    return std::max({(int64_t)(PHASE_BUDGET / row), std::min<int64_t>(128, (int64_t)(PHASE_MOST / row)), (int64_t)32});
}
int64_t precess32_max_blocks(int64_t ns) {
    return std::max<int64_t>(1, (int64_t)(BLOCK_BUDGET / (sizeof(cplx<float>) * (size_t)pad_spins(ns))));
}
size_t precess32_work_bytes(int64_t ns, int64_t nsamples, int32_t nblocks) {
    const size_t np = (size_t)pad_spins(ns);
    return align256(sizeof(float) * np * (size_t)nsamples) + align256(sizeof(cplx<float>) * np * (size_t)nblocks) +
           align256(sizeof(RowInfo) * (size_t)nsamples);
}
size_t precess32_run_bytes(int64_t ns, int32_t nc, int64_t nnodes, int64_t nadc, int64_t nblocks, int64_t block_adc) {
    const int64_t blocks = std::min(nblocks, precess32_max_blocks(ns));
    const int64_t samples = std::min({nadc, precess32_max_samples(ns), blocks * block_adc});
    return precess32_node_bytes(nnodes) + precess32_work_bytes(ns, samples, (int32_t)blocks) +
           coil_cut_bound(pad_spins(ns) / CHUNK, nc, samples, PARTIAL_BUDGET, 148 * 3);
}
CoilCut precess32_cut(int64_t ns, int32_t nc, int64_t nsamples) {
    // Three CTAs per SM for up to 8 coils, unless these only add partial sums to read:
    // with few tiles a part is a few chunks already.  Two per SM and three, 4 segments
    // x 8 coils: 30,000 spins x 256 samples 0.358 and 0.361 ms, x 512 0.544 and 0.545,
    // x 768 0.757 and 0.744, x 2,048 1.73 and 1.68; 75,000 x 128 0.353 and 0.356, x 2,048
    // 3.42 and 3.26; below 12,000 spins within 2% of one another (48 repetitions of 128
    // samples: 3.87 and 3.98 ms).
    const int64_t places = coil_tiles(nc) == 1 && nsamples > 6 * 128 ? 148 * 3 : 148 * 2;
    return coil_cut(pad_spins(ns) / CHUNK, nc, nsamples, PARTIAL_BUDGET, places);
}

cudaError_t precess32_run(const Precess32Args &a, const CoilCut &cut, cudaEvent_t ev_start, cudaEvent_t ev_stop,
                          unsigned ev_flags, int64_t *launches, cudaStream_t stream) {
    const int64_t ns = a.phantom.ns;
    const double twopig = 2.0 * 3.141592653589793 * a.gamma;
    WalkArgs w;
    w.p = a.phantom;
    w.st = a.state;
    w.nodes = static_cast<const float *>(a.nodes);
    w.node_stride = node_stride(a.nnodes);
    w.n_lo = a.n_lo;
    w.n_hi = a.n_hi;
    w.ns_pad = pad_spins(ns);
    w.block_start = a.block_start;
    w.method = a.method;
    w.c_twopig = (float)twopig;
    w.c_neg = (float)(-twopig);
    w.neg_zero = -0.0f;
    w.w = carve(a.work, ns, a.nsamples, a.nblocks);
    if (ev_start) cudaEventRecordWithFlags(ev_start, stream, ev_flags);
    cudaError_t e = (a.method & HOMS_HO3) ? launch_walk<3>(w, stream)
                                          : (a.method & HOMS_HO2) ? launch_walk<2>(w, stream) : launch_walk<1>(w, stream);
    if (e != cudaSuccess) return e;
    if (launches) *launches += 1;
    if (a.nsamples > 0) {
        const int tile = cut.tile(a.phantom.nc), groups = (a.phantom.nc + COIL_GROUP - 1) / COIL_GROUP;
        const int64_t tiles = (a.nsamples + tile - 1) / tile;
        for (int64_t t0 = 0; t0 < tiles; t0 += cut.round_tiles) {
            const int64_t nt = std::min(cut.round_tiles, tiles - t0);
            CoilArgs ca;
            ca.ns = ns;
            ca.ns_pad = w.ns_pad;
            ca.sample0 = t0 * tile;
            ca.round_samples = std::min<int64_t>(nt * tile, a.nsamples - ca.sample0);
            ca.nchunks = w.ns_pad / CHUNK;
            ca.nc = a.phantom.nc;
            ca.parts = cut.parts;
            ca.T2 = a.phantom.T2;
            ca.csm_rows = a.phantom.csm;
            ca.w = w.w;
            ca.partial = a.partial;
            switch (coil_tiles(ca.nc)) {
                case 1: e = launch_coil<1>(cut.wj, ca, nt, groups, stream); break;
                case 2: e = launch_coil<2>(cut.wj, ca, nt, groups, stream); break;
                default: e = launch_coil<4>(cut.wj, ca, nt, groups, stream); break;
            }
            if (e != cudaSuccess) return e;
            if (ev_stop && t0 + cut.round_tiles >= tiles) cudaEventRecordWithFlags(ev_stop, stream, ev_flags);
            e = launch_partial_finalize<double, float>(a.partial, (int64_t)cut.parts * (8 / cut.wj), ca.round_samples,
                                                       ca.nc, a.sig + ca.sample0, a.ldsig, stream);
            if (e != cudaSuccess) return e;
            if (launches) *launches += 2;
        }
    } else if (ev_stop) {
        cudaEventRecordWithFlags(ev_stop, stream, ev_flags);
    }
    return cudaSuccess;
}

}  // namespace homs
