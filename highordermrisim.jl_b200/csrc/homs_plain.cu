// RF excitation and short precession segments in the phantom's own precision (FP64
// or FP32) on CUDA cores, fused with a deterministic multi-coil reduction of the
// samples acquired meanwhile, and the standalone coil reduction.  No per-spin ADC
// history is written to HBM: ADC states are staged in shared memory and contracted
// with the receive sensitivities on chip, one CTA partial per (CTA, sample, coil),
// then summed over CTAs in a fixed order.
//
// This translation unit is compiled with -fmad=false so that every product
// and sum rounds exactly as in HighOrderMRISim.jl's CPU path
// (src/simulation/Bloch/BlochHighOrderSimulatitonMethod.jl:43-134), which does
// not contract multiply-adds; the FP64 kernel therefore agrees with the FP64
// CPU restatement to ~1e-15.
#include <cfloat>
#include <type_traits>

#include "homs_common.cuh"
#include "homs_fp64mma.cuh"

namespace homs {

template <typename T>
struct Math;

template <>
struct Math<double> {
    static __device__ __forceinline__ double ex(double x) { return exp(x); }
    static __device__ __forceinline__ void sc(double x, double *s, double *c) { sincos(x, s, c); }
    static __device__ __forceinline__ double hyp(double a, double b) { return hypot(a, b); }
    static __device__ __forceinline__ double sq(double a) { return sqrt(a); }
    static __device__ __forceinline__ double eps() { return DBL_EPSILON; }
};

template <>
struct Math<float> {
    static __device__ __forceinline__ float ex(float x) { return expf(x); }
    static __device__ __forceinline__ void sc(float x, float *s, float *c) { sincosf(x, s, c); }
    static __device__ __forceinline__ float hyp(float a, float b) { return hypotf(a, b); }
    static __device__ __forceinline__ float sq(float a) { return sqrtf(a); }
    static __device__ __forceinline__ float eps() { return FLT_EPSILON; }
};

// Julia's complex product: (ar*br - ai*bi, ar*bi + ai*br).
template <typename T>
__device__ __forceinline__ cplx<T> cmul(cplx<T> a, cplx<T> b) {
    return cplx<T>{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}

constexpr int NODE_CHUNK = 32;

// Shared-memory node cache for one chunk of nodes [c0, c0 + NODE_CHUNK].
template <typename T>
struct NodeCache {
    T dt[NODE_CHUNK + 1];
    T g[3][NODE_CHUNK + 1];
    T psi[NODE_CHUNK + 1];
    cplx<T> b1[NODE_CHUNK + 1];
    T ab1[NODE_CHUNK + 1];  // |B1| of the node
    T dfg[NODE_CHUNK + 1];  // df / gamma of the node
    uint8_t adc[NODE_CHUNK + 1];
    uint8_t bnd[NODE_CHUNK + 1];
};

template <typename T>
__device__ void load_nodes(NodeCache<T> &nc, const SeqDev<T> &q, int64_t c0, int64_t c_end, T gamma) {
    // nodes c0 .. min(c0 + NODE_CHUNK, c_end) inclusive
    const int n = (int)imin64(NODE_CHUNK, c_end - c0) + 1;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        int64_t g = c0 + i;
        nc.dt[i] = (g < q.nnodes - 1) ? q.dt[g] : T(0);
        nc.adc[i] = q.adc[g];
        nc.bnd[i] = q.boundary[g];
        nc.g[0][i] = q.gx[g];
        nc.g[1][i] = q.gy[g];
        nc.g[2][i] = q.gz[g];
        const cplx<T> b1 = q.b1[g];
        nc.b1[i] = b1;
        nc.psi[i] = q.psi[g];
        // Spin-independent parts of the RF step, computed once per node
        // with the same operations as the per-spin code used.
        nc.ab1[i] = Math<T>::hyp(b1.re, b1.im);
        nc.dfg[i] = q.df[g] / gamma;
    }
}

// Contract `na` staged ADC states X[a][s] (s < PLAIN_THREADS) with the
// sensitivities of this CTA's spins and write one partial row per sample:
// out[a * nc + c] = sum_s X[a][s] * csm[s][c], summed in type A over spins in a
// fixed order (a per-lane sweep, then splits in index order).
template <typename T, typename A>
__device__ void reduce_stage(const cplx<T> *X, cplx<A> *P, int na, const cplx<T> *csm_rows, int csm_ld,
                             int nvalid, int32_t nc, cplx<A> *out) {
    const int t = threadIdx.x;
    for (int cg = 0; cg < nc; cg += 32) {
        const int left = min(32, nc - cg);
        int cw = 1;
        while (cw < left) cw <<= 1;
        const int cl = t % cw, split = t / cw;
        const int c = cg + cl;
        cplx<A> acc[PLAIN_STAGE];
#pragma unroll
        for (int a = 0; a < PLAIN_STAGE; ++a) acc[a] = cplx<A>{A(0), A(0)};
        if (cl < left) {
            for (int i = 0; i < cw; ++i) {
                const int s = split * cw + i;
                if (s >= nvalid) break;
                const cplx<T> wt = csm_rows[(int64_t)s * csm_ld + c];
                const cplx<A> w{A(wt.re), A(wt.im)};
                // Complex multiply-accumulate as four fused multiply-adds: the
                // reference's coil sum is a BLAS product, which fuses them too.
#pragma unroll
                for (int a = 0; a < PLAIN_STAGE; ++a) {
                    if (a < na) {
                        const cplx<T> xt = X[a * PLAIN_THREADS + s];
                        const cplx<A> x{A(xt.re), A(xt.im)};
                        acc[a].re = fma(x.re, w.re, fma(-x.im, w.im, acc[a].re));
                        acc[a].im = fma(x.re, w.im, fma(x.im, w.re, acc[a].im));
                    }
                }
            }
        }
#pragma unroll
        for (int a = 0; a < PLAIN_STAGE; ++a)
            if (a < na) P[(split * PLAIN_STAGE + a) * cw + cl] = acc[a];
        __syncthreads();
        const int nsplit = PLAIN_THREADS / cw;
        if (t < na * cw) {
            const int a = t / cw, c2 = t % cw;
            cplx<A> s{A(0), A(0)};
            for (int j = 0; j < nsplit; ++j) {
                cplx<A> v = P[(j * PLAIN_STAGE + a) * cw + c2];
                s.re = s.re + v.re;
                s.im = s.im + v.im;
            }
            if (c2 < left) out[(int64_t)a * nc + cg + c2] = s;
        }
        __syncthreads();
    }
}

template <typename T>
size_t segment_smem_bytes(int32_t nc) {
    size_t bytes = sizeof(NodeCache<T>) + 2 * sizeof(cplx<T>) * PLAIN_STAGE * PLAIN_THREADS;
    size_t csm_bytes = sizeof(cplx<T>) * (size_t)nc * PLAIN_THREADS;
    if (csm_bytes <= 128 * 1024) bytes += csm_bytes;
    return (bytes + 127) & ~size_t(127);
}

// Excitation kernel.  One thread per spin; all threads of a CTA walk the same
// node range in lockstep, so ADC staging and the coil reduction are
// CTA-uniform.  Per node a hard-pulse spinor
// (BlochHighOrderSimulatitonMethod.jl:100-134; kernels/HighOrderGPU.jl:181-192).
// ADC: the launch acquires samples (256 threads, the coil reduction's shape).
// Else (FP32 only; FP64 pulses without samples run in homs_excite64.cu) the node
// cache is all it holds, CTAs of 64 threads spread the warps evenly over the
// SMs, and the spinors of UNROLL nodes, which do not depend on the state, are
// formed together before they are applied.  Bound by latency and issue (about
// 150 unfused instructions per node in a chain of square root, sine, reciprocal
// and complex products): 29,929 spins x 64 nodes 27.3 -> 24.8 us.  The
// operations and their order stay the reference's: FP32 roundings of a pulse's
// nodes add up in one direction, and the rotation form of homs_excite64.cu, though
// more exact, ends 4e-5 away from them after 48 pulses.
template <typename T, bool ADC>
__global__ void __launch_bounds__(ADC ? PLAIN_THREADS : 64, ADC ? 3 : 8)
    excitation_kernel(PhantomDev<T> p, SeqDev<T> q, StateDev<T> st, SegmentArgs<T> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    NodeCache<T> &nc = *reinterpret_cast<NodeCache<T> *>(smem_raw);
    cplx<T> *X = reinterpret_cast<cplx<T> *>(smem_raw + ((sizeof(NodeCache<T>) + 15) & ~size_t(15)));
    cplx<T> *P = X + PLAIN_STAGE * PLAIN_THREADS;
    cplx<T> *csm_s = P + PLAIN_STAGE * PLAIN_THREADS;

    const int64_t spin0 = (int64_t)blockIdx.x * blockDim.x;
    const int64_t s = spin0 + threadIdx.x;
    const bool active = s < p.ns;
    const int nvalid = (int)imin64(PLAIN_THREADS, p.ns - spin0);
    const int32_t ncoil = p.nc;
    const bool csm_in_smem = ADC && sizeof(cplx<T>) * (size_t)ncoil * PLAIN_THREADS <= 128 * 1024;

    // Stage this CTA's sensitivities (rows s, coil-fastest).
    const cplx<T> *csm_rows;
    int csm_ld = ncoil;
    if (csm_in_smem) {
        const int64_t total = (int64_t)nvalid * ncoil;
        for (int64_t i = threadIdx.x; i < total; i += PLAIN_THREADS) csm_s[i] = p.csm[spin0 * ncoil + i];
        csm_rows = csm_s;
    } else {
        csm_rows = p.csm + spin0 * ncoil;
    }

    const uint32_t m = a.method;
    const T gamma = a.gamma;
    // Constants converted from FP64 exactly as the reference's T(2π*γ).
    const double twopig_d = 2.0 * 3.141592653589793 * a.gamma_d;
    const T c_twopig = T(twopig_d);
    const T c_neg = T(-twopig_d);

    const int64_t si = active ? s : 0;
    const T px = p.x[si], py = p.y[si], pz = p.z[si];
    const T T1 = p.T1[si], T2 = p.T2[si], rho = p.rho[si];
    cplx<T> xy = active ? st.xy[si] : cplx<T>{T(0), T(0)};
    T mz = active ? st.z[si] : T(0);

    const T off = (m & HOMS_DW_EXCITATION) ? p.dw[si] / c_twopig : T(0);

    T dt_rel = T(-1), e1_rel = T(0), e2_rel = T(0);  // RF relaxation factors of the last dt
    int staged = 0;
    int64_t sample = 0;
    cplx<T> *out_base = a.partial + (int64_t)blockIdx.x * a.nsamples * ncoil;

    for (int64_t c0 = a.n_lo; c0 < a.n_hi; c0 += NODE_CHUNK) {
        __syncthreads();
        load_nodes<T>(nc, q, c0, a.n_hi, gamma);
        __syncthreads();
        const int nint = (int)imin64(NODE_CHUNK, a.n_hi - c0);
        if (c0 == a.n_lo && a.block_start) {
            T sn, cs;
            Math<T>::sc(-nc.psi[0], &sn, &cs);
            xy = cmul(xy, cplx<T>{cs, sn});
        }
        // Spinor of the interval that starts at cached node i.
        auto spinor = [&](int i, cplx<T> &al, cplx<T> &be) {
            const T dbz = off - nc.dfg[i];
            const T bz = ((nc.g[0][i] * px + nc.g[1][i] * py) + nc.g[2][i] * pz) + dbz;
            const cplx<T> b1 = nc.b1[i];
            const T ab1 = nc.ab1[i];
            T B = Math<T>::sq(ab1 * ab1 + bz * bz);
            if (B == T(0)) B = Math<T>::eps();
            const T phi = c_neg * (B * nc.dt[i]);
            T sh, ch;
            Math<T>::sc(phi / T(2), &sh, &ch);
            // Unit field direction (one reciprocal; within an ulp of three divisions).
            const T rB = T(1) / B;
            const T nz = bz * rB, nxr = b1.re * rB, nxi = b1.im * rB;
            al = cplx<T>{ch, -(nz * sh)};
            be = cplx<T>{nxi * sh, -(nxr * sh)};
        };
        // Rotation by the spinor, then relaxation over the interval.
        auto apply = [&](int i, const cplx<T> &al, const cplx<T> &be) {
            const T dt = nc.dt[i];
            cplx<T> t1 = cmul(cplx<T>{T(2) * al.re, -(T(2) * al.im)}, be);
            t1.re = t1.re * mz;
            t1.im = t1.im * mz;
            const cplx<T> ca{al.re, -al.im};
            const cplx<T> t2 = cmul(cmul(ca, ca), xy);
            const cplx<T> t3 = cmul(cmul(be, be), cplx<T>{xy.re, -xy.im});
            const cplx<T> nxy{(t1.re + t2.re) - t3.re, (t1.im + t2.im) - t3.im};
            // |alpha|^2 - |beta|^2 as sums of squares (the reference's abs2;
            // within an ulp of hypot()^2).
            const T aa2 = al.re * al.re + al.im * al.im, bb2 = be.re * be.re + be.im * be.im;
            const cplx<T> pr = cmul(cmul(al, be), cplx<T>{xy.re, -xy.im});
            const T nz2 = (aa2 - bb2) * mz - T(2) * pr.re;
            // Relaxation factors depend on dt only: reuse them while dt repeats.
            if (!(dt == dt_rel)) {
                e2_rel = Math<T>::ex(-dt / T2);
                e1_rel = Math<T>::ex(-dt / T1);
                dt_rel = dt;
            }
            xy = cplx<T>{nxy.re * e2_rel, nxy.im * e2_rel};
            mz = nz2 * e1_rel + rho * (T(1) - e1_rel);
        };
        // Block end: leave the frame of psi, and enter it again for the next block.
        auto frame = [&](int i) {
            if (nc.bnd[i + 1]) {
                T sn, cs;
                Math<T>::sc(nc.psi[i + 1], &sn, &cs);
                xy = cmul(xy, cplx<T>{cs, sn});
                if (c0 + i + 1 < a.n_hi) {
                    Math<T>::sc(-nc.psi[i + 1], &sn, &cs);
                    xy = cmul(xy, cplx<T>{cs, sn});
                }
            }
        };
        if (ADC) {
            for (int i = 0; i < nint; ++i) {
                cplx<T> al, be;
                spinor(i, al, be);
                apply(i, al, be);
                if (nc.adc[i + 1]) {
                    T sn, cs;
                    Math<T>::sc(nc.psi[i + 1], &sn, &cs);
                    const cplx<T> xs = cmul(xy, cplx<T>{cs, sn});
                    X[staged * PLAIN_THREADS + threadIdx.x] = active ? xs : cplx<T>{T(0), T(0)};
                    staged++;
                    if (staged == PLAIN_STAGE) {
                        __syncthreads();
                        reduce_stage(X, P, staged, csm_rows, csm_ld, nvalid, ncoil, out_base + sample * ncoil);
                        sample += staged;
                        staged = 0;
                    }
                }
                frame(i);
            }
        } else {
            constexpr int UNROLL = 4;
            int i = 0;
            for (; i + UNROLL <= nint; i += UNROLL) {
                cplx<T> al[UNROLL], be[UNROLL];
#pragma unroll
                for (int u = 0; u < UNROLL; ++u) spinor(i + u, al[u], be[u]);
#pragma unroll
                for (int u = 0; u < UNROLL; ++u) {
                    apply(i + u, al[u], be[u]);
                    frame(i + u);
                }
            }
            for (; i < nint; ++i) {
                cplx<T> al, be;
                spinor(i, al, be);
                apply(i, al, be);
                frame(i);
            }
        }
    }
    if (ADC && staged > 0) {
        __syncthreads();
        reduce_stage(X, P, staged, csm_rows, csm_ld, nvalid, ncoil, out_base + sample * ncoil);
    }
    if (active) {
        st.xy[s] = xy;
        st.z[s] = mz;
    }
}

// Short precession segments: one thread per spin walks the nodes, field, phase sum,
// sine, cosine and decay as they come (BlochHighOrderSimulatitonMethod.jl:54-92, in
// the CPU order), samples staged and contracted as in the excitation kernel, but
// summed in FP64 for either type (as the parallel kernels sum).
// Against the kernels that are parallel over samples (homs_precess64.cu,
// homs_precess32.cu) it needs no tables and pads no sample tile, and its time grows
// by every node: precession_is_short has the line between them.
template <typename T>
struct FieldCache {
    T dt[NODE_CHUNK + 1];
    T f[16][NODE_CHUNK + 1];  // field coefficients; 1..3: the nominal gradients where the first order is off
    uint8_t adc[NODE_CHUNK + 1];
    uint8_t bnd[NODE_CHUNK + 1];
};

// Bz at cached node i (BlochHighOrderSimulatitonMethod.jl:70-75).
template <typename T>
__device__ __forceinline__ T field_cached(const FieldCache<T> &nc, int i, const T *b, T dwterm, uint32_t m) {
    const T bz1 = (b[1] * nc.f[1][i] + b[2] * nc.f[2][i]) + b[3] * nc.f[3][i];
    T bz = ((m & HOMS_HO0) ? nc.f[0][i] : T(0)) + bz1;
    if (m & HOMS_HO2) {
        T t = b[4] * nc.f[4][i];
#pragma unroll
        for (int k = 5; k <= 8; ++k) t = t + b[k] * nc.f[k][i];
        bz = bz + t;
    }
    if (m & HOMS_HO3) {
        T t = b[9] * nc.f[9][i];
#pragma unroll
        for (int k = 10; k <= 15; ++k) t = t + b[k] * nc.f[k][i];
        bz = bz + t;
    }
    return (m & HOMS_DW_PRECESSION) ? bz + dwterm : bz;
}

template <typename T>
__global__ void __launch_bounds__(PLAIN_THREADS, sizeof(T) == 4 ? 3 : 2)
    short_kernel(PhantomDev<T> p, SeqDev<T> q, StateDev<T> st, SegmentArgs<T> a, cplx<double> *partial) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FieldCache<T> &nc = *reinterpret_cast<FieldCache<T> *>(smem_raw);
    cplx<T> *X = reinterpret_cast<cplx<T> *>(smem_raw + ((sizeof(FieldCache<T>) + 15) & ~size_t(15)));
    cplx<double> *P = reinterpret_cast<cplx<double> *>(X + PLAIN_STAGE * PLAIN_THREADS);
    const int64_t spin0 = (int64_t)blockIdx.x * PLAIN_THREADS, s = spin0 + threadIdx.x;
    const bool active = s < p.ns;
    const int64_t si = active ? s : 0;
    const int nvalid = (int)imin64(PLAIN_THREADS, p.ns - spin0);
    const uint32_t m = a.method;
    const double twopig_d = 2.0 * 3.141592653589793 * a.gamma_d;
    const T c_neg = T(-twopig_d), dwterm = p.dw[si] / T(twopig_d);
    const T x = p.x[si], y = p.y[si], z = p.z[si], T1 = p.T1[si], T2 = p.T2[si], rho = p.rho[si];
    const T x2 = x * x, y2 = y * y, z2 = z * z, r2 = (x2 + y2) + z2;
    const T b[16] = {T(1), x, y, z, x * y, z * y, T(3) * z2 - r2, x * z, x2 - y2, (T(3) * y) * x2 - (y2 * y), (x * z) * y,
                     (T(5) * z2 - r2) * y, T(5) * (z2 * z) - (T(3) * z) * r2, (T(5) * z2 - r2) * x, x2 * z - y2 * z,
                     (x2 * x) - (T(3) * x) * y2};
    cplx<T> xy = active ? st.xy[si] : cplx<T>{T(0), T(0)};
    T mz = active ? st.z[si] : T(0);
    T acc = T(0), tp = T(0), prev = T(0);
    int staged = 0;
    int64_t sample = 0;
    cplx<double> *out_base = partial + (int64_t)blockIdx.x * a.nsamples * p.nc;
    auto reduce = [&] {
        __syncthreads();
        reduce_stage(X, P, staged, p.csm + spin0 * p.nc, p.nc, nvalid, p.nc, out_base + sample * p.nc);
        sample += staged;
        staged = 0;
    };
    for (int64_t c0 = a.n_lo; c0 < a.n_hi; c0 += NODE_CHUNK) {
        const int nint = (int)imin64(NODE_CHUNK, a.n_hi - c0);
        __syncthreads();
        for (int i = threadIdx.x; i < 16 * (NODE_CHUNK + 1); i += PLAIN_THREADS) {
            const int k = i / (NODE_CHUNK + 1), n = i % (NODE_CHUNK + 1);
            const int64_t g = c0 + n;
            if (n > nint) continue;
            const T *f = q.h[k];
            if (k >= 1 && k <= 3 && !(m & HOMS_HO1)) f = k == 1 ? q.gx : k == 2 ? q.gy : q.gz;
            nc.f[k][n] = f[g];
            if (k == 0) {
                nc.dt[n] = n < nint ? q.dt[g] : T(0);
                nc.adc[n] = q.adc[g];
                nc.bnd[n] = q.boundary[g];
            }
        }
        __syncthreads();
        if (c0 == a.n_lo) prev = field_cached(nc, 0, b, dwterm, m);
        for (int i = 0; i < nint; ++i) {
            const T next = field_cached(nc, i + 1, b, dwterm, m);
            acc = acc + (next + prev) * nc.dt[i];
            tp = tp + nc.dt[i];
            prev = next;
            if (!nc.adc[i + 1] && !nc.bnd[i + 1]) continue;
            T sn, cs;
            Math<T>::sc(c_neg * (T(0.5) * acc), &sn, &cs);
            const T e = Math<T>::ex(T(0) - tp / T2);
            const cplx<T> xs = cmul(xy, cplx<T>{e * cs, e * sn});
            if (nc.adc[i + 1]) {
                X[staged * PLAIN_THREADS + threadIdx.x] = active ? xs : cplx<T>{T(0), T(0)};
                if (++staged == PLAIN_STAGE) reduce();
            }
            if (nc.bnd[i + 1]) {  // Mxy of the block's last node, Mz relaxed over it, the phase sum restarts
                xy = xs;
                const T e1 = Math<T>::ex(-tp / T1);
                mz = mz * e1 + rho * (T(1) - e1);
                acc = T(0);
                tp = T(0);
            }
        }
    }
    if (staged > 0) reduce();
    if (active) {
        st.xy[s] = xy;
        st.z[s] = mz;
        if (sizeof(T) == 4) st.acc[s] = acc;  // a later round of the run starts from it
    }
}

// sig[(j) + c*ldsig] = sum over parts k of partial[(k*nsamples + j)*nc + c].
// A block takes 32 consecutive outputs; warp q of its FIN_SLICES sums the parts
// k = q, q + FIN_SLICES, ... in increasing order (coalesced: 32 outputs of one
// part per load), then warp 0 adds those sums in warp order.  The order depends
// only on nparts, so repeated runs are bit-identical.  Bound by the latency of
// a warp's chain of loads: 32 slices from 64 parts on (1,024 outputs of 296
// parts: 12.5 us with 8 slices, 6.8 us with 32), 8 below, where most of 32
// warps would have nothing to add.
constexpr int FIN_OUT = 32;
template <typename T, typename S, int FIN_SLICES>
__global__ void __launch_bounds__(FIN_OUT *FIN_SLICES)
    partial_finalize_kernel(const cplx<T> *partial, int64_t nparts, int64_t nsamples, int32_t nc, cplx<S> *sig,
                            int64_t ldsig) {
    __shared__ cplx<T> red[FIN_SLICES][FIN_OUT];
    const int64_t total = nsamples * nc;
    const int ol = threadIdx.x % FIN_OUT, q = threadIdx.x / FIN_OUT;
    for (int64_t o0 = (int64_t)blockIdx.x * FIN_OUT; o0 < total; o0 += (int64_t)gridDim.x * FIN_OUT) {
        const int64_t o = o0 + ol;
        cplx<T> acc{T(0), T(0)};
        if (o < total)
            for (int64_t k = q; k < nparts; k += FIN_SLICES) {
                const cplx<T> v = partial[k * total + o];
                acc.re = acc.re + v.re;
                acc.im = acc.im + v.im;
            }
        red[q][ol] = acc;
        __syncthreads();
        if (q == 0 && o < total) {
            cplx<T> s = red[0][ol];
            for (int qq = 1; qq < FIN_SLICES; ++qq) {
                s.re = s.re + red[qq][ol].re;
                s.im = s.im + red[qq][ol].im;
            }
            const int64_t jj = o / nc;
            const int32_t c = (int32_t)(o % nc);
            sig[jj + (int64_t)c * ldsig] = cplx<S>{S(s.re), S(s.im)};
        }
        __syncthreads();
    }
}

// Standalone coil reduction (states^T csm, no conjugation), split-K over spin
// ranges.  CTA (p, jt, ct) sums the p-th range of 32-spin chunks for samples
// 8 WJ jt .. and coils 8 NT ct .. into its partial block.  Both operands are
// column-major, so a chunk is a set of short rows (32 consecutive spins of a
// sample or of a coil), staged by asynchronous copies a chunk ahead, and the
// product is taken by FP64 matrix instructions (m8n8k4, samples x spins times
// spins x coils; FP32 operands are widened, their products and sums kept in
// FP64).  Warp w takes the tile's samples 8 (w % WJ) .. +7; the 8 / WJ warps that
// share them split a chunk's spins and are added at the end in warp order.
//
// What bounds it: for many coils the FP64 pipe, 4 multiply-adds per spin, sample
// and coil (FP32: 3, by three products, whose extra rounding is lost in FP64; in
// FP64 they would raise the error from 2.65e-15 to 2.78e-15), 91 us at its peak for
// 200,000 x 64 x 32 in FP64; for few, memory.  Measured (B200, with the finalize;
// against register-blocked multiply-adds from shared memory, which spent their
// issue slots on loads): 200,000 x 64 x 32 FP64 200 -> 138 us, FP32 121 -> 111;
// 200,000 x 64 x 8 FP64 188 -> 59; 200,000 x 96 x 1 FP32 205 -> 80; 30,011 x 33 x 31
// FP64 47 -> 35; 5,000 x 17 x 3 FP64 41 -> 10.  Chunks of 16 spins in 3 stages: 142 us
// for the first; 32 in 3, which leaves one CTA per SM: 171.
constexpr int CR_SK = 32, CR_THREADS = 256, CR_CTAS_PER_SM = 2, CR_STAGES = 2;
// Bytes of a staged row (CR_SK spins and a pad that keeps fragment loads conflict-free).
template <typename T>
constexpr int cr_row() {
    return (int)sizeof(cplx<T>) * CR_SK + (sizeof(T) == 8 ? 64 : 32);
}
template <typename T>
constexpr int cr_stage(int nt, int wj) {
    return 8 * (nt + wj) * cr_row<T>();
}
// P: type of the partial sums.
template <typename T, typename P, int NT, int WJ>
__global__ void __launch_bounds__(CR_THREADS, CR_CTAS_PER_SM)
    coil_reduce_kernel(int64_t ns, int64_t nadc, int32_t nc, const cplx<T> *states, int64_t ldstates,
                       const cplx<T> *csm, int64_t ldcsm, int64_t parts, int width, cplx<P> *partial) {
    using Pair = std::conditional_t<sizeof(T) == 8, double2, float2>;
    constexpr int ROW = cr_row<T>(), STAGE = cr_stage<T>(NT, WJ), KS = 8 / WJ, JB = 8 * WJ, CB = 8 * NT;
    extern __shared__ __align__(16) uint8_t cr_smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = lane & 3, r = lane >> 2;
    const int wj = warp % WJ, kw = warp / WJ;
    const int64_t p = blockIdx.x, j0 = (int64_t)blockIdx.y * JB;
    const int c0 = (int)blockIdx.z * CB;
    const int jn = (int)imin64(JB, nadc - j0), cn = (int)imin64(CB, nc - c0);
    const int64_t nch = (ns + CR_SK - 1) / CR_SK, ch0 = nch * p / parts, ch1 = nch * (p + 1) / parts;
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(cr_smem);
    // Rows past the last sample or coil are zero in every stage.
    for (int i = tid; i < CR_STAGES * STAGE / 16; i += CR_THREADS) {
        const int row = i % (STAGE / 16) / (ROW / 16);
        if (row < JB ? row >= jn : row - JB >= cn)
            *reinterpret_cast<float4 *>(cr_smem + (size_t)i * 16) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    // One chunk into a stage, in pieces of `width` bytes (the alignment that the
    // operands have); spins past the last one are zero.
    const int pieces = CR_SK * (int)sizeof(cplx<T>) / width;  // per row: a power of two
    const int shift = 31 - __clz(pieces);
    auto issue = [&](int64_t ch, int stage) {
        const int64_t s0 = ch * CR_SK;
        const int64_t left = (ns - s0) * (int64_t)sizeof(cplx<T>);  // bytes of the rows from here on
        for (int i = tid; i < (jn + cn) << shift; i += CR_THREADS) {
            const int k = i >> shift, at = (i & (pieces - 1)) * width;
            const char *src = reinterpret_cast<const char *>(k < jn ? states + (j0 + k) * ldstates + s0
                                                                    : csm + (int64_t)(c0 + k - jn) * ldcsm + s0);
            const uint32_t dst = sbase + (uint32_t)(stage * STAGE + (k < jn ? k : JB + k - jn) * ROW + at);
            const int n = (int)imax64(0, imin64(width, left - at));
            if (n > 0) src += at;
            if (width == 16)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
            else if (width == 8)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
            else
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
        }
    };
    double re[NT][2], im[NT][2], k3[NT][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) re[nt][e] = im[nt][e] = k3[nt][e] = 0.0;
#pragma unroll
    for (int s = 0; s < CR_STAGES - 1; ++s) {
        if (ch0 + s < ch1) issue(ch0 + s, s);
        cp_commit();
    }
    int stage = 0;
    for (int64_t ch = ch0; ch < ch1; ++ch) {
        cp_wait<CR_STAGES - 2>();
        __syncthreads();
        if (ch + CR_STAGES - 1 < ch1) issue(ch + CR_STAGES - 1, stage == 0 ? CR_STAGES - 1 : stage - 1);
        cp_commit();
        const uint8_t *st = cr_smem + stage * STAGE;
        if (++stage == CR_STAGES) stage = 0;
#pragma unroll
        for (int k = 0; k < CR_SK / 4; k += KS) {
            const int at = (4 * (k + kw) + q) * (int)sizeof(cplx<T>);
            const auto x = *reinterpret_cast<const Pair *>(st + (8 * wj + r) * ROW + at);
            const double xr = x.x, xi = x.y;
            double wr[NT], wi[NT];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const auto w = *reinterpret_cast<const Pair *>(st + (JB + 8 * nt + r) * ROW + at);
                wr[nt] = w.x;
                wi[nt] = w.y;
            }
            if (sizeof(T) == 8) {
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) dmma(re[nt], xr, wr[nt]);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) dmma(im[nt], xr, wi[nt]);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) dmma(re[nt], -xi, wi[nt]);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) dmma(im[nt], xi, wr[nt]);
            } else {
                // three products: Re = k1 - k3, Im = k1 + k2
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    dmma(re[nt], xr + xi, wr[nt]);
                    dmma(im[nt], xr, wi[nt] - wr[nt]);
                    dmma(k3[nt], xi, wr[nt] + wi[nt]);
                }
            }
        }
    }
    cp_wait<0>();
    if (sizeof(T) == 4) {
        int top = 0;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) from_three(re[nt][e], im[nt][e], k3[nt][e], top);
        // Infinite operands: this warp's sums by four products, straight from memory.
        if (__any_sync(0xffffffffu, top >= NOT_FINITE)) {
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) re[nt][e] = im[nt][e] = 0.0;
            const bool row = 8 * wj + r < jn;
#pragma unroll 1
            for (int64_t k = (CR_SK / 4) * ch0 + kw; k < (CR_SK / 4) * ch1; k += KS) {
                const int64_t s = 4 * k + q;
                const bool ok = s < ns;
                const cplx<T> x = row && ok ? states[(j0 + 8 * wj + r) * ldstates + s] : cplx<T>{T(0), T(0)};
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const int c = 8 * nt + r;
                    const cplx<T> w = c < cn && ok ? csm[(c0 + c) * ldcsm + s] : cplx<T>{T(0), T(0)};
                    dmma4(re[nt], im[nt], x.re, x.im, w.re, w.im);
                }
            }
        }
    }
    if (KS > 1) {  // add the warps that share the samples, in warp order
        double *sums = reinterpret_cast<double *>(cr_smem);
        __syncthreads();
        if (kw > 0)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    double *d = sums + ((((kw - 1) * WJ + wj) * NT + nt) * 2 + e) * 64 + lane;
                    d[0] = re[nt][e];
                    d[32] = im[nt][e];
                }
        __syncthreads();
        if (kw > 0) return;
        for (int k = 0; k < KS - 1; ++k)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const double *d = sums + (((k * WJ + wj) * NT + nt) * 2 + e) * 64 + lane;
                    re[nt][e] += d[0];
                    im[nt][e] += d[32];
                }
    }
    const int j = 8 * wj + r;
    if (j < jn) {
        cplx<P> *out = partial + (p * nadc + j0 + j) * nc + c0;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int c = 8 * nt + 2 * q + e;
                if (c < cn) out[c] = cplx<P>{(P)re[nt][e], (P)im[nt][e]};
            }
    }
}

template <typename T>
cudaError_t launch_excitation(const PhantomDev<T> &p, const SeqDev<T> &q, StateDev<T> &st, const SegmentArgs<T> &a,
                              int grid, cudaStream_t stream) {
    if (a.nsamples == 0) {
        if constexpr (sizeof(T) == 8) {
            return launch_excite64(p, q, st, a, stream);
        } else {
            excitation_kernel<T, false><<<(unsigned)((p.ns + 63) / 64), 64, sizeof(NodeCache<T>), stream>>>(p, q, st, a);
            return cudaGetLastError();
        }
    }
    cudaError_t e = allow_max_dynamic_smem((const void *)excitation_kernel<T, true>);
    if (e != cudaSuccess) return e;
    excitation_kernel<T, true><<<grid, PLAIN_THREADS, segment_smem_bytes<T>(p.nc), stream>>>(p, q, st, a);
    return cudaGetLastError();
}

// Nodes, and more so samples and coils, cost the sequential kernel time; the
// parallel kernels pay per segment: three or four launches, a sample tile of which
// few rows are used, and in a block call the tables.  The lines come from sweeps of
// 300 to 1,000,000 spins, 1 to 48 (128) nodes and 1, 3, 8 and 32 coils.  Segments of
// prepared runs with a pulse of one node each, parallel and sequential: FP32, 3,000
// spins x 8 coils, 8 nodes with 4 samples 34 and 28 us, 32 with 32 38 and 43; 200,000
// x 8, 8 with 4 75 and 45, 48 with 24 90 and 104; FP64 the same 40 and 30, 41 and 50,
// 104 and 59, 104 and 140.  Block calls, every node a sample: FP32, 3,000 x 8, 16
// nodes 66 and 48, 48 nodes 68 and 71; 200,000 x 8, 16 nodes 117 and 93, 32 nodes 124
// and 136; FP64 59 and 49, 59 and 77, 136 and 111, 140 and 167.  Where the rule takes
// the sequential kernel, it is the faster one; on the other side it would have been by
// up to 0.2 of the time (FP64 x 1,000,000 spins: 0.34).
bool precession_is_short(int64_t ns, int32_t nc, int64_t nodes, int64_t nsamples, bool f64, bool block_call) {
    if (nsamples == 0) return nodes <= (block_call ? 16 : 4);
    static constexpr int limit[2][2][3] = {{{84, 168, 108}, {256, 264, 152}},    // FP32: prepared, block call
                                           {{140, 212, 104}, {176, 248, 128}}};  // FP64
    return 2 * nodes + 5 * nsamples + 3 * (int64_t)nc <= limit[f64][block_call][ns <= 16384 ? 0 : ns <= 100000 ? 1 : 2];
}

template <typename T>
cudaError_t launch_short(const PhantomDev<T> &p, const SeqDev<T> &q, StateDev<T> &st, const SegmentArgs<T> &a,
                         cplx<double> *partial, int grid, cudaStream_t stream) {
    // Node cache, staged samples and the reduction's sums: 52 KB in FP32, 71 KB in FP64.
    size_t smem = (sizeof(FieldCache<T>) + 15) & ~size_t(15);
    if (a.nsamples > 0) smem += (sizeof(cplx<T>) + sizeof(cplx<double>)) * PLAIN_STAGE * PLAIN_THREADS;
    const cudaError_t e = allow_max_dynamic_smem((const void *)short_kernel<T>);
    if (e != cudaSuccess) return e;
    short_kernel<T><<<grid, PLAIN_THREADS, smem, stream>>>(p, q, st, a, partial);
    return cudaGetLastError();
}

template <typename T, typename S>
cudaError_t launch_partial_finalize(const cplx<T> *partial, int64_t nparts, int64_t nsamples, int32_t nc,
                                    cplx<S> *sig, int64_t ldsig, cudaStream_t stream) {
    const int64_t total = nsamples * nc;
    if (total == 0) return cudaSuccess;
    const int64_t blocks = std::min<int64_t>((total + FIN_OUT - 1) / FIN_OUT, 148 * 16);
    if (nparts >= 64)
        partial_finalize_kernel<T, S, 32><<<(int)blocks, FIN_OUT * 32, 0, stream>>>(partial, nparts, nsamples, nc, sig,
                                                                                    ldsig);
    else
        partial_finalize_kernel<T, S, 8><<<(int)blocks, FIN_OUT * 8, 0, stream>>>(partial, nparts, nsamples, nc, sig,
                                                                                  ldsig);
    return cudaGetLastError();
}

// Tile of the reduction: 8-coil tiles (1, 2 or 4) and warps along the samples (2,
// 4 or 8), the smallest that take all coils (samples) or the largest.
static int cr_coil_tiles(int32_t nc) { return nc <= 8 ? 1 : nc <= 16 ? 2 : 4; }
static int cr_sample_warps(int64_t nadc) { return nadc <= 16 ? 2 : nadc <= 32 ? 4 : 8; }

// Parts of the split-K: one wave of CR_CTAS_PER_SM CTAs per SM over all (sample, coil)
// tiles, 256 spins per part at least; more parts, of two chunks at least and with
// FP64 partial sums within CR_PARTIAL_BYTES, where that leaves SMs idle: up to the wave
// for the larger tiles, else one CTA per SM (more only add partial sums to read).
// Before, and so (per call, back to back): 8,001 spins x 64 x 32, an odd leading
// dimension, FP32 37 and 19 us, FP64 38 and 19; 4,000 x 48 x 8 FP64 20 and 11.
CoilReduceCut coil_reduce_cut(int64_t ns, int64_t nadc, int32_t nc, bool f64) {
    const int jb = 8 * cr_sample_warps(nadc), cb = 8 * cr_coil_tiles(nc);
    const int64_t tiles = ((nadc + jb - 1) / jb) * ((nc + cb - 1) / cb), wave = 148 * CR_CTAS_PER_SM / tiles;
    const int64_t few = std::max<int64_t>(1, std::min(wave, (ns + PLAIN_THREADS - 1) / PLAIN_THREADS));
    const int64_t more = std::min({jb * cb >= 1024 ? wave : 148 / tiles, CR_PARTIAL_BYTES / (16 * nadc * nc),
                                   (ns + 2 * CR_SK - 1) / (2 * CR_SK)});
    return more > few ? CoilReduceCut{more, true} : CoilReduceCut{few, f64};
}

template <typename T, typename P, int NT, int WJ>
static cudaError_t cr_launch(dim3 grid, int64_t ns, int64_t nadc, int32_t nc, const cplx<T> *states, int64_t ldstates,
                             const cplx<T> *csm, int64_t ldcsm, int width, cplx<P> *partial, cudaStream_t stream) {
    const size_t smem = std::max<size_t>(CR_STAGES * cr_stage<T>(NT, WJ), sizeof(double) * 128 * NT * (8 - WJ));
    cudaError_t e = allow_max_dynamic_smem((const void *)coil_reduce_kernel<T, P, NT, WJ>);
    if (e != cudaSuccess) return e;
    coil_reduce_kernel<T, P, NT, WJ><<<grid, CR_THREADS, smem, stream>>>(ns, nadc, nc, states, ldstates, csm, ldcsm,
                                                                         (int64_t)grid.x, width, partial);
    return cudaGetLastError();
}

template <typename T, typename P>
static cudaError_t cr_run(int64_t parts, int64_t ns, int64_t nadc, int32_t nc, const cplx<T> *states, int64_t ldstates,
                          const cplx<T> *csm, int64_t ldcsm, cplx<P> *partial, cplx<T> *sig, int64_t ldsig,
                          cudaStream_t stream) {
    const int nt = cr_coil_tiles(nc), wj = cr_sample_warps(nadc);
    const int64_t jt = (nadc + 8 * wj - 1) / (8 * wj), ct = (nc + 8 * nt - 1) / (8 * nt);
    if (jt > 65535 || ct > 65535) return cudaErrorInvalidValue;
    const dim3 grid((unsigned)parts, (unsigned)jt, (unsigned)ct);
    // Widest copy that every row of both operands is aligned to.
    const uint64_t bits = reinterpret_cast<uintptr_t>(states) | reinterpret_cast<uintptr_t>(csm) |
                          (uint64_t)ldstates * sizeof(cplx<T>) | (uint64_t)ldcsm * sizeof(cplx<T>);
    const int width = (bits & 15) == 0 ? 16 : (bits & 7) == 0 ? 8 : 4;
    cudaError_t e = cudaErrorInvalidValue;
#define CR_CASE(NT_, WJ_) \
    if (nt == NT_ && wj == WJ_) \
        e = cr_launch<T, P, NT_, WJ_>(grid, ns, nadc, nc, states, ldstates, csm, ldcsm, width, partial, stream);
    CR_CASE(1, 2) CR_CASE(1, 4) CR_CASE(1, 8)
    CR_CASE(2, 2) CR_CASE(2, 4) CR_CASE(2, 8)
    CR_CASE(4, 2) CR_CASE(4, 4) CR_CASE(4, 8)
#undef CR_CASE
    return e != cudaSuccess ? e : launch_partial_finalize(partial, parts, nadc, nc, sig, ldsig, stream);
}

template <typename T>
cudaError_t launch_coil_reduce(const CoilReduceCut &cut, int64_t ns, int64_t nadc, int32_t nc, const cplx<T> *states,
                               int64_t ldstates, const cplx<T> *csm, int64_t ldcsm, void *partial, cplx<T> *sig,
                               int64_t ldsig, cudaStream_t stream) {
    if (ns == 0 || nadc == 0 || nc == 0) return cudaSuccess;
    if (cut.wide)
        return cr_run<T, double>(cut.parts, ns, nadc, nc, states, ldstates, csm, ldcsm,
                                 static_cast<cplx<double> *>(partial), sig, ldsig, stream);
    if constexpr (sizeof(T) == 4)
        return cr_run<T, float>(cut.parts, ns, nadc, nc, states, ldstates, csm, ldcsm,
                                static_cast<cplx<float> *>(partial), sig, ldsig, stream);
    return cudaErrorInvalidValue;
}

// Load every kernel of the reduction and of its partial sums on the current device
// (the driver loads a kernel, and may allocate for it, at its first use).
template <typename T, typename P>
static cudaError_t load_reduce_kernels() {
    const void *const kernels[] = {
        (const void *)coil_reduce_kernel<T, P, 1, 2>, (const void *)coil_reduce_kernel<T, P, 1, 4>,
        (const void *)coil_reduce_kernel<T, P, 1, 8>, (const void *)coil_reduce_kernel<T, P, 2, 2>,
        (const void *)coil_reduce_kernel<T, P, 2, 4>, (const void *)coil_reduce_kernel<T, P, 2, 8>,
        (const void *)coil_reduce_kernel<T, P, 4, 2>, (const void *)coil_reduce_kernel<T, P, 4, 4>,
        (const void *)coil_reduce_kernel<T, P, 4, 8>, (const void *)partial_finalize_kernel<P, T, 8>,
        (const void *)partial_finalize_kernel<P, T, 32>};
    for (const void *k : kernels) {
        cudaFuncAttributes a;
        const cudaError_t e = cudaFuncGetAttributes(&a, k);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}
cudaError_t load_coil_reduce() {
    cudaError_t e = load_reduce_kernels<double, double>();
    if (e == cudaSuccess) e = load_reduce_kernels<float, float>();
    return e != cudaSuccess ? e : load_reduce_kernels<float, double>();
}

template cudaError_t launch_excitation<double>(const PhantomDev<double> &, const SeqDev<double> &, StateDev<double> &,
                                               const SegmentArgs<double> &, int, cudaStream_t);
template cudaError_t launch_excitation<float>(const PhantomDev<float> &, const SeqDev<float> &, StateDev<float> &,
                                              const SegmentArgs<float> &, int, cudaStream_t);
template cudaError_t launch_short<double>(const PhantomDev<double> &, const SeqDev<double> &, StateDev<double> &,
                                          const SegmentArgs<double> &, cplx<double> *, int, cudaStream_t);
template cudaError_t launch_short<float>(const PhantomDev<float> &, const SeqDev<float> &, StateDev<float> &,
                                         const SegmentArgs<float> &, cplx<double> *, int, cudaStream_t);
template cudaError_t launch_partial_finalize<double, double>(const cplx<double> *, int64_t, int64_t, int32_t,
                                                             cplx<double> *, int64_t, cudaStream_t);
template cudaError_t launch_partial_finalize<float, float>(const cplx<float> *, int64_t, int64_t, int32_t,
                                                           cplx<float> *, int64_t, cudaStream_t);
template cudaError_t launch_partial_finalize<double, float>(const cplx<double> *, int64_t, int64_t, int32_t,
                                                            cplx<float> *, int64_t, cudaStream_t);
template cudaError_t launch_coil_reduce<double>(const CoilReduceCut &, int64_t, int64_t, int32_t, const cplx<double> *,
                                                int64_t, const cplx<double> *, int64_t, void *, cplx<double> *, int64_t,
                                                cudaStream_t);
template cudaError_t launch_coil_reduce<float>(const CoilReduceCut &, int64_t, int64_t, int32_t, const cplx<float> *,
                                               int64_t, const cplx<float> *, int64_t, void *, cplx<float> *, int64_t,
                                               cudaStream_t);
template size_t segment_smem_bytes<double>(int32_t);
template size_t segment_smem_bytes<float>(int32_t);

}  // namespace homs
