// RF excitation in FP64 without acquisition during the pulse: one thread per
// spin walks the pulse's nodes.
//
// Per node the magnetisation turns about B = (Re B1, Im B1, Bz) by the angle
// -2 pi gamma |B| dt and relaxes (hard-pulse spinor of
// src/simulation/kernels/HighOrderGPU.jl:181-192 and
// src/simulation/Bloch/BlochHighOrderSimulatitonMethod.jl:100-134).  As a
// rotation of (Mx, My, Mz): with half-angle cosine w and sine v about the unit
// field n, t = q x M and M' = M + w' t + q x t for q = sqrt(2) v n, w' = sqrt(2) w:
// 15 operations where the spinor's complex products take about 60.  w and v / |B|
// are even in |B|, so a small angle needs no root: two series in z = (half-angle)^2
// (no root, reciprocal and quarter-turn reduction: 17.87 -> 15.65 ms for the TR loop
// below).
//
// What bounds it: the FP64 pipe and its latency, about 34 operations per spin and
// node (field 4, z 1, series 8, rotation vector 3, rotation 15, relaxation 3).
// The rotations of UNROLL nodes are formed before they are
// applied, so that only rotation and relaxation are in the spin's dependent
// chain.  CTAs of 64 threads spread an uneven number of warps over the SMs.
//
// Measured (B200, against the spinor kernel of homs_plain.cu): 80,000 spins x 400
// nodes 449 -> 105 us; a TR loop of 35 such pulses with its split-mode readouts
// 28.2 -> 15.7 ms.
#include <algorithm>
#include <type_traits>

#include "homs_common.cuh"
#include "homs_fp64math.cuh"

namespace homs {

namespace excite64 {

constexpr int THREADS = 64;
constexpr int NODES = 64;  // nodes per stage
constexpr int UNROLL = 4;  // rotations formed together (2, 3, 4, 6: 15.78, 15.76, 15.65, 15.87 ms for the TR loop)

// sqrt(2) cos(h) and sqrt(2) sin(h) / h from z = h^2: interpolants at the
// Chebyshev nodes of [0, 1/32] (degree 4) and [0, 5/8] (degree 7), within 1.3e-16
// with their rounded coefficients.
constexpr uint32_t NEAR_HI = 0x3FA00000, MID_HI = 0x3FE40000;  // high words of 1/32 and 5/8
__device__ __forceinline__ void half_near(double z, double &c, double &s) {
    c = 3.504430601676957e-05;
    s = 3.894426466665344e-06;
    c = fma(c, z, -0.0019641846711878626);
    s = fma(s, z, -0.0002805978533901853);
    c = fma(c, z, 0.05892556508959255);
    s = fma(s, z, 0.0117851130189315);
    c = fma(c, z, -0.7071067811865113);
    s = fma(s, z, -0.23570226039551254);
    c = fma(c, z, 1.4142135623730951);
    s = fma(s, z, 1.4142135623730951);
}
__device__ __forceinline__ void half_mid(double z, double &c, double &s) {
    c = -1.6053921180070224e-11;
    s = -1.0715752882141984e-12;
    c = fma(c, z, 2.9522487684836804e-09);
    s = fma(s, z, 2.2709913861981155e-10);
    c = fma(c, z, -3.897192557835503e-07);
    s = fma(s, z, -3.542902614020508e-08);
    c = fma(c, z, 3.507474110389768e-05);
    s = fma(s, z, 3.897193457367114e-06);
    c = fma(c, z, -0.0019641855032917683);
    s = fma(s, z, -0.0002805979290420337);
    c = fma(c, z, 0.058925565098878634);
    s = fma(s, z, 0.011785113019775773);
    c = fma(c, z, -0.7071067811865475);
    s = fma(s, z, -0.23570226039551584);
    c = fma(c, z, 1.4142135623730951);
    s = fma(s, z, 1.4142135623730951);
}
// Any z (infinities and NaN included).
__device__ __forceinline__ void half_far(double z, double &c, double &s) {
    constexpr double SQRT2 = 1.4142135623730951;
    const double r = z < 1e-300 ? 0.0 : rsqrt(z), h = z * r;  // no field: no rotation
    cis_turns(h * (0.5 / 3.141592653589793), c, s);
    c *= SQRT2;
    s *= SQRT2 * r;
}

// Spin-independent part of a node's step (the interval that starts there).
// Its relaxation relative to the stage's first interval dt0: SAME for an equal
// dt; NEAR for one within 1e-9 dt0 (the differences of rounded node times), dt -
// dt0 to first order; OTHER anew.
enum : int { SAME, NEAR, OTHER };
struct alignas(16) Node {  // fields times k = -pi gamma dt (half-angle in radians per tesla)
    double gx, gy, gz, df;  // gradient, -df / gamma
    double b1r, b1i, b2;    // B1, |B1|^2
    double k;
    double dt;  // dt, or dt - dt0 (NEAR)
    int relax;
};
struct Rotation {
    double w, x, y, z;
};

// Relaxation factor over dt0 + d for |d| <= 1e-9 dt0, from e = exp(-dt0 / T) to
// first order in d.  A factor of 0 (T = 0, or far below dt0) or infinity stays:
// its correction is 0 times or minus infinity, and nothing is lost, since exp
// leaves the range of FP64 at |dt0 / T| = 745, where the correction is below 1e-6.
__device__ __forceinline__ double near_factor(double e, double d, double T) {
    const double f = fma(e, -d / T, e);
    return isnan(f) ? e : f;
}

__global__ void __launch_bounds__(THREADS, 9)
    excite_kernel(PhantomDev<double> p, SeqDev<double> q, StateDev<double> st, SegmentArgs<double> a) {
    __shared__ Node nodes[NODES];
    const int64_t s = (int64_t)blockIdx.x * THREADS + threadIdx.x;
    const bool active = s < p.ns;
    const int64_t si = active ? s : 0;
    const double px = p.x[si], py = p.y[si], pz = p.z[si], rho = p.rho[si], T1 = p.T1[si], T2 = p.T2[si];
    const double off = (a.method & HOMS_DW_EXCITATION) ? p.dw[si] / (2.0 * 3.141592653589793 * a.gamma_d) : 0.0;
    double mx = active ? st.xy[si].re : 0.0, my = active ? st.xy[si].im : 0.0, mz = active ? st.z[si] : 0.0;
    auto turn = [&](double psi) {  // Mxy cis(psi)
        double sn, cs;
        sincos(psi, &sn, &cs);
        const double x = mx * cs - my * sn;
        my = mx * sn + my * cs;
        mx = x;
    };
    // The frame of psi: entered at the first block's start and left at the last
    // one's end; the blocks between leave and enter it at the same node.
    if (a.block_start) turn(-q.psi[a.n_lo]);

    // Relaxation over the stage's first interval: factors, rho (1 - e1).
    double e1 = 0.0, e2 = 0.0, c1 = 0.0;
    // Rotations of U nodes: one choice of the half-angle's range for all of them.
    auto rotations = [&](const Node *n, Rotation *r, auto count) {
        constexpr int U = decltype(count)::value;
        double z[U];
        uint32_t top = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            r[u].z = fma(n[u].gx, px, fma(n[u].gy, py, fma(n[u].gz, pz, fma(n[u].k, off, n[u].df))));
            z[u] = fma(r[u].z, r[u].z, n[u].b2);
            top = max(top, (uint32_t)__double2hiint(z[u]));
        }
        double c[U], f[U];
        if (__all_sync(0xffffffffu, top < NEAR_HI)) {
#pragma unroll
            for (int u = 0; u < U; ++u) half_near(z[u], c[u], f[u]);
        } else if (__all_sync(0xffffffffu, top < MID_HI)) {
#pragma unroll
            for (int u = 0; u < U; ++u) half_mid(z[u], c[u], f[u]);
        } else {
#pragma unroll
            for (int u = 0; u < U; ++u) half_far(z[u], c[u], f[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) r[u] = Rotation{c[u], n[u].b1r * f[u], n[u].b1i * f[u], r[u].z * f[u]};
    };
    auto step = [&](const Rotation &r, const Node &n) {
        const double tx = fma(r.y, mz, -(r.z * my)), ty = fma(r.z, mx, -(r.x * mz)), tz = fma(r.x, my, -(r.y * mx));
        const double nx = fma(r.w, tx, mx), ny = fma(r.w, ty, my), nz = fma(r.w, tz, mz);
        double f2 = e2, f1 = e1, g1 = c1;
        if (n.relax != SAME) {
            f2 = n.relax == NEAR ? near_factor(e2, n.dt, T2) : exp(-n.dt / T2);
            f1 = n.relax == NEAR ? near_factor(e1, n.dt, T1) : exp(-n.dt / T1);
            g1 = rho * (1.0 - f1);
        }
        mx = fma(r.y, tz, fma(-r.z, ty, nx)) * f2;
        my = fma(r.z, tx, fma(-r.x, tz, ny)) * f2;
        mz = fma(fma(r.x, ty, fma(-r.y, tx, nz)), f1, g1);
    };
    for (int64_t n0 = a.n_lo; n0 < a.n_hi; n0 += NODES) {
        const int cnt = (int)imin64(NODES, a.n_hi - n0);
        __syncthreads();
        const double dt0 = q.dt[n0];
        for (int i = threadIdx.x; i < cnt; i += THREADS) {
            const int64_t g = n0 + i;
            const cplx<double> b1 = q.b1[g];
            const double dt = q.dt[g], d = dt - dt0;
            const int relax = d == 0.0 ? SAME : fabs(d) <= 1e-9 * dt0 ? NEAR : OTHER;
            const double k = -3.141592653589793 * a.gamma_d * dt, br = k * b1.re, bi = k * b1.im;
            nodes[i] = Node{k * q.gx[g], k * q.gy[g], k * q.gz[g], 3.141592653589793 * q.df[g] * dt, br, bi,
                            br * br + bi * bi, k, relax == NEAR ? d : dt, relax};
        }
        if (n0 == a.n_lo || dt0 != q.dt[n0 - NODES]) {
            e2 = exp(-dt0 / T2);
            e1 = exp(-dt0 / T1);
            c1 = rho * (1.0 - e1);
        }
        __syncthreads();
        constexpr int U = UNROLL;
        int i = 0;
        for (; i + U <= cnt; i += U) {
            Rotation r[U];
            rotations(nodes + i, r, std::integral_constant<int, U>());
#pragma unroll
            for (int u = 0; u < U; ++u) step(r[u], nodes[i + u]);
        }
        for (; i < cnt; ++i) {
            Rotation r[1];
            rotations(nodes + i, r, std::integral_constant<int, 1>());
            step(r[0], nodes[i]);
        }
    }
    if (q.boundary[a.n_hi]) turn(q.psi[a.n_hi]);
    if (active) {
        st.xy[s] = cplx<double>{mx, my};
        st.z[s] = mz;
    }
}

}  // namespace excite64

cudaError_t launch_excite64(const PhantomDev<double> &p, const SeqDev<double> &q, StateDev<double> &st,
                            const SegmentArgs<double> &a, cudaStream_t stream) {
    const int64_t grid = (p.ns + excite64::THREADS - 1) / excite64::THREADS;
    excite64::excite_kernel<<<(unsigned)grid, excite64::THREADS, 0, stream>>>(p, q, st, a);
    return cudaGetLastError();
}

}  // namespace homs
