// Per-site operations of the two fused RK4 sweeps (see rk4_level.cu for the
// two-sweep factorisation of classic RK4) and their host-side constants,
// shared by the single-level and the ensemble advance.
#pragma once

#include "sweep.cuh"

namespace axs {

// Two sites of sweep A with packed FP32 (the arithmetic of stage_a below): the
// increments d3, d4 with what E and Q are made of, and E, Q themselves, apart
// because the halo sites of the one-pass step need d3, d4 only.
struct StageAPair {
    F2 d[4];                // d3_1, d3_2, d4_1, d4_2
    F2 f11, f12, f21, f22;  // F1, F2
    F2 hq1, hq2;            // h Pi
};
template <bool COMP>
__device__ __forceinline__ StageAPair stage_a_pair(const SweepArgs<float> &a, F2 p1, F2 p2, F2 q1, F2 q2, F2 l0, F2 l1,
                                                   F2 l2, F2 l3)
{
    StageAPair s;
    const F2 hh(a.h_half);
    rhs_pair(a.c1, p1, p2, l0, l1, s.f11, s.f12);
    if constexpr (!COMP) {
        const F2 c1 = fma(hh, q1, p1), c2 = fma(hh, q2, p2);
        rhs_pair(a.c2, c1, c2, fma(hh, l2, l0), fma(hh, l3, l1), s.f21, s.f22);
        s.hq1 = F2(a.h) * q1;
        s.hq2 = F2(a.h) * q2;
        s.d[0] = fma(F2(a.h2_quarter), s.f11, hh * q1);
        s.d[1] = fma(F2(a.h2_quarter), s.f12, hh * q2);
        s.d[2] = fma(F2(a.h2_half), s.f21, s.hq1);
        s.d[3] = fma(F2(a.h2_half), s.f22, s.hq2);
    } else {
        auto cm = [](F2 c, F2 cl, F2 x, F2 y) { return fma(cl, x, fma(c, x, y)); };  // (c + c_lo) x + y
        const F2 hhl(a.h_half_lo), z(0.f, 0.f);
        const F2 c1 = cm(hh, hhl, q1, p1), c2 = cm(hh, hhl, q2, p2);
        rhs_pair(a.c2, c1, c2, cm(hh, hhl, l2, l0), cm(hh, hhl, l3, l1), s.f21, s.f22);
        s.hq1 = cm(F2(a.h), F2(a.h_lo), q1, z);
        s.hq2 = cm(F2(a.h), F2(a.h_lo), q2, z);
        const F2 hhq1 = cm(hh, hhl, q1, z), hhq2 = cm(hh, hhl, q2, z);
        const F2 H2Q(a.h2_quarter), H2Ql(a.h2_quarter_lo), H2H(a.h2_half), H2Hl(a.h2_half_lo);
        s.d[0] = cm(H2Q, H2Ql, s.f11, hhq1);
        s.d[1] = cm(H2Q, H2Ql, s.f12, hhq2);
        s.d[2] = cm(H2H, H2Hl, s.f21, s.hq1);
        s.d[3] = cm(H2H, H2Hl, s.f22, s.hq2);
    }
    return s;
}
template <bool COMP>
__device__ __forceinline__ void stage_a_eq(const SweepArgs<float> &a, const StageAPair &s, F2 l0, F2 l1, F2 (&eq)[4])
{
    const F2 hh(a.h_half);
    if constexpr (!COMP) {
        eq[0] = fma(F2(a.h2_sixth), (s.f11 + s.f21) + l0, s.hq1);
        eq[1] = fma(F2(a.h2_sixth), (s.f12 + s.f22) + l1, s.hq2);
        eq[2] = fma(hh, l0, fma(F2(a.h_third), s.f21, F2(a.h_sixth) * s.f11));
        eq[3] = fma(hh, l1, fma(F2(a.h_third), s.f22, F2(a.h_sixth) * s.f12));
    } else {
        auto cm = [](F2 c, F2 cl, F2 x, F2 y) { return fma(cl, x, fma(c, x, y)); };
        const F2 hhl(a.h_half_lo), z(0.f, 0.f);
        const F2 H26(a.h2_sixth), H26l(a.h2_sixth_lo), H3(a.h_third), H3l(a.h_third_lo);
        const F2 H6(a.h_sixth), H6l(a.h_sixth_lo);
        eq[0] = cm(H26, H26l, (s.f11 + s.f21) + l0, s.hq1);
        eq[1] = cm(H26, H26l, (s.f12 + s.f22) + l1, s.hq2);
        eq[2] = cm(hh, hhl, l0, cm(H3, H3l, s.f21, cm(H6, H6l, s.f11, z)));
        eq[3] = cm(hh, hhl, l1, cm(H3, H3l, s.f22, cm(H6, H6l, s.f12, z)));
    }
}

// FP64 only: F(u) with |u|^2 - R^2 as one chain of fused multiply-adds (an
// operation and a rounding less than the sum of squares minus R^2).
__device__ __forceinline__ void rhs_pair_f64(const StageCoef<double> &c, double u1, double u2, double l1, double l2,
                                             double &f1, double &f2)
{
    const double k = fma(-c.hlam, fma(u1, u1, fma(u2, u2, -c.R2)), c.kappa);
    f1 = fma(k, u1, l1);
    f2 = fma(k, u2, l2);
}

// Stage arithmetic of sweep A on V sites: from the Laplacians and centre
// values of (psi1, psi2, Pi1, Pi2) to the increments
//   o = (d3_1, d3_2, d4_1, d4_2, E_1, E_2, Q_1, Q_2),
//   d3 = h/2 Pi + h^2/4 F1            (S3 = psi + d3)
//   d4 = h Pi + h^2/2 F2              (S4 = psi + d4)
//   E  = h Pi + h^2/6 (F1 + F2 + L)   (psi_{n+1} = psi + E + h^2/6 (F3 - L))
//   Q  = h/6 F1 + h/3 F2 + h/2 L      (Pi_{n+1}  = Pi + Q + h/3 (F3 - L) + h/6 (F4 - L))
// with L = lap psi_n. Every stored quantity is an increment, of the size of
// h Pi rather than of psi: sweep B rebuilds S3, S4 and the new state by adding
// them to psi_n, Pi_n, so the state is rounded once per step at its own scale
// and the stage Laplacians lap S = L + lap d never see a stage value rounded
// at the scale of psi. The separate sweeps and the fused steps all call this
// function, so their results agree bit for bit.
//
// COMP, the compensated FP32 step: every product with a step fraction c
// (h, h/2, h^2/4, ...) is formed as (c + c_lo) x = fma(c_lo, x, fma(c, x, y)),
// c_lo the FP32 remainder of c. FP32 rounds each fraction once for the whole
// run, in the same direction at every site, a bias of ~3e-8 per step that the
// plain form integrates (with the Laplacian weights' remainders, lap_pair).
template <typename T, int V, bool COMP = false>
__device__ __forceinline__ void stage_a(const SweepArgs<T> &a, const T (&lap)[4][V], const T (&ctr)[4][V],
                                        T (&o)[8][V])
{
    if constexpr (kPackedPairs<T, V>) {
#pragma unroll
        for (int v = 0; v < V; v += 2) {
            auto pr = [&](const T (&x)[V]) { return F2(x[v], x[v + 1]); };
            const StageAPair s = stage_a_pair<COMP>(a, pr(ctr[0]), pr(ctr[1]), pr(ctr[2]), pr(ctr[3]), pr(lap[0]),
                                                    pr(lap[1]), pr(lap[2]), pr(lap[3]));
            F2 eq[4];
            stage_a_eq<COMP>(a, s, pr(lap[0]), pr(lap[1]), eq);
            const F2 r[8] = {s.d[0], s.d[1], s.d[2], s.d[3], eq[0], eq[1], eq[2], eq[3]};
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                o[c][v] = r[c].v.x;
                o[c][v + 1] = r[c].v.y;
            }
        }
    } else if constexpr (std::is_same<T, double>::value) {
        // FP64 sweeps wait for the FP64 pipe (2 operations per SM and clock): the same
        // increments in 32 operations where the expressions below take 38 (rhs_pair_f64;
        // Q without its factor h/6, which sweep B applies to all of its sum). 256^3 step
        // with sweep B's part: 3.03 -> 2.87 ms.
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const double p1 = ctr[0][v], p2 = ctr[1][v];
            const double a1 = a.h_half * ctr[2][v], a2 = a.h_half * ctr[3][v];
            const double l1 = lap[0][v], l2 = lap[1][v];
            double f11, f12, f21, f22;
            rhs_pair_f64(a.c1, p1, p2, l1, l2, f11, f12);
            rhs_pair_f64(a.c2, fma(a.h_half, ctr[2][v], p1), fma(a.h_half, ctr[3][v], p2),
                         fma(a.h_half, lap[2][v], l1), fma(a.h_half, lap[3][v], l2), f21, f22);
            const double hq1 = 2.0 * a1, hq2 = 2.0 * a2;
            const double s1 = (f11 + f21) + l1, s2 = (f12 + f22) + l2;
            o[0][v] = fma(a.h2_quarter, f11, a1);
            o[1][v] = fma(a.h2_quarter, f12, a2);
            o[2][v] = fma(a.h2_half, f21, hq1);
            o[3][v] = fma(a.h2_half, f22, hq2);
            o[4][v] = fma(a.h2_sixth, s1, hq1);
            o[5][v] = fma(a.h2_sixth, s2, hq2);
            o[6][v] = s1 + fma(2.0, l1, f21);  // 6/h Q = F1 + 2 F2 + 3 L
            o[7][v] = s2 + fma(2.0, l2, f22);
        }
    } else {
        static_assert(!COMP, "the compensated step is built for packed FP32 pairs");
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const T p1 = ctr[0][v], p2 = ctr[1][v], q1 = ctr[2][v], q2 = ctr[3][v];
            T f11, f12, f21, f22;
            rhs_pair(a.c1, p1, p2, lap[0][v], lap[1][v], f11, f12);  // F1 = F(t, psi_n)
            // F2 = F(t + h/2, chi), chi = psi_n + h/2 Pi_n, lap(chi) = lap(psi) + h/2 lap(Pi)
            const T c1 = fma(a.h_half, q1, p1), c2 = fma(a.h_half, q2, p2);
            rhs_pair(a.c2, c1, c2, fma(a.h_half, lap[2][v], lap[0][v]), fma(a.h_half, lap[3][v], lap[1][v]), f21, f22);
            const T hq1 = a.h * q1, hq2 = a.h * q2;
            o[0][v] = fma(a.h2_quarter, f11, a.h_half * q1);                      // d3
            o[1][v] = fma(a.h2_quarter, f12, a.h_half * q2);
            o[2][v] = fma(a.h2_half, f21, hq1);                                   // d4
            o[3][v] = fma(a.h2_half, f22, hq2);
            o[4][v] = fma(a.h2_sixth, (f11 + f21) + lap[0][v], hq1);              // E
            o[5][v] = fma(a.h2_sixth, (f12 + f22) + lap[1][v], hq2);
            o[6][v] = fma(a.h_half, lap[0][v], fma(a.h_third, f21, a.h_sixth * f11));  // Q
            o[7][v] = fma(a.h_half, lap[1][v], fma(a.h_third, f22, a.h_sixth * f12));
        }
    }
}

// Two sites of sweep B with packed FP32 (the arithmetic of stage_b below): d =
// (d3_1, d3_2, d4_1, d4_2) and their Laplacians, e = (E, Q), y = (psi_n, Pi_n).
template <bool COMP>
__device__ __forceinline__ void stage_b_pair(const SweepArgs<float> &a, F2 d0, F2 d1, F2 d2, F2 d3, const F2 (&lap)[4],
                                             const F2 (&e)[4], const F2 (&y)[4], F2 (&o)[4])
{
    F2 g31, g32, g41, g42;
    rhs_pair(a.c2, y[0] + d0, y[1] + d1, lap[0], lap[1], g31, g32);
    rhs_pair(a.c4, y[0] + d2, y[1] + d3, lap[2], lap[3], g41, g42);
    if constexpr (!COMP) {
        o[0] = y[0] + fma(F2(a.h2_sixth), g31, e[0]);
        o[1] = y[1] + fma(F2(a.h2_sixth), g32, e[1]);
        o[2] = y[2] + fma(F2(a.h_sixth), g41, fma(F2(a.h_third), g31, e[2]));
        o[3] = y[3] + fma(F2(a.h_sixth), g42, fma(F2(a.h_third), g32, e[3]));
    } else {
        auto cm = [](F2 c, F2 cl, F2 x, F2 y) { return fma(cl, x, fma(c, x, y)); };
        const F2 H26(a.h2_sixth), H26l(a.h2_sixth_lo), H3(a.h_third), H3l(a.h_third_lo);
        const F2 H6(a.h_sixth), H6l(a.h_sixth_lo);
        o[0] = y[0] + cm(H26, H26l, g31, e[0]);
        o[1] = y[1] + cm(H26, H26l, g32, e[1]);
        o[2] = y[2] + cm(H6, H6l, g41, cm(H3, H3l, g31, e[2]));
        o[3] = y[3] + cm(H6, H6l, g42, cm(H3, H3l, g32, e[3]));
    }
}

// Stage arithmetic of sweep B on V sites: from the Laplacians and centre
// values of (d3_1, d3_2, d4_1, d4_2) and the pointwise
// pq = (E_1, E_2, Q_1, Q_2, psi1, psi2, Pi1, Pi2) of the step's start to
// o = (psi1, psi2, Pi1, Pi2) at its end. With S = psi_n + d, the stage RHS is
// F(S) = L + G with G = lap d + (kappa - lambda/2 (|S|^2 - R^2)) S; the L
// parts are already in E and Q.
template <typename T, int V, typename PQ, bool COMP = false>
__device__ __forceinline__ void stage_b(const SweepArgs<T> &a, const T (&lap)[4][V], const T (&ctr)[4][V],
                                        const PQ &pq, T (&o)[4][V])
{
    if constexpr (kPackedPairs<T, V>) {
#pragma unroll
        for (int v = 0; v < V; v += 2) {
            auto pr = [&](const T (&x)[V]) { return F2(x[v], x[v + 1]); };
            const F2 l[4] = {pr(lap[0]), pr(lap[1]), pr(lap[2]), pr(lap[3])};
            const F2 e[4] = {pr(pq[0]), pr(pq[1]), pr(pq[2]), pr(pq[3])};
            const F2 y[4] = {pr(pq[4]), pr(pq[5]), pr(pq[6]), pr(pq[7])};
            F2 r[4];
            stage_b_pair<COMP>(a, pr(ctr[0]), pr(ctr[1]), pr(ctr[2]), pr(ctr[3]), l, e, y, r);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                o[c][v] = r[c].v.x;
                o[c][v + 1] = r[c].v.y;
            }
        }
    } else if constexpr (std::is_same<T, double>::value) {
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const double p1 = pq[4][v], p2 = pq[5][v];
            double g31, g32, g41, g42;
            rhs_pair_f64(a.c2, p1 + ctr[0][v], p2 + ctr[1][v], lap[0][v], lap[1][v], g31, g32);  // F3 - L at S3
            rhs_pair_f64(a.c4, p1 + ctr[2][v], p2 + ctr[3][v], lap[2][v], lap[3][v], g41, g42);  // F4 - L at S4
            o[0][v] = p1 + fma(a.h2_sixth, g31, pq[0][v]);
            o[1][v] = p2 + fma(a.h2_sixth, g32, pq[1][v]);
            // pq[2], pq[3]: 6/h Q (stage_a)
            o[2][v] = fma(a.h_sixth, fma(2.0, g31, pq[2][v]) + g41, pq[6][v]);
            o[3][v] = fma(a.h_sixth, fma(2.0, g32, pq[3][v]) + g42, pq[7][v]);
        }
    } else {
        static_assert(!COMP, "the compensated step is built for packed FP32 pairs");
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const T p1 = pq[4][v], p2 = pq[5][v];
            T g31, g32, g41, g42;
            rhs_pair(a.c2, p1 + ctr[0][v], p2 + ctr[1][v], lap[0][v], lap[1][v], g31, g32);  // F3 - L at S3
            rhs_pair(a.c4, p1 + ctr[2][v], p2 + ctr[3][v], lap[2][v], lap[3][v], g41, g42);  // F4 - L at S4
            o[0][v] = p1 + fma(a.h2_sixth, g31, pq[0][v]);
            o[1][v] = p2 + fma(a.h2_sixth, g32, pq[1][v]);
            o[2][v] = pq[6][v] + fma(a.h_sixth, g41, fma(a.h_third, g31, pq[2][v]));
            o[3][v] = pq[7][v] + fma(a.h_sixth, g42, fma(a.h_third, g32, pq[3][v]));
        }
    }
}

// Sweep A: stencil on (psi_n, Pi_n); writes d3, d4 (with periodic copies) and E, Q.
template <bool COMP> struct ForwardAT {
    static constexpr int kPointwise = 0;
    static constexpr bool kLambdaGrad = false;
    static constexpr bool kComp = COMP;
    template <typename T, int V, bool HINT, typename PQ>
    __device__ static void apply(const SweepArgs<T> &a, const BoxGeom &b, const T (&lap)[4][V],
                                 const T (&ctr)[4][V], const PQ &, int64_t off, int x, int y, LamAcc<T> &,
                                 uint64_t pol)
    {
        T o[8][V];
        stage_a<T, V, COMP>(a, lap, ctr, o);
#pragma unroll
        for (int c = 0; c < 4; ++c)
            store_with_copies<T, V, HINT>(a.out[c], off, x, y, b.nx, b.ny, b.js, o[c], pol, b.periodic);
#pragma unroll
        for (int c = 4; c < 8; ++c) st_out<T, V, HINT>(a.out[c] + off, o[c], pol);
    }
};

// The stage increments d3, d4 of sweep A alone, at the sites (no periodic copies):
// what the adjoint step recomputes. 4 words a site less to write than with E and Q:
// the FP32 adjoint step 121 -> 111 us at 128^3, 656 -> 613 at 256^3.
template <bool COMP> struct ForwardStagesT {
    static constexpr int kPointwise = 0;
    static constexpr bool kLambdaGrad = false;
    static constexpr bool kComp = COMP;
    template <typename T, int V, bool HINT, typename PQ>
    __device__ static void apply(const SweepArgs<T> &a, const BoxGeom &, const T (&lap)[4][V], const T (&ctr)[4][V],
                                 const PQ &, int64_t off, int, int, LamAcc<T> &, uint64_t pol)
    {
        T o[8][V];
        stage_a<T, V, COMP>(a, lap, ctr, o);
#pragma unroll
        for (int c = 0; c < 4; ++c) st_out<T, V, HINT>(a.out[c] + off, o[c], pol);
    }
};

// Sweep B: stencil on (d3, d4), pointwise (E, Q) and (psi_n, Pi_n); writes
// psi_{n+1}, Pi_{n+1} (over psi_n, Pi_n: each site reads its own inputs first).
template <bool COMP> struct ForwardBT {
    static constexpr int kPointwise = 8;
    static constexpr bool kLambdaGrad = false;
    static constexpr bool kComp = COMP;
    template <typename T, int V, bool HINT, typename PQ>
    __device__ static void apply(const SweepArgs<T> &a, const BoxGeom &b, const T (&lap)[4][V],
                                 const T (&ctr)[4][V], const PQ &pq, int64_t off, int x, int y, LamAcc<T> &,
                                 uint64_t pol)
    {
        T o[4][V];
        stage_b<T, V, PQ, COMP>(a, lap, ctr, pq, o);
#pragma unroll
        for (int c = 0; c < 4; ++c)
            store_with_copies<T, V, HINT>(a.out[c], off, x, y, b.nx, b.ny, b.js, o[c], pol, b.periodic);
    }
};
using ForwardA = ForwardAT<false>;
using ForwardB = ForwardBT<false>;

// Host: step constants shared by every box (Laplacian weights for dx, RK4 step
// fractions) and the bounded-wait limit of this launch.
template <typename T> inline void fill_step_constants(SweepArgs<T> &a, double dx, double dt)
{
    const double inv_dx2 = 1.0 / (dx * dx);
    a.wA = T((4.0 / 3.0) * inv_dx2);
    a.wB = T((-1.0 / 12.0) * inv_dx2);
    a.wC = T(-7.5 * inv_dx2);
    // lap_site scales wT by powers of two within 2^+-554
    a.wT = T(inv_dx2 > 0x1p-400 && inv_dx2 < 0x1p400 ? inv_dx2 / 12.0 : 0.0);
    if constexpr (std::is_same<T, double>::value) {
        // 1 - 12 dx^2 wT from exact products (at most 2^-51, so the remainder fits)
        const double x = 12.0 * a.wT, xl = std::fma(12.0, a.wT, -x), p = dx * dx, pl = std::fma(dx, dx, -p);
        if (a.wT != 0.0) a.wT_lo = (int)std::nearbyint((std::fma(-x, p, 1.0) - xl * p - x * pl) * 0x1p64);
    }
    a.h = T(dt);
    a.h_half = T(0.5 * dt);
    a.h2_quarter = T(0.25 * dt * dt);
    a.h2_half = T(0.5 * dt * dt);
    a.h_sixth = T(dt / 6.0);
    a.h_third = T(dt / 3.0);
    a.h2_sixth = T(dt * dt / 6.0);
    a.wA_lo = T((4.0 / 3.0) * inv_dx2 - (double)a.wA);
    a.wB_lo = T((-1.0 / 12.0) * inv_dx2 - (double)a.wB);
    a.h_lo = T(dt - (double)a.h);
    a.h_half_lo = T(0.5 * dt - (double)a.h_half);
    a.h2_quarter_lo = T(0.25 * dt * dt - (double)a.h2_quarter);
    a.h2_half_lo = T(0.5 * dt * dt - (double)a.h2_half);
    a.h_sixth_lo = T(dt / 6.0 - (double)a.h_sixth);
    a.h_third_lo = T(dt / 3.0 - (double)a.h_third);
    a.h2_sixth_lo = T(dt * dt / 6.0 - (double)a.h2_sixth);
    a.wait_polls = device_wait_polls();
}

// Host: kappa, lambda/2 and R^2 at one stage time (the reference's
// specific_eval_rhs coefficients, AxionStringsLevel.cpp:850-921).
template <typename T> inline StageCoef<T> stage_coef(const axs_background &bg, double tau)
{
    axs_rhs_coeffs c;
    rhs_coeffs(bg, tau, c);
    return StageCoef<T>{T(c.kappa), T(0.5 * c.lambda), T(c.R2)};
}

}  // namespace axs
