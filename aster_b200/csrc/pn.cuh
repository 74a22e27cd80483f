// Pairwise post-Newtonian terms of the reference's compute_gravitational
// (src/physics/tool_chain_impl.cpp:120-137): get_pn1 (c^-2, :110-118), get_pn2
// (c^-4, :79-107) and get_pn25 (c^-5, :65-77), selected by the force-law bits.
// Shared by the all-pairs kernels and the batched ensemble kernel.
#pragma once

#include "aster_internal.cuh"

// Post-Newtonian constants and the terms in use: f bit 0 = 1PN, bit 1 = 2PN,
// bit 2 = 2.5PN. PN level PNL (a template parameter of the kernels): 0 Newton
// only, 1 Newton + 1PN, 2 Newton + the terms f selects. c2 = c^-2, c4 = c^-4,
// ic = c^-1 (c^-5 is formed as c^-4 ic inside a product that stays in FP32
// range: c^-5 itself is below FP32's normal range in SI units).
template <class T>
struct PnK {
    T c2, c4, ic;
    int f;
};

// Acceleration on body i from body j, divided by G, FP64: the Newtonian term and
// the terms of level PNL added to a. j == i contributes 0 (inv = 0: zero
// separation). d = x_j - x_i, inv = 1/r; n = -d/r the unit vector from j to i (the
// reference's -norm), p_i = G m_i / r, p_j = G m_j / r:
//   Newton : m_j/r^2 [-n]
//   1PN : c^-2 m_j/r^2 [n A + (v_i - v_j) B]
//   2PN : c^-4 m_j/r^2 [n S_n + (v_i - v_j) S_v + n (-57/4 p_i^2 - 9 p_j^2 - 69/2 p_i p_j)]
//   2.5PN: c^-5 4/5 p_i m_j/r^2 [(v_i - v_j) I_1 + n (n.(v_i - v_j)) I_2]
// with A, B, S_n, S_v, I_1, I_2 the scalar brackets of get_pn1, get_pn2 and
// get_pn25. The 2PN mass term is the reference's G^2 m_j/r^4 (-57/4 m_i^2 -
// 9 m_j^2 - 69/2 m_i m_j) written with p_i, p_j, which keeps every factor in
// FP32 range for masses of ~1e30 (m^2 would overflow; the FP32 forms below share
// it). The brackets of all the terms are gathered into one factor of n and one of
// v_i - v_j, so that the components cost nine operations in all instead of
// nine a term, and the products of each bracket by Horner's rule: FP64 issue
// bounds every kernel that uses this (every term, all-pairs of 30,000 bodies 8.59
// -> 6.17 ms, tree walk of 300,000 8.20 -> 6.02, 20 steps of 16,384 ensemble systems
// 15.7 -> 11.1; 1PN walk of 20,011 0.52 -> 0.38, ensemble 6.22 -> 5.81).
template <int PNL>
__device__ __forceinline__ void newton_pn_f64(const PnK<double>& k, double dx, double dy, double dz, double inv,
                                              double mi, double mj, const double4 vi, const double4 vj, double G,
                                              double& ax, double& ay, double& az) {
    const double nx = -dx * inv, ny = -dy * inv, nz = -dz * inv;
    const double dvx = vi.x - vj.x, dvy = vi.y - vj.y, dvz = vi.z - vj.z;
    const double vi2 = vi.w, vj2 = vj.w;  // |v|^2
    const double v12 = vi.x * vj.x + vi.y * vj.y + vi.z * vj.z;
    const double nv1 = nx * vi.x + ny * vi.y + nz * vi.z;
    const double nv2 = nx * vj.x + ny * vj.y + nz * vj.z;
    const double nv22 = nv2 * nv2, p1 = G * mi * inv, p2 = G * mj * inv;
    double cn = -1.0, cv = 0.0;  // the factors of n and of v_i - v_j
    if (PNL == 1 || (PNL == 2 && (k.f & 1))) {
        const double A = fma(5.0, p1, fma(4.0, p2, fma(1.5, nv22, fma(4.0, v12, fma(-2.0, vj2, -vi2)))));
        cn = fma(k.c2, A, cn);
        cv = k.c2 * fma(4.0, nv1, -3.0 * nv2);
    }
    if (PNL == 2 && (k.f & 2)) {
        const double e = vj2 - v12;
        const double a1 = fma(1.5, vi2, fma(4.5, vj2, fma(-6.0, v12, -1.875 * nv22)));
        const double a2 = fma(-3.75, vi2, fma(1.25, vj2, fma(-2.5, v12, fma(8.5, nv22, nv1 * fma(19.5, nv1, -39.0 * nv2)))));
        const double a3 = fma(4.0, vj2, fma(-8.0, v12, fma(-6.0, nv22, nv1 * fma(2.0, nv1, -4.0 * nv2))));
        const double Sm = fma(p1, fma(-14.25, p1, -34.5 * p2), -9.0 * p2 * p2);
        const double Sn = fma(-2.0 * e, e, fma(nv22, a1, fma(p1, a2, fma(p2, a3, Sm))));
        const double b1 = fma(4.0, e, fma(-6.0, nv22, fma(-15.75, p1, -2.0 * p2)));
        const double b2 = fma(-5.0, vj2, fma(4.0, v12, fma(4.5, nv22, fma(13.75, p1, fma(-2.0, p2, vi2)))));
        cn = fma(k.c4, Sn, cn);
        cv = fma(k.c4, fma(nv1, b1, nv2 * b2), cv);
    }
    if (PNL == 2 && (k.f & 4)) {
        const double sq = fma(dvx, dvx, fma(dvy, dvy, dvz * dvz));
        const double I1 = fma(2.0, p1, fma(-8.0, p2, -sq));
        const double I2 = (nv1 - nv2) * fma(3.0, sq, fma(-6.0, p1, (52.0 / 3.0) * p2));
        const double g = 0.8 * p1 * k.c4 * k.ic;
        cn = fma(g, I2, cn);
        cv = fma(g, I1, cv);
    }
    const double f = mj * (inv * inv);
    cn *= f;
    cv *= f;
    ax = fma(nx, cn, fma(dvx, cv, ax));
    ay = fma(ny, cn, fma(dvy, cv, ay));
    az = fma(nz, cn, fma(dvz, cv, az));
}

// Newton + 1PN for two sources at once with the paired FP32 instructions of
// sm_100 (add/mul/fma .f32x2), one source in each half of every operand.
// d = x_j - x_i (both sources), mj their masses, vj their velocities and
// vj2 = |v_j|^2; per target, broadcast to both halves: vi its velocity,
// vi4 = 4 v_i, nvi2 = -|v_i|^2 and mi5G = 5 G m_i; G4 = 4 G. Adds the
// Newtonian m_j d / r^3 to a (divided by G) and to p the 1PN sum
//   P = sum_j m_j r^-3 [d A + (v_i - v_j) B'],
//   A = -|v_i|^2 - 2 |v_j|^2 + 4 v_i.v_j + 3/2 (d.v_j / r)^2 + (5 m_i + 4 m_j) G / r,
//   B' = 4 d.v_i - 3 d.v_j,
// whose -c^-2 multiple is the 1PN acceleration divided by G: newton_pn_f64's with
// n = -d / r, B = -B' / r and f = c^-2 m_j / r^2 gathered into m_j r^-3, so
// that the unit vector and f cost no instructions of their own. GUARD: a zero
// r^2 (the target itself when unsoftened) contributes nothing.
template <bool GUARD>
__device__ __forceinline__ void newton_pn1_x2(const float2 dx, const float2 dy, const float2 dz, const float2 mj,
                                              const float2 vjx, const float2 vjy, const float2 vjz, const float2 vj2,
                                              const float2 vix, const float2 viy, const float2 viz,
                                              const float2 vi4x, const float2 vi4y, const float2 vi4z,
                                              const float2 nvi2, const float2 mi5G, const float2 eps2,
                                              const float2 G4, float2& ax, float2& ay, float2& az, float2& px,
                                              float2& py, float2& pz) {
    float2 r2 = __ffma2_rn(dz, dz, eps2);
    r2 = __ffma2_rn(dy, dy, r2);
    r2 = __ffma2_rn(dx, dx, r2);
    float2 s = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
    if (GUARD) {
        s.x = r2.x > 0.f ? s.x : 0.f;
        s.y = r2.y > 0.f ? s.y : 0.f;
    }
    const float2 ms = __fmul2_rn(mj, s);
    const float2 sN = __fmul2_rn(ms, __fmul2_rn(s, s));  // m_j / r^3
    ax = __ffma2_rn(dx, sN, ax);
    ay = __ffma2_rn(dy, sN, ay);
    az = __ffma2_rn(dz, sN, az);
    const float2 w = __ffma2_rn(dx, vjx, __ffma2_rn(dy, vjy, __fmul2_rn(dz, vjz)));     // d.v_j
    const float2 u4 = __ffma2_rn(dx, vi4x, __ffma2_rn(dy, vi4y, __fmul2_rn(dz, vi4z)));  // 4 d.v_i
    const float2 Bp = __ffma2_rn(w, make_float2(-3.f, -3.f), u4);
    const float2 ws = __fmul2_rn(w, s);
    float2 A = __ffma2_rn(vj2, make_float2(-2.f, -2.f), nvi2);
    A = __ffma2_rn(vi4x, vjx, A);
    A = __ffma2_rn(vi4y, vjy, A);
    A = __ffma2_rn(vi4z, vjz, A);
    A = __ffma2_rn(__fmul2_rn(ws, ws), make_float2(1.5f, 1.5f), A);
    A = __ffma2_rn(ms, G4, A);
    A = __ffma2_rn(s, mi5G, A);
    const float2 sA = __fmul2_rn(sN, A), sB = __fmul2_rn(sN, Bp);
    const float2 m1 = make_float2(-1.f, -1.f);
    const float2 dvx = __ffma2_rn(vjx, m1, vix), dvy = __ffma2_rn(vjy, m1, viy), dvz = __ffma2_rn(vjz, m1, viz);
    px = __ffma2_rn(dx, sA, __ffma2_rn(dvx, sB, px));
    py = __ffma2_rn(dy, sA, __ffma2_rn(dvy, sB, py));
    pz = __ffma2_rn(dz, sA, __ffma2_rn(dvz, sB, pz));
}

// Newton and every post-Newtonian term the flags select (bit 0 1PN, bit 1 2PN,
// bit 2 2.5PN), two sources per paired FP32 instruction: the algebra of
// newton_pn_f64 with the sums gathered under the Newtonian factor
// m_j / r^3 and the c^-2, c^-4 factors applied once per target, as in
// newton_pn1_x2. Inputs as newton_pn1_x2's, plus vi2 = |v_i|^2 and
// Gmi = G m_i per target and nk = -0.8 c^-1. Adds m_j d / r^3 to a, to p the
// 1PN sum P of newton_pn1_x2 (the 1PN term is -c^-2 P) and to q the sum Q whose
// -c^-4 multiple is the 2PN + 2.5PN term (all divided by G). With
// n = -d s, nv1 = n.v_i = -s d.v_i, nv2 = -s d.v_j, p1 = G m_i s, p2 = G m_j s:
//   2PN:   c^-4 m_j s^2 [n (Sn + Sm) + dv Sv] = -c^-4 [m_j s^3 (Sn + Sm) d - m_j s^2 Sv dv],
//   2.5PN: 0.8 c^-5 p1 m_j s^2 [dv I1 + n I2] = -c^-4 (-0.8 c^-1) p1 m_j s^2 [dv I1 - s I2 d].
template <bool GUARD>
__device__ __forceinline__ void newton_pn_all_x2(const float2 dx, const float2 dy, const float2 dz, const float2 mj,
                                                 const float2 vjx, const float2 vjy, const float2 vjz,
                                                 const float2 vj2, const float2 vix, const float2 viy,
                                                 const float2 viz, const float2 vi4x, const float2 vi4y,
                                                 const float2 vi4z, const float2 nvi2, const float2 vi2,
                                                 const float2 mi5G, const float2 Gmi, const float2 eps2,
                                                 const float2 G4, const float2 G2, const float2 nk, int f,
                                                 float2& ax, float2& ay, float2& az, float2& px, float2& py,
                                                 float2& pz, float2& qx, float2& qy, float2& qz) {
    auto k2 = [](float v) { return make_float2(v, v); };
    float2 r2 = __ffma2_rn(dz, dz, eps2);
    r2 = __ffma2_rn(dy, dy, r2);
    r2 = __ffma2_rn(dx, dx, r2);
    float2 s = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
    if (GUARD) {
        s.x = r2.x > 0.f ? s.x : 0.f;
        s.y = r2.y > 0.f ? s.y : 0.f;
    }
    const float2 ms = __fmul2_rn(mj, s);
    const float2 mss = __fmul2_rn(ms, s);   // m_j / r^2
    const float2 sN = __fmul2_rn(mss, s);   // m_j / r^3
    ax = __ffma2_rn(dx, sN, ax);
    ay = __ffma2_rn(dy, sN, ay);
    az = __ffma2_rn(dz, sN, az);
    if (!(f & 7)) return;
    const float2 m1 = k2(-1.f);
    const float2 w = __ffma2_rn(dx, vjx, __ffma2_rn(dy, vjy, __fmul2_rn(dz, vjz)));     // d.v_j
    const float2 u4 = __ffma2_rn(dx, vi4x, __ffma2_rn(dy, vi4y, __fmul2_rn(dz, vi4z)));  // 4 d.v_i
    const float2 dvx = __ffma2_rn(vjx, m1, vix), dvy = __ffma2_rn(vjy, m1, viy), dvz = __ffma2_rn(vjz, m1, viz);
    if (f & 1) {  // 1PN: newton_pn1_x2's sum
        const float2 Bp = __ffma2_rn(w, k2(-3.f), u4);
        const float2 ws = __fmul2_rn(w, s);
        float2 A = __ffma2_rn(vj2, k2(-2.f), nvi2);
        A = __ffma2_rn(vi4x, vjx, A);
        A = __ffma2_rn(vi4y, vjy, A);
        A = __ffma2_rn(vi4z, vjz, A);
        A = __ffma2_rn(__fmul2_rn(ws, ws), k2(1.5f), A);
        A = __ffma2_rn(ms, G4, A);
        A = __ffma2_rn(s, mi5G, A);
        const float2 sA = __fmul2_rn(sN, A), sB = __fmul2_rn(sN, Bp);
        px = __ffma2_rn(dx, sA, __ffma2_rn(dvx, sB, px));
        py = __ffma2_rn(dy, sA, __ffma2_rn(dvy, sB, py));
        pz = __ffma2_rn(dz, sA, __ffma2_rn(dvz, sB, pz));
    }
    if (!(f & 6)) return;
    const float2 nv1 = __fmul2_rn(u4, __fmul2_rn(s, k2(-0.25f)));  // n.v_i
    const float2 nv2 = __fmul2_rn(__fmul2_rn(w, s), m1);           // n.v_j
    const float2 v12 = __ffma2_rn(vix, vjx, __ffma2_rn(viy, vjy, __fmul2_rn(viz, vjz)));
    const float2 p1 = __fmul2_rn(Gmi, s), p2 = __fmul2_rn(G2, ms);  // G m_i / r, G m_j / r
    if (f & 2) {  // 2PN (as newton_pn_f64)
        const float2 nv22 = __fmul2_rn(nv2, nv2), nv12 = __fmul2_rn(nv1, nv1), n12 = __fmul2_rn(nv1, nv2);
        // -2 vj2^2 + 4 vj2 v12 - 2 v12^2 = -2 (vj2 - v12)^2
        const float2 t = __ffma2_rn(v12, m1, vj2);
        float2 Sn = __fmul2_rn(__fmul2_rn(t, t), k2(-2.f));
        // + nv22 (1.5 vi2 + 4.5 vj2 - 6 v12) - 1.875 nv22^2
        const float2 c1 = __ffma2_rn(v12, k2(-6.f), __ffma2_rn(vj2, k2(4.5f), __fmul2_rn(vi2, k2(1.5f))));
        Sn = __ffma2_rn(nv22, c1, Sn);
        Sn = __ffma2_rn(__fmul2_rn(nv22, nv22), k2(-1.875f), Sn);
        // + p1 (-3.75 vi2 + 1.25 vj2 - 2.5 v12 + 19.5 nv12 - 39 nv1 nv2 + 8.5 nv22)
        float2 e1 = __ffma2_rn(vj2, k2(1.25f), __fmul2_rn(vi2, k2(-3.75f)));
        e1 = __ffma2_rn(v12, k2(-2.5f), e1);
        e1 = __ffma2_rn(nv12, k2(19.5f), e1);
        e1 = __ffma2_rn(n12, k2(-39.f), e1);
        e1 = __ffma2_rn(nv22, k2(8.5f), e1);
        Sn = __ffma2_rn(p1, e1, Sn);
        // + p2 (4 vj2 - 8 v12 + 2 nv12 - 4 nv1 nv2 - 6 nv22)
        float2 e2 = __ffma2_rn(v12, k2(-8.f), __fmul2_rn(vj2, k2(4.f)));
        e2 = __ffma2_rn(nv12, k2(2.f), e2);
        e2 = __ffma2_rn(n12, k2(-4.f), e2);
        e2 = __ffma2_rn(nv22, k2(-6.f), e2);
        Sn = __ffma2_rn(p2, e2, Sn);
        // Sv = nv1 (4 vj2 - 4 v12 - 6 nv22 - 15.75 p1 - 2 p2) + nv2 (vi2 - 5 vj2 + 4 v12 + 4.5 nv22 + 13.75 p1 - 2 p2)
        float2 A1 = __ffma2_rn(v12, k2(-4.f), __fmul2_rn(vj2, k2(4.f)));
        A1 = __ffma2_rn(nv22, k2(-6.f), A1);
        A1 = __ffma2_rn(p1, k2(-15.75f), A1);
        A1 = __ffma2_rn(p2, k2(-2.f), A1);
        float2 A2 = __ffma2_rn(vj2, k2(-5.f), vi2);
        A2 = __ffma2_rn(v12, k2(4.f), A2);
        A2 = __ffma2_rn(nv22, k2(4.5f), A2);
        A2 = __ffma2_rn(p1, k2(13.75f), A2);
        A2 = __ffma2_rn(p2, k2(-2.f), A2);
        const float2 Sv = __ffma2_rn(nv1, A1, __fmul2_rn(nv2, A2));
        // Sm = -14.25 p1^2 - 9 p2^2 - 34.5 p1 p2
        const float2 Sm = __ffma2_rn(p1, __ffma2_rn(p1, k2(-14.25f), __fmul2_rn(p2, k2(-34.5f))),
                                     __fmul2_rn(__fmul2_rn(p2, p2), k2(-9.f)));
        // Q += m_j s^3 (Sn + Sm) d - m_j s^2 Sv dv
        const float2 a1 = __fmul2_rn(sN, __fadd2_rn(Sn, Sm)), a2 = __fmul2_rn(__fmul2_rn(mss, Sv), m1);
        qx = __ffma2_rn(dx, a1, __ffma2_rn(dvx, a2, qx));
        qy = __ffma2_rn(dy, a1, __ffma2_rn(dvy, a2, qy));
        qz = __ffma2_rn(dz, a1, __ffma2_rn(dvz, a2, qz));
    }
    if (f & 4) {  // 2.5PN (as newton_pn_f64)
        const float2 sq = __ffma2_rn(dvx, dvx, __ffma2_rn(dvy, dvy, __fmul2_rn(dvz, dvz)));
        const float2 I1 = __ffma2_rn(p2, k2(-8.f), __ffma2_rn(p1, k2(2.f), __fmul2_rn(sq, m1)));
        const float2 I2 = __fmul2_rn(__fadd2_rn(nv1, __fmul2_rn(nv2, m1)),
                                     __ffma2_rn(p2, k2(52.f / 3.f), __ffma2_rn(sq, k2(3.f), __fmul2_rn(p1, k2(-6.f)))));
        // Q += (-0.8 c^-1) p1 m_j s^2 (dv I1 - s I2 d)
        const float2 g = __fmul2_rn(__fmul2_rn(p1, mss), nk);
        const float2 gI1 = __fmul2_rn(g, I1), gsI2 = __fmul2_rn(__fmul2_rn(g, s), __fmul2_rn(I2, m1));
        qx = __ffma2_rn(dvx, gI1, __ffma2_rn(dx, gsI2, qx));
        qy = __ffma2_rn(dvy, gI1, __ffma2_rn(dy, gsI2, qy));
        qz = __ffma2_rn(dvz, gI1, __ffma2_rn(dz, gsI2, qz));
    }
}

// The force-law bits of p as PN constants (powers of 1/c formed in the
// reference's order, inv_c * inv_c * ...).
inline PnK<double> make_pn(const aster_params* p) {
    PnK<double> k{0.0, 0.0, 0.0, 0};
    k.f = ((p->force_law & ASTER_PN1) ? 1 : 0) | ((p->force_law & ASTER_PN2) ? 2 : 0) |
          ((p->force_law & ASTER_PN25) ? 4 : 0);
    if (k.f) {
        const double ic = 1.0 / p->c;
        k.c2 = ic * ic;
        k.c4 = ic * ic * ic * ic;
        k.ic = ic;
    }
    return k;
}

// PN level of a force law: 0, 1 (1PN only) or 2 (2PN or 2.5PN present).
inline int pn_level(const aster_params* p) {
    if (p->force_law & (ASTER_PN2 | ASTER_PN25)) return 2;
    return (p->force_law & ASTER_PN1) ? 1 : 0;
}

__host__ __device__ inline PnK<float> pn_float(const PnK<double>& k) { return PnK<float>{(float)k.c2, (float)k.c4, (float)k.ic, k.f}; }
