// rpy_sym6.cuh -- pair blocks with torques and spins, both directions at once:
// the grand mobility of unit spheres above the wall, or of equal spheres without
// one, is symmetric, so the block M (j <- i) is the transpose of M (i <- j), and
// the scalar functions of the pair are evaluated once.  Same mathematics as
// wall_pair_f32 / free_pair_f32 <6, 6> (rpy_pairs.cuh).
//
// With d = x_i - x_j, d' = (dx, dy, hz), hz = z_i + z_j, and the symmetric
// coefficients of wall_pair_sym for velocities from forces:
//   spin of i from the force F on j
//     (tau_j F1 + Y dy, -tau_j F0 - Y dx, kappa (F0 dy - F1 dx)),  Y = (p_j - kappa) F2 - (d'.F) s_j
//   velocity of i from the torque T on j, the transpose of j's spin from a force on i, with X = dx T1 - dy T0
//     (-tau_i T1 - kappa dy T2 + s_i X dx, tau_i T0 + kappa dx T2 + s_i X dy, q_i X)
//   spin of i from the torque T on j
//     m0 T + r1 (d.T) d + m1 ((d'.T) (-dx, -dy, hz) + 2 X (-dy, dx, 0))
// where, with C = 1/(8 pi |d|^3), c = w^3 / 6 pi, w = 1/|d'|, u = w^2, E = hz^2 u and z the height of the index's sphere,
//   kappa = C - 3/4 c,  tau = +-C dz - 3/4 c hz + 3/2 c (z - hz u)   (+ for i <- j with z_j, - for j <- i with z_i),
//   s = c u (9/2 z - 15/2 hz u),  p = c (9 z hz u + (3/2 - 15 E) u),  q = p - kappa - hz s,
//   m0 = c (3/8 - 9/4 E) - C/2,  m1 = 9/8 c u,  r1 = 3/2 C / |d|^2.
// j <- i follows by changing the signs of dx, dy and dz.
#pragma once

#include "rpy_pairs.cuh"

namespace cufil {

// Forces and torques f[0..5]; velocities and spins v[0..5].  TJ, TI: j's and i's torques and spins take part (a blob has
// neither).
template <bool SI, bool SJ>
__device__ __forceinline__ void wall_pair_sym6_f32(float dx, float dy, float dz, float zi, float zj, const float *fj,
                                                   const float *fi, float *vi, float *vj) {
    const float c6 = RpyConst::inv6pi;
    const float c8 = RpyConst::inv8pi;
    const float q2 = fmaf(dx, dx, dy * dy);
    const float s = rsqrtf(fmaf(dz, dz, q2));
    const float s2 = s * s;
    const float g = c8 * s;
    const float A = g * fmaf(2.0f / 3.0f, s2, 1.0f);
    const float C = g * s2;
    const float B = C * fmaf(-2.0f, s2, 1.0f);
    const float hz = zi + zj;
    const float w = rsqrtf(fmaf(hz, hz, q2));
    const float u = w * w;
    const float cw = c6 * w, cu = cw * u;
    const float hu = hz * u, E = hz * hu;
    const float P = (zi * zj) * u;
    const float n5 = fmaf(7.5f, E, -1.5f);
    const float u5 = 5.0f * u;
    const float G = fmaf(0.5f * u5, fmaf(-7.0f, E, 1.0f), n5);
    const float k0 = fmaf(u, fmaf(u * (1.0f / 3.0f), n5, fmaf(-1.5f, E, 0.5f)), fmaf(1.5f, P, 0.75f));
    const float AK = fmaf(-cw, k0, A);
    const float a = -cu * fmaf(u, G, fmaf(-4.5f, P, 0.75f));
    const float z15 = 1.5f * zj;
    const float b = cu * fmaf(-9.0f * P, hz, fmaf(hu, fmaf(2.0f, G, u5), z15));
    const float c = cu * fmaf(-u5, hu, z15);
    const float e = -cu * fmaf(2.0f * z15, zj, fmaf(u, fmaf(-15.0f, E, 2.0f), 3.0f * E));
    const float AKe = AK + e;
    float kap = 0, tauj = 0, taui = 0, sj = 0, si = 0, pj = 0, pi = 0, qj = 0, qi = 0, m0 = 0, m1 = 0, r1 = 0;
    if constexpr (SI || SJ) {
        const float c75 = 0.75f * cu, c15 = 1.5f * cu, cuu = cu * u;
        kap = C - c75;
        const float t0 = -c75 * hz, hu9 = 9.0f * hu, hu75 = 7.5f * hu, e15 = u * fmaf(-15.0f, E, 1.5f);
        if constexpr (SI) {  // i's spin, and j's velocity from i's torque: functions of z_j
            tauj = fmaf(c15, zj - hu, fmaf(C, dz, t0));
            sj = cuu * fmaf(4.5f, zj, -hu75);
            pj = fmaf(cu, fmaf(hu9, zj, e15), -kap);
            qj = fmaf(-hz, sj, pj);
        }
        if constexpr (SJ) {
            taui = fmaf(c15, zi - hu, fmaf(-C, dz, t0));
            si = cuu * fmaf(4.5f, zi, -hu75);
            pi = fmaf(cu, fmaf(hu9, zi, e15), -kap);
            qi = fmaf(-hz, si, pi);
        }
        if constexpr (SI && SJ) {
            m0 = fmaf(cu, fmaf(-2.25f, E, 0.375f), -0.5f * C);
            m1 = 1.125f * cuu;
            r1 = 1.5f * C * s2;
        }
    }
    {  // i <- j
        const float p = fmaf(dx, fj[0], dy * fj[1]);
        const float dp = fmaf(hz, fj[2], p);
        const float t0 = B * fmaf(dz, fj[2], p);
        const float t1 = fmaf(a, dp, b * fj[2]);
        const float t = t0 + t1;
        vi[0] = fmaf(t, dx, fmaf(AK, fj[0], vi[0]));
        vi[1] = fmaf(t, dy, fmaf(AK, fj[1], vi[1]));
        vi[2] = fmaf(c, dp, fmaf(t1, hz, fmaf(t0, dz, fmaf(AKe, fj[2], vi[2]))));
        if constexpr (SI) {
            const float Y = fmaf(pj, fj[2], -sj * dp);
            vi[3] = fmaf(Y, dy, fmaf(tauj, fj[1], vi[3]));
            vi[4] = fmaf(-Y, dx, fmaf(-tauj, fj[0], vi[4]));
            vi[5] = fmaf(kap, fmaf(fj[0], dy, -fj[1] * dx), vi[5]);
        }
        if constexpr (SJ) {
            const float X = fmaf(dx, fj[4], -dy * fj[3]), sX = si * X, kt = kap * fj[5];
            vi[0] = fmaf(sX, dx, fmaf(-kt, dy, fmaf(-taui, fj[4], vi[0])));
            vi[1] = fmaf(sX, dy, fmaf(kt, dx, fmaf(taui, fj[3], vi[1])));
            vi[2] = fmaf(qi, X, vi[2]);
            if constexpr (SI) {
                const float pt = fmaf(dx, fj[3], dy * fj[4]);
                const float a1 = r1 * fmaf(dz, fj[5], pt), a2 = m1 * fmaf(hz, fj[5], pt), a3 = (m1 + m1) * X;
                const float a12 = a1 - a2;
                vi[3] = fmaf(-a3, dy, fmaf(a12, dx, fmaf(m0, fj[3], vi[3])));
                vi[4] = fmaf(a3, dx, fmaf(a12, dy, fmaf(m0, fj[4], vi[4])));
                vi[5] = fmaf(a2, hz, fmaf(a1, dz, fmaf(m0, fj[5], vi[5])));
            }
        }
    }
    {  // j <- i: the transposed translation block, and dx, dy, dz with their signs changed
        const float p = fmaf(dx, fi[0], dy * fi[1]);
        const float dp = fmaf(hz, fi[2], p);
        const float t0 = B * fmaf(dz, fi[2], p);
        const float t1 = fmaf(a, dp, c * fi[2]);
        const float t = t0 + t1;
        vj[0] = fmaf(t, dx, fmaf(AK, fi[0], vj[0]));
        vj[1] = fmaf(t, dy, fmaf(AK, fi[1], vj[1]));
        vj[2] = fmaf(b, dp, fmaf(t1, hz, fmaf(t0, dz, fmaf(AKe, fi[2], vj[2]))));
        if constexpr (SJ) {
            const float Y = fmaf(pi, fi[2], -si * fmaf(hz, fi[2], -p));
            vj[3] = fmaf(-Y, dy, fmaf(taui, fi[1], vj[3]));
            vj[4] = fmaf(Y, dx, fmaf(-taui, fi[0], vj[4]));
            vj[5] = fmaf(-kap, fmaf(fi[0], dy, -fi[1] * dx), vj[5]);
        }
        if constexpr (SI) {
            const float X = fmaf(dx, fi[4], -dy * fi[3]), sX = sj * X, kt = kap * fi[5];
            vj[0] = fmaf(sX, dx, fmaf(kt, dy, fmaf(-tauj, fi[4], vj[0])));
            vj[1] = fmaf(sX, dy, fmaf(-kt, dx, fmaf(tauj, fi[3], vj[1])));
            vj[2] = fmaf(-qj, X, vj[2]);
            if constexpr (SJ) {
                const float pt = fmaf(dx, fi[3], dy * fi[4]);
                const float a1 = r1 * fmaf(dz, fi[5], pt), a2 = m1 * fmaf(hz, fi[5], -pt), a3 = (m1 + m1) * X;
                const float a12 = a1 + a2;
                vj[3] = fmaf(-a3, dy, fmaf(a12, dx, fmaf(m0, fi[3], vj[3])));
                vj[4] = fmaf(a3, dx, fmaf(a12, dy, fmaf(m0, fi[4], vj[4])));
                vj[5] = fmaf(a2, hz, fmaf(a1, dz, fmaf(m0, fi[5], vj[5])));
            }
        }
    }
}

// Equal spheres of radius a without a wall:
//   v_i = A F + B (d.F) d + C T x d,   w_i = C F x d + P T + Q (d.T) d,
// far (r > 2a): A, B as free_pair_sym, C = c8 / r^3, P = -C / 2, Q = 3 C / (2 r^2); touching spheres (Zuk et al.) in
// the rare branch.  j <- i: d changes sign.
struct FreeSym6 {
    FreeSym t;
    float c8, c6;                  // 1 / (8 pi mu), 1 / (6 pi mu a)
    float c0, c1, p0, p1, p3, q0;  // touching: C = c0 - c1 r, P = p0 - p1 r + p3 r^3, Q = q0 (6 a^2 / r - r)
    float a2;
};
inline FreeSym6 free_sym6(double a, double mu) {
    const double pm = 3.14159265358979323846 * mu, a3 = a * a * a, a4 = a3 * a, a6 = a3 * a3;
    FreeSym6 q;
    q.t = free_sym(a);
    q.c8 = static_cast<float>(1.0 / (8.0 * pm));
    q.c6 = static_cast<float>(1.0 / (6.0 * pm * a));
    q.c0 = static_cast<float>(1.0 / (16.0 * pm * a3));
    q.c1 = static_cast<float>(3.0 / (128.0 * pm * a4));
    q.p0 = static_cast<float>(1.0 / (8.0 * pm * a3));
    q.p1 = static_cast<float>(54.0 / (512.0 * pm * a4));
    q.p3 = static_cast<float>(5.0 / (512.0 * pm * a6));
    q.q0 = static_cast<float>(3.0 / (512.0 * pm * a6));
    q.a2 = static_cast<float>(a * a);
    return q;
}
template <bool SI, bool SJ>
__device__ __forceinline__ void free_pair_sym6_f32(float dx, float dy, float dz, const FreeSym6 &k, const float *fj,
                                                   const float *fi, float *vi, float *vj) {
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    const float s = rsqrtf(r2);
    const float s2 = s * s;
    const float g = k.c8 * s;
    float A = g * fmaf(k.t.k, s2, 1.0f);
    float C = g * s2;
    float B = C * fmaf(-3.0f * k.t.k, s2, 1.0f);
    float P = -0.5f * C, Q = 1.5f * C * s2;
    if (r2 <= k.t.a4) {
        const bool apart = r2 > 0.0f;
        const float r = apart ? r2 * s : 0.0f;
        A = k.c6 * fmaf(-9.0f / 32.0f * k.t.ia, r, 1.0f);
        B = apart ? k.c6 * k.t.ia * (3.0f / 32.0f) * s : 0.0f;
        C = fmaf(-k.c1, r, k.c0);
        P = fmaf(k.p3 * r, r2, fmaf(-k.p1, r, k.p0));
        Q = apart ? k.q0 * fmaf(6.0f * k.a2, s, -r) : 0.0f;
    }
    const float cx = C * dx, cy = C * dy, cz = C * dz;
    {
        const float t = B * fmaf(dx, fj[0], fmaf(dy, fj[1], dz * fj[2]));
        vi[0] = fmaf(t, dx, fmaf(A, fj[0], vi[0]));
        vi[1] = fmaf(t, dy, fmaf(A, fj[1], vi[1]));
        vi[2] = fmaf(t, dz, fmaf(A, fj[2], vi[2]));
        if constexpr (SJ) {
            vi[0] = fmaf(fj[4], cz, fmaf(-fj[5], cy, vi[0]));
            vi[1] = fmaf(fj[5], cx, fmaf(-fj[3], cz, vi[1]));
            vi[2] = fmaf(fj[3], cy, fmaf(-fj[4], cx, vi[2]));
        }
        if constexpr (SI) {
            vi[3] = fmaf(fj[1], cz, fmaf(-fj[2], cy, vi[3]));
            vi[4] = fmaf(fj[2], cx, fmaf(-fj[0], cz, vi[4]));
            vi[5] = fmaf(fj[0], cy, fmaf(-fj[1], cx, vi[5]));
            if constexpr (SJ) {
                const float q = Q * fmaf(dx, fj[3], fmaf(dy, fj[4], dz * fj[5]));
                vi[3] = fmaf(q, dx, fmaf(P, fj[3], vi[3]));
                vi[4] = fmaf(q, dy, fmaf(P, fj[4], vi[4]));
                vi[5] = fmaf(q, dz, fmaf(P, fj[5], vi[5]));
            }
        }
    }
    {
        const float t = B * fmaf(dx, fi[0], fmaf(dy, fi[1], dz * fi[2]));
        vj[0] = fmaf(t, dx, fmaf(A, fi[0], vj[0]));
        vj[1] = fmaf(t, dy, fmaf(A, fi[1], vj[1]));
        vj[2] = fmaf(t, dz, fmaf(A, fi[2], vj[2]));
        if constexpr (SI) {
            vj[0] = fmaf(-fi[4], cz, fmaf(fi[5], cy, vj[0]));
            vj[1] = fmaf(-fi[5], cx, fmaf(fi[3], cz, vj[1]));
            vj[2] = fmaf(-fi[3], cy, fmaf(fi[4], cx, vj[2]));
        }
        if constexpr (SJ) {
            vj[3] = fmaf(-fi[1], cz, fmaf(fi[2], cy, vj[3]));
            vj[4] = fmaf(-fi[2], cx, fmaf(fi[0], cz, vj[4]));
            vj[5] = fmaf(-fi[0], cy, fmaf(fi[1], cx, vj[5]));
            if constexpr (SI) {
                const float q = Q * fmaf(dx, fi[3], fmaf(dy, fi[4], dz * fi[5]));
                vj[3] = fmaf(q, dx, fmaf(P, fi[3], vj[3]));
                vj[4] = fmaf(q, dy, fmaf(P, fi[4], vj[4]));
                vj[5] = fmaf(q, dz, fmaf(P, fi[5], vj[5]));
            }
        }
    }
}

}  // namespace cufil
