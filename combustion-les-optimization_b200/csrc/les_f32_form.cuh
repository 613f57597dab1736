// les_f32_form.cuh -- the arithmetic of the FP32 form's right-hand sides, operation by operation.
//
// A TENO candidate of the G equation counts or not by comparing its smoothness with a fixed number, and one
// candidate more or less moves a cell of the front by up to 1e-3 of G within a few steps.  Two
// FP32 forms that round differently anywhere (velocities, viscosity, flame speed, G itself) therefore part by
// that much at single cells.  So that an FP32 run stays the run it has always been, and a member of a
// group the solo run, every operation here and its order is fixed: the reference's formulas in the
// reference's order, with the fused multiply-adds written out, on a type whose products and sums the
// compiler does not contract further.  The FP64 form, whose picks are decided nine digits deeper,
// takes the shorter forms of les_kernels.cuh.
//
// The passes are bound by instruction issue (192x96x96: properties 86 %, flow 76 %, scalar 70 %; 922, 1131 and
// 1853 instructions a cell).  256x128x128, ms per step of four launches, with forms as short as the
// FP64 ones and with these: properties 0.505 and 0.530, flow 0.743 and 0.896, scalar 0.82 and 1.13.
#pragma once

#include "les_common.cuh"

namespace les {

struct Fl {
    float v;
    Fl() = default;
    __device__ __forceinline__ Fl(float x) : v(x) {}
    friend __device__ __forceinline__ Fl operator+(Fl a, Fl b) { return __fadd_rn(a.v, b.v); }
    friend __device__ __forceinline__ Fl operator-(Fl a, Fl b) { return __fsub_rn(a.v, b.v); }
    friend __device__ __forceinline__ Fl operator*(Fl a, Fl b) { return __fmul_rn(a.v, b.v); }
    friend __device__ __forceinline__ Fl operator-(Fl a) { return -a.v; }
    friend __device__ __forceinline__ bool operator<(Fl a, Fl b) { return a.v < b.v; }
    friend __device__ __forceinline__ bool operator>(Fl a, Fl b) { return a.v > b.v; }
    friend __device__ __forceinline__ bool operator<=(Fl a, Fl b) { return a.v <= b.v; }
    friend __device__ __forceinline__ bool operator>=(Fl a, Fl b) { return a.v >= b.v; }
};
__device__ __forceinline__ Fl mad(Fl a, Fl b, Fl c) { return __fmaf_rn(a.v, b.v, c.v); }
__device__ __forceinline__ Fl over(Fl a, Fl b) { return qdiv_normal(a.v, b.v); }     // b not subnormal
__device__ __forceinline__ Fl sum3(Fl a, Fl ra, Fl b, Fl rb, Fl c, Fl rc) { return mad(c, rc, mad(a, ra, b * rb)); }

// ---------------------------------------------------------------------------- properties

// cell_props_fast (les_kernels.cuh) for the FP32 form: the operations of the general path
// (cell_props_any) without its branches; species it skips take part with weight 0.
template <typename StoreD>
__device__ __forceinline__ bool f32_cell_props(const Consts& C, float T, const float* Yf, float rhof, const StoreD& store_d,
                                               CellProps<float>& o) {
    const ConstsF& K = C.f;
    Fl X[NSP], syw = 0.0f;
#pragma unroll
    for (int s = 0; s < NSP; s++) {
        X[s] = Fl(Yf[s]) * Fl(K.d_mwk[s].r);
        syw = s == 0 ? X[0] : syw + X[s];
    }
    if (!(C.fit_ok && T > (float)FIT_TMIN && T < (float)FIT_TMAX && syw.v >= 1e-9f && syw.v < 1e9f && rhof > 1e-3f &&
          rhof < 1e9f))
        return false;
    const Fl isyw = over(1.0f, syw);
    Fl w[NSP];
    bool pure = false;
#pragma unroll
    for (int s = 0; s < NSP; s++) {
        X[s] = X[s] * isyw;
        pure = pure || fabsf((Fl(1.0f) - X[s]).v) < 1e-9f;
        w[s] = X[s] > Fl(1e-12f) ? X[s] : Fl(0.0f);
    }
    if (pure) return false;
    const Fl L = qlog(T), L2 = L * L, L3 = L2 * L;
    auto fit = [&](const float (&c)[4]) { return mad(c[3], L3, mad(c[2], L2, mad(c[1], L, c[0]))); };
    {
        // Hirschfelder-Curtiss (:1716-1749), sums over b != a in ascending b
        Fl sx[NSP];
#pragma unroll
        for (int s = 0; s < NSP; s++) sx[s] = 0.0f;
#pragma unroll
        for (int a = 0; a < NSP; a++)
#pragma unroll
            for (int b = a + 1; b < NSP; b++) {
                const Fl y = Fl(qexp((-fit(K.dco[a][b])).v)) * Fl(1e4f);
                sx[a] = mad(w[b], y, sx[a]);
                sx[b] = mad(w[a], y, sx[b]);
            }
#pragma unroll
        for (int s = 0; s < NSP; s++) {
            const Fl d = over(Fl(1.0f) - X[s], sx[s]);
            o.D[s] = fmaxf(1e-9f, fminf(1e-2f, sx[s] > Fl(1e-12f) ? d.v : 1e-5f));
        }
        store_d(o.D);
    }
    Fl cp = 0.0f;
    {
        const Fl T1 = T, T2 = T1 * T1, T3 = T2 * T1, T4 = T2 * T2;
        auto add = [&](const float (&a)[7], int s) {
            const Fl cpr = mad(a[4], T4, mad(a[3], T3, mad(a[2], T2, mad(a[1], T1, a[0]))));
            cp = mad(Yf[s], (cpr * Fl((float)R_UNIV)) * Fl(K.d_mwk[s].r), cp);
        };
        if (T > K.t_split) {
#pragma unroll
            for (int s = 0; s < NSP; s++) add(K.nasa_high[s], s);
        } else {
#pragma unroll
            for (int s = 0; s < NSP; s++) add(K.nasa_low[s], s);
        }
    }
    const float Cp = fmaxf(100.0f, cp.v);
    // Wilke (:1530-1546) and Wassiljew (:1842-1863)
    Fl mu = 0.0f, lam = 0.0f, muk[NSP], rsmu[NSP];
#pragma unroll
    for (int s = 0; s < NSP; s++) {
        muk[s] = Fl(qexp(fit(K.eta[s]).v)) * Fl(0.1f);
        rsmu[s] = rsqrtf(muk[s].v);
    }
#pragma unroll
    for (int a = 0; a < NSP; a++) {
        const Fl smu = qsqrt(muk[a].v);
        Fl den = 0.0f;
#pragma unroll
        for (int b = 0; b < NSP; b++) {
            const Fl sr = a == b ? Fl(1.0f) : smu * rsmu[b];
            const Fl t = mad(sr, K.wpow[a][b], 1.0f);
            den = mad(w[b], (t * t) * Fl(K.d_wden[a][b].r), den);
        }
        const Fl wa = den > Fl(1e-9f) ? w[a] : Fl(0.0f), iden = den > Fl(1e-9f) ? over(1.0f, den) : Fl(0.0f);
        const Fl lamk = Fl(qexp(fit(K.lam[a]).v)) * Fl(1e-5f);
        mu = mad(wa * muk[a], iden, mu);
        lam = mad(wa * lamk, iden, lam);
    }
    o.cp = Cp;
    o.mu_mix = fmaxf(1e-7f, mu.v);
    o.lam = fmaxf(1e-3f, lam.v);
    o.nu = fmaxf(1e-7f, qdiv_normal(o.mu_mix, rhof));
    o.aT = qdiv_normal(o.lam, (Fl(rhof) * Fl(Cp)).v);
    o.alpha = fmaxf(1e-7f, o.aT);
    return true;
}

// Resolved strain (:1569-1680): |S|, nu_t, div u and the numerator of the SSR model.
__device__ __forceinline__ void f32_strain(const ConstsF& K, const ModelK<float>& M, const F11<float>& F, int id, int sI, int sJ,
                                           float G, float& Smag, float& nut, float& div, float& num) {
    auto d = [&](int q, int s) { return Fl(F.p[q][id + s]) - Fl(F.p[q][id - s]); };
    const Fl rx = K.d_2dx.r, ry = K.d_2dy.r, rz = K.d_2dz.r, half = 0.5f, two = 2.0f;
    const Fl S11 = d(0, sI) * rx, S22 = d(1, sJ) * ry, S33 = d(2, 1) * rz;
    const Fl S12 = half * mad(d(0, sJ), ry, d(1, sI) * rx), S13 = half * mad(d(0, 1), rz, d(2, sI) * rx),
             S23 = half * mad(d(1, 1), rz, d(2, sJ) * ry);
    const Fl off = mad(S23, S23, mad(S12, S12, S13 * S13));
    const Fl Sij = mad(S33, S33, mad(S22, S22, mad(S11, S11, two * off)));
    Smag = qsqrt((two * Sij).v);
    const Fl dv = (S11 + S22) + S33;
    float g = G;
    if (g < 0.0f) g = 0.0f;
    if (g > 1.0f) g = 1.0f;
    Fl cs = mad(Fl(M.cs_b) - Fl(M.cs_u), g, M.cs_u);
    cs = mad(Fl(M.cs_boost) * Fl(4.0f) * Fl(g), Fl(1.0f) - Fl(g), cs);
    const Fl l = cs * Fl(K.dx);
    nut = ((l * l) * Fl(Smag)).v;
    div = dv.v;
    num = mad(-(dv * dv), float(1.0 / 3.0), Sij).v;
}

// SSR-SGS turbulent flame speed (:1926-1957).  The wrinkling ratio (8 exp(c / (8 eta)) eta / dx)^(2 - D3) is below 1
// where 8 eta > dx and the exponent is negative (c >= 0); without dilatation the speed is then S_L
// whatever its value, and the exponential and the power are left out.
__device__ __forceinline__ float f32_flame_speed(const ConstsF& K, float num, float div, float nu) {
    const Fl dx = K.dx, X = over(K.dx4, Fl(nu) * Fl(nu)) * Fl(num);
    Fl d_eta = Fl(1.0f) + Fl((float)SMALL);      // D / eta + SMALL
    if (!(X < Fl((float)SMALL))) {
        const Fl pX = qpow(X.v, 0.75f), arg = Fl((float)SSR_B) * pX;
        d_eta = mad(Fl((float)SSR_A) * pX, arg > Fl(1.0f) ? qlog(arg.v) : 0.0f, (float)SMALL);
    }
    const Fl eta = over(dx, d_eta), dce = Fl(8.0f) * eta;
    const float dl = fmaxf(0.0f, div);
    if (!(dl > 0.0f) && K.ssr_exp <= 0.0f && K.ssr_cdF >= 0.0f && dce.v >= 1.001f * K.dx) return K.s_l;
    const Fl asf = Fl(8.0f) * Fl(qexp(over(K.ssr_cdF, dce + Fl((float)SMALL)).v));
    const Fl wr = qpow(((asf * eta) * Fl(K.d_dx.r)).v, K.ssr_exp);
    const Fl ratio = K.tau_sl > (float)SMALL ? mad(dx * Fl(dl), K.d_tau_sl.r, wr) : wr;
    return fmaxf(K.s_l, (Fl(K.s_l) * Fl(fmaxf(0.0f, ratio.v))).v);
}

// ---------------------------------------------------------------------------- G equation

// teno5_reconstruct (:2190-2236) of the two faces along the velocity, v0..v5 from three cells upstream to
// two downstream (mirrored for a negative velocity the reference's two branches are this one): the
// difference of the reconstructed values.  The faces share the second differences and one candidate.
__device__ __forceinline__ Fl f32_smooth(Fl aa, Fl b) { return Fl(float(13.0 / 12.0)) * aa + Fl(0.25f) * (b * b); }
__device__ __forceinline__ Fl f32_smooth_fused(Fl aa, Fl b) { return mad(float(13.0 / 12.0), aa, Fl(0.25f) * (b * b)); }
__device__ __forceinline__ Fl f32_teno_face(Fl i0, Fl i1, Fl i2, Fl p0, Fl p1, Fl p2, Fl p0_alone) {
    const float cut = (float)TENO_CUT;
    const bool d0 = i0 < cut, d1 = i1 < cut, d2 = i2 < cut;
    const Fl w0 = d0 ? 0.1f : 0.0f, w1 = d1 ? 0.6f : 0.0f, w2 = d2 ? 0.3f : 0.0f;
    // reciprocals of the weights' sums
    const Fl r = d1 ? (d0 ? (d2 ? 1.0f : float(1.0 / 0.7)) : (d2 ? float(1.0 / 0.9) : float(1.0 / 0.6)))
                    : (d0 ? (d2 ? 2.5f : 10.0f) : float(1.0 / 0.3));
    const Fl best = (i0 <= i1 && i0 <= i2) ? p0_alone : ((i1 <= i0 && i1 <= i2) ? p1 : p2);
    return (d0 || d1 || d2) ? mad(w2, p2, mad(w0, p0, w1 * p1)) * r : best;
}
// Smoothness ties decide as well: the outermost stencil's sum of each face ends in a fused multiply-add.
// Which products of the candidates are rounded before they are added depends on the face, the axis and the sign of
// the velocity, for the first candidate also on whether it is weighted or taken alone.
template <int AXIS>
__device__ __forceinline__ Fl f32_teno_diff(bool pos, Fl v0, Fl v1, Fl v2, Fl v3, Fl v4, Fl v5) {
    const Fl r6 = float(1.0 / 6.0), two = 2.0f, four = 4.0f;
    const Fl a1 = v0 - two * v1 + v2, a2 = v1 - two * v2 + v3, a3 = v2 - two * v3 + v4, a4 = v3 - two * v4 + v5;
    const Fl t1 = a1 * a1, t2 = a2 * a2, t3 = a3 * a3, t4 = a4 * a4;
    const Fl m3 = Fl(3.0f) * v2, p3 = Fl(3.0f) * v3;
    const Fl m0 = mad(11.0f, v2, mad(two, v0, -(Fl(7.0f) * v1))) * r6;
    const Fl m1 = (mad(5.0f, v2, -v1) + two * v3) * r6;
    const Fl m2 = ((pos ? two * v2 + Fl(5.0f) * v3 : mad(5.0f, v3, two * v2)) - v4) * r6;
    const Fl m = f32_teno_face(f32_smooth_fused(t1, v0 - four * v1 + m3), f32_smooth(t2, v1 - v3),
                               f32_smooth(t3, m3 - four * v3 + v4), m0, m1, m2, m0);
    const Fl p0a = mad(11.0f, v3, mad(-7.0f, v2, two * v1)) * r6;
    const Fl p0 = AXIS == 2 ? mad(11.0f, v3, mad(two, v1, -(Fl(7.0f) * v2))) * r6 : p0a;
    const Fl p1 = ((AXIS == 0 && pos ? Fl(5.0f) * v3 - v2 : mad(5.0f, v3, -v2)) + two * v4) * r6;
    const Fl p2 = (mad(5.0f, v4, two * v3) - v5) * r6;
    const Fl p = f32_teno_face(f32_smooth(t2, v1 - four * v2 + p3), f32_smooth(t3, v2 - v4),
                               f32_smooth_fused(t4, p3 - four * v4 + v5), p0, p1, p2, p0a);
    return p - m;
}

// calculate_weno5_gradient_1d (:735-827) times the spacing, from the cells -2..+3.
__device__ __forceinline__ Fl f32_weno_half(Fl i0, Fl i1, Fl i2, Fl g0, Fl g1, Fl g2, Fl s0, Fl s1, Fl s2) {
    const Fl eps = 1.0e-6f;
    const Fl e0 = eps + i0, e1 = eps + i1, e2 = eps + i2;
    const Fl a0 = over(g0, e0 * e0), a1 = over(g1, e1 * e1), a2 = over(g2, e2 * e2);
    const Fl y = qdiv(1.0f, (a0 + a1 + a2).v);
    return sum3(a0 * y, s0, a1 * y, s1, a2 * y, s2);
}
__device__ __forceinline__ Fl f32_weno_diff(Fl p0, Fl p1, Fl p2, Fl p3, Fl p4, Fl p5) {
    const Fl r6 = float(1.0 / 6.0), two = 2.0f, four = 4.0f;
    const Fl a1 = p0 - two * p1 + p2, a2 = p1 - two * p2 + p3, a3 = p2 - two * p3 + p4, a4 = p3 - two * p4 + p5;
    const Fl m3 = Fl(3.0f) * p2, h3 = Fl(3.0f) * p3;
    const Fl s0 = mad(11.0f, p3, mad(-7.0f, p2, two * p1)) * r6;
    const Fl s1 = (mad(5.0f, p3, -p2) + two * p4) * r6;
    const Fl s2 = (mad(5.0f, p4, two * p3) - p5) * r6;
    const Fl h = f32_weno_half(f32_smooth(a2 * a2, p1 - four * p2 + h3), f32_smooth(a3 * a3, p2 - p4),
                               f32_smooth_fused(a4 * a4, h3 - four * p4 + p5), 3.0f / 10.0f, 6.0f / 10.0f,
                               1.0f / 10.0f, s0, s1, s2);
    const Fl m0 = (mad(5.0f, p1, -p0) + two * p2) * r6;
    const Fl m1 = (mad(5.0f, p2, two * p1) - p3) * r6;
    const Fl m2 = (mad(-7.0f, p3, Fl(11.0f) * p2) + two * p4) * r6;
    const Fl l = f32_weno_half(f32_smooth_fused(a1 * a1, p0 - four * p1 + m3), f32_smooth(a2 * a2, p1 - p3),
                               f32_smooth_fused(a3 * a3, m3 - four * p3 + p4), 1.0f / 10.0f, 6.0f / 10.0f,
                               3.0f / 10.0f, m0, m1, m2);
    return h - l;
}

// Laplacian and SGS flux divergence (:2751-2760, :2853-2860) from a cell c and its neighbours
// p above and m below along each axis; gp and gm the SGS coefficients of the faces there.
__device__ __forceinline__ Fl f32_lap(const ConstsF& K, Fl c, const Fl (&p)[3], const Fl (&m)[3]) {
    const Fl c2 = Fl(2.0f) * c;
    return sum3(p[0] - c2 + m[0], K.d_dxx.r, p[1] - c2 + m[1], K.d_dyy.r, p[2] - c2 + m[2], K.d_dzz.r);
}
__device__ __forceinline__ Fl f32_sgs(const ConstsF& K, Fl c, const Fl (&p)[3], const Fl (&m)[3], const Fl (&gp)[3],
                                      const Fl (&gm)[3]) {
    const Fl r[3] = {K.d_dx.r, K.d_dy.r, K.d_dz.r};
    Fl s[3];
#pragma unroll
    for (int a = 0; a < 3; a++) s[a] = mad(gp[a] * (p[a] - c), r[a], -((gm[a] * (c - m[a])) * r[a]));
    return sum3(s[0], r[0], s[1], r[1], s[2], r[2]);
}

// Momentum (:2552-2697) and G (:2706-2825) right-hand sides of one fluid cell: flow_rhs of les_kernels.cuh.
__device__ __forceinline__ void f32_flow_rhs(const Consts& C, const ModelK<float>& M, const F11<float>& F,
                                             const PropBuf<float>& P, const Scalars* __restrict__ Sc, int i, int j, int k,
                                             int id, const FlowCell<float>& cell, float (&kv)[4]) {
    const float (&c0)[3] = cell.p0;
    const float g0 = cell.G0;
    const ConstsF& K = C.f;
    const int nx = C.nx, ny = C.ny, nz = C.nz;
    const int st[3] = {ny * nz, nz, 1};
    const Fl r[3] = {K.d_dx.r, K.d_dy.r, K.d_dz.r};
    const bool band2 = (i < 2 || i >= nx - 2 || j < 2 || j >= ny - 2 || k < 2 || k >= nz - 2);
    const bool band3 = (i < 3 || i >= nx - 3 || j < 3 || j >= ny - 3 || k < 3 || k >= nz - 3);
    const Fl half = 0.5f, r0 = cell.r0, G0 = g0, n0 = cell.n0;
    const float* __restrict__ G = F.p[4];
    Fl km[3];
    {
        Fl mp[3], mm[3];
#pragma unroll
        for (int x = 0; x < 3; x++) {
            const float* __restrict__ rho = F.p[5];
            const float* __restrict__ va = F.p[x];
            mp[x] = (half * (Fl(rho[id + st[x]]) + r0)) * (half * (Fl(va[id + st[x]]) + Fl(c0[x])));
            mm[x] = (half * (Fl(rho[id - st[x]]) + r0)) * (half * (Fl(va[id - st[x]]) + Fl(c0[x])));
        }
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const float* __restrict__ ph = F.p[q];
            const Fl c = c0[q];
            Fl p[3], m[3], d[3];
#pragma unroll
            for (int x = 0; x < 3; x++) {
                p[x] = ph[id + st[x]];
                m[x] = ph[id - st[x]];
                const Fl fp = band2 ? (mp[x] > Fl(0.0f) ? c : p[x]) : half * c + half * p[x];
                const Fl fm = band2 ? (mm[x] > Fl(0.0f) ? m[x] : c) : half * m[x] + half * c;
                d[x] = mad(mp[x], fp, -(mm[x] * fm));
            }
            km[q] = mad(cell.mu, f32_lap(K, c, p, m), -sum3(d[0], r[0], d[1], r[1], d[2], r[2]));
        }
    }
    Fl kG, lap, cen[3];
    {
        Fl p[3], m[3], gp[3], gm[3], t[3];
#pragma unroll
        for (int x = 0; x < 3; x++) {
            const bool pos = c0[x] >= 0.0f;
            const int o = pos ? -st[x] : st[x];
            const Fl U = G[id + o], Dn = G[id - o], nu = P.nu_t[id + o], nd = P.nu_t[id - o];
            p[x] = pos ? Dn : U;
            m[x] = pos ? U : Dn;
            gp[x] = ((pos ? nd : nu) + n0) * Fl(K.d_sct2.r);
            gm[x] = ((pos ? nu : nd) + n0) * Fl(K.d_sct2.r);
            const Fl va = fabsf(c0[x]);
            if (band2) t[x] = va * (G0 - U);                     // first-order upwind (:642-651)
            else if (band3) t[x] = Fl(c0[x]) * ((half * G0 + half * p[x]) - (half * m[x] + half * G0));   // :652-677
            else {
                const Fl U3 = G[id + 3 * o], U2 = G[id + 2 * o], D2 = G[id - 2 * o];
                t[x] = va * (x == 0   ? f32_teno_diff<0>(pos, U3, U2, U, G0, Dn, D2)
                             : x == 1 ? f32_teno_diff<1>(pos, U3, U2, U, G0, Dn, D2)
                                      : f32_teno_diff<2>(pos, U3, U2, U, G0, Dn, D2));
            }
            cen[x] = p[x] - m[x];
        }
        const Fl conv = band2   ? mad(t[0], r[0], t[1] * r[1]) + t[2] * r[2]
                        : band3 ? sum3(t[0], r[0], t[1], r[1], t[2], r[2])
                                : t[0] * r[0] + t[1] * r[1] + t[2] * r[2];
        lap = f32_lap(K, G0, p, m);
        const Fl sgs = f32_sgs(K, G0, p, m, gp, gm);
        Fl g[3];
        if (Sc->t_loop >= C.weno_step && !band3) {
#pragma unroll
            for (int x = 0; x < 3; x++)
                g[x] = f32_weno_diff(G[id - 2 * st[x]], m[x], G0, p[x], G[id + 2 * st[x]], G[id + 3 * st[x]]) * r[x];
        } else {
            g[0] = cen[0] * Fl(K.d_2dx.r);
            g[1] = cen[1] * Fl(K.d_2dy.r);
            g[2] = cen[2] * Fl(K.d_2dz.r);
        }
        const Fl gmag = qsqrt(sum3(g[0], g[0], g[1], g[1], g[2], g[2]).v);
        if (P.grad_g) P.grad_g[id] = gmag.v;   // grad_G_magnitude_for_debug (:2783)
        kG = (Fl(P.ST[id]) * gmag - conv) + sgs;
    }
    Fl fo[3] = {0.0f, 0.0f, 0.0f}, art = 0.0f;
    if (C.flame_accel && g0 > 0.01f && g0 < 0.99f) {
        const Fl df = G0 - Fl(M.accel_center);
        const Fl window = qexp((-(df * df) * Fl(M.d_w2.r)).v);
        const Fl zp = Fl((float)k) * Fl(K.dz);
        const Fl ramp = zp < Fl((float)RAMP_DIST) ? zp * Fl(K.d_ramp.r) : Fl(1.0f);
        // tip_mask is the literal 1.0 in the momentum source (:2638)
        const Fl cf = Fl(M.accel_strength) * r0 * window;
        const Fl gx = cen[0] * Fl(K.d_2dx.r), gy = cen[1] * Fl(K.d_2dy.r), gz = cen[2] * Fl(K.d_2dz.r);
        const bool above = mad((float)k, K.dz, -Fl(K.inlet_center_z)) > Fl(0.0f);
        fo[0] = cf * (gx < Fl(0.0f) ? Fl(0.0f) : gx) * Fl(0.05f) * ramp;
        fo[1] = cf * (gy < Fl(0.0f) ? Fl(0.0f) : gy) * ramp;
        fo[2] = cf * ((above ? gz < Fl(0.0f) : gz > Fl(0.0f)) ? Fl(0.0f) : gz) * ramp;
        // tip_mask = 1 - exp(-r^2 / 0^2) is exactly 1 for every fluid cell (j >= 1)
        // because TIP_PROTECTION_RADIUS is 0.0 (:234, :2806-2807).
        if (g0 > 0.1f) art = Fl(5.0f) * (n0 + Fl(1.0e-5f)) * window * lap;
    }
    const Fl lim = (float)FORCE_LIMIT;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        if (fo[q] > lim) fo[q] = lim;
        if (fo[q] < -lim) fo[q] = -lim;
    }
    kv[0] = (mad(r0 - Fl((float)Sc->rho_avg), (float)G_GRAVITY, km[0]) + fo[0]).v;
    kv[1] = (km[1] + fo[1]).v;
    kv[2] = (km[2] + fo[2]).v;
    kv[3] = (kG + art).v;
}

// ---------------------------------------------------------------------------- scalars

// Half the limited slope of a face (:2017-2028, :2058-2094), 0.5 superbee(a / b), to be multiplied by b: a the
// difference across the face behind, b across the face itself.  superbee takes 0, 1 or 2 over whole ranges
// of the quotient, and there exact comparisons of |a| and |b| decide; where it is the quotient or its double,
// that is the hardware's.  A NaN in a gives 2, as the reference's does, and |b| < SMALL too (it sets r = 1e9).
__device__ __forceinline__ Fl f32_half_superbee(float a, float b) {
    const float m = fabsf(a), n = fabsf(b), q = qdiv_normal(a, b);
    const float low = m > 0.5f * n ? 0.5f : fminf(q, 0.5f);
    const float high = m >= 2.0f * n ? 1.0f : fmaxf(0.5f, fminf(0.5f * q, 1.0f));
    const float h = m <= n ? low : high;
    return n < (float)SMALL ? 1.0f : q < 0.0f ? 0.0f : h;
}

// One scalar of a cell (:2837-2962): target nudging - advection + molecular + SGS diffusion, c the cell,
// up/dn/uu its neighbours along the velocity as in Star, gp/gm the SGS coefficients above and below; the
// target is the product of the last two.  FUSED is whether the upwind sum of the band next to the faces ends in a
// fused multiply-add (T and Y0).
template <bool FUSED, typename S>
__device__ __forceinline__ float f32_scalar_rhs(const ConstsF& K, const S& q, const bool (&pos)[3], bool band2,
                                                const float (&vel)[3], const Fl (&gp)[3], const Fl (&gm)[3], Fl D, Fl relax,
                                                Fl to, Fl toward) {
    const Fl r[3] = {K.d_dx.r, K.d_dy.r, K.d_dz.r}, c = q.c;
    Fl p[3], m[3], t[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const Fl up = q.up[a], dn = q.dn[a];
        p[a] = pos[a] ? dn : up;
        m[a] = pos[a] ? up : dn;
        const Fl d1 = up - Fl(q.uu[a]), d2 = c - up, d3 = dn - c;
        const Fl d = band2 ? d2 : mad(f32_half_superbee(d2.v, d3.v), d3, c) - mad(f32_half_superbee(d1.v, d2.v), d2, up);
        t[a] = Fl(fabsf(vel[a])) * d;
    }
    const Fl xy = t[0] * r[0] + t[1] * r[1];
    const Fl conv = band2 ? (FUSED ? mad(t[2], r[2], xy) : xy + t[2] * r[2]) : sum3(t[0], r[0], t[1], r[1], t[2], r[2]);
    const Fl sgs = f32_sgs(K, c, p, m, gp, gm);
    return mad(relax, mad(to, toward, -c), mad(D, f32_lap(K, c, p, m), -conv) + sgs).v;
}

}  // namespace les
