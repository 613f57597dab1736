// les_kernels.cuh -- solver-step kernels, templated on the field type R (double for the
// plain form, float for the precision form).  Global sums and maxima are always
// accumulated in double.
//
// One RK4 stage is four passes over the grid:
//   A  k_filter       : 7-point box filter of the 11 stage fields (apply_box_filter,
//                       les_combustion_solver.c:1307-1470); partial sums for <rho_f>.
//   B  k_props        : cell-local mixture properties (update_nu_mix :1489, update_Dk :1684,
//                       update_Cp_mix :1762, update_lambda_mix_alpha :1798), resolved strain,
//                       G-dependent Smagorinsky nu_t (calculate_nu_t :1569), SSR-SGS flame
//                       speed (:1913) and mu_eff = mu + rho_f nu_t.
//   C1 k_rhs_scalar   : species and temperature right-hand sides (:2837-2962) fused with
//                       the RK4 stage update (:4432-4455) or the final combine (:4517-4544)
//                       of T, Y_k and rho; the new density is handed to C2.
//   C2 k_rhs_flow     : momentum and G right-hand sides (calculate_RHS :2552-2825) fused with
//                       the same update of u, v, w and G.
// After the fourth stage one kernel over the faces replays apply_boundary_conditions
// (:2967-3161) in the reference's face order.
//
// Every kernel takes the constant table by value (__grid_constant__): divisors, their
// reciprocals and the species data are read from the constant bank.  The arithmetic is explicit
// about contraction, so that every instance of a kernel gives the same bits: the FP64 unit is built
// without it, with fma() where it is wanted, and the FP32 form's right-hand sides and properties are those of
// les_f32_form.cuh.
#pragma once

#include <type_traits>

#include "les_common.cuh"

namespace les {

template <typename R>
struct F11 {                 // u v w T G rho Y0..Y4
    R* p[NSTATE];
};
template <typename R>
struct PropBuf {
    R* mu_mix;
    R* nu;
    R* D[NSP];
    R* aT;                   // lambda / (rho_f Cp), or 0 when the reference skips the term
    R* nu_t;
    R* S_mag;
    R* ST;
    R* mu_eff;
    R* dbg_cp;               // optional (nullptr): Cp, lambda, alpha for inspection
    R* dbg_lam;
    R* dbg_alpha;
    R* grad_g;               // optional (nullptr): |grad G| of the last RHS evaluation
};
template <typename R>
struct AccBuf {              // RK4 running sum of k: rhou rhov rhow T G Y0..Y4
    R* p[NACC];
};
template <typename R>
struct KDbg {                // optional (nullptr): the stage's k-arrays for inspection
    R* p[NACC];
};

// What the properties of a cell are kept in.
template <typename R>
struct CellProps {
    R D[NSP], mu_mix, nu, aT, cp, lam, alpha;
};

// What the flow pass loads of a cell before it knows its attribute.
template <typename R>
struct FlowCell {
    R p0[3], r0, G0, n0, mu;
    __device__ __forceinline__ void load(const F11<R>& F, const PropBuf<R>& P, int id) {
        p0[0] = F.p[0][id]; p0[1] = F.p[1][id]; p0[2] = F.p[2][id];
        r0 = F.p[5][id]; G0 = F.p[4][id]; n0 = P.nu_t[id]; mu = P.mu_eff[id];
    }
};

}  // namespace les

#include "les_f32_form.cuh"

namespace les {

#define LES_KERNEL_CONSTS const __grid_constant__ Consts C

// A member's fields in a batched launch: every per-cell field lives in the member's arena at
// the same offset as in the first member's, so its pointers are the first member's shifted by
// the arenas' distance.  Optional buffers outside the arena (inspection, |grad G|) are off in
// batched launches.
template <typename T>
__device__ __forceinline__ void shift_all(T& s, long long d) {
#pragma unroll
    for (int q = 0; q < (int)(sizeof(s.p) / sizeof(s.p[0])); q++) s.p[q] = shifted(s.p[q], d);
}
template <typename R>
__device__ __forceinline__ void shift_props(PropBuf<R>& P, long long d) {
    P.mu_mix = shifted(P.mu_mix, d);
    P.nu = shifted(P.nu, d);
#pragma unroll
    for (int s = 0; s < NSP; s++) P.D[s] = shifted(P.D[s], d);
    P.aT = shifted(P.aT, d);
    P.nu_t = shifted(P.nu_t, d);
    P.S_mag = shifted(P.S_mag, d);
    P.ST = shifted(P.ST, d);
    P.mu_eff = shifted(P.mu_eff, d);
    P.dbg_cp = P.dbg_lam = P.dbg_alpha = nullptr;
    P.grad_g = nullptr;
}

// Minimum resident blocks per SM requested from the register allocator (properties / flow /
// scalar).  Swept on B200 at 256x128x128, ms per step (four launches): FP64 properties 1.13 at 5
// blocks, 1.11 at 4, 1.16 at 3, 1.32 at 2; flow 0.95 at 5, 0.91 at 4, 1.01 at 3, 1.29 at 2; scalar
// 1.40 at 5, 1.38 at 4, 1.51 at 3 and 2; FP32 properties 0.530 at 6 and 5, 0.560 at 4; flow 0.916
// at 6, 0.900 at 5, 0.906 at 4; scalar 1.11 at 6 (96x48x48 0.109), 1.14 at 5 (0.097), 1.33 at 3.
#ifndef LES_MINB_PROPS
#define LES_MINB_PROPS 4
#endif
#ifndef LES_MINB_FLOW
#define LES_MINB_FLOW 4
#endif
#ifndef LES_MINB_SCALAR
#define LES_MINB_SCALAR 4
#endif
#ifndef LES_MINB_PROPS_F32
#define LES_MINB_PROPS_F32 6
#endif
#ifndef LES_MINB_FLOW_F32
#define LES_MINB_FLOW_F32 5
#endif
#ifndef LES_MINB_SCALAR_F32
#define LES_MINB_SCALAR_F32 5
#endif
template <typename R>
struct MinBlocks {
    static constexpr int props = LES_MINB_PROPS, flow = LES_MINB_FLOW,
                         scalar = LES_MINB_SCALAR;
};
template <>
struct MinBlocks<float> {
    static constexpr int props = LES_MINB_PROPS_F32, flow = LES_MINB_FLOW_F32,
                         scalar = LES_MINB_SCALAR_F32;
};
// The same register budget for a block of `ntb` threads: the resident threads per SM of the
// 256-thread budget in whole blocks (at least one).
constexpr int lb_blocks(int minb, int ntb) { return (minb * NT) / ntb > 0 ? (minb * NT) / ntb : 1; }

// ---------------------------------------------------------------------------- helpers

// The scalar and flow passes read Phi_n and the RK running sum once per stage, the scalar pass the
// diffusivities too, and write the running sum back for the next stage only: these go through
// ld.global.cs / st.global.cs (evict first), so they do not push the stencil fields' halo planes out of
// L2.  The FP64 scalar pass moves 318 bytes a cell per launch so, 326 of them its own fields.
#ifndef LES_SCALAR_STREAM
#define LES_SCALAR_STREAM 1
#endif
template <typename T>
__device__ __forceinline__ T ld_stream(const T* p) {
    if constexpr (LES_SCALAR_STREAM != 0) return __ldcs(p);
    else return *p;
}
template <typename T>
__device__ __forceinline__ void st_stream(T* p, T v) {
    if constexpr (LES_SCALAR_STREAM != 0) __stcs(p, v);
    else *p = v;
}

template <typename R>
__device__ __forceinline__ R fit_prop(const R co[4], int zero, R L, R L2, R L3) {
    // calculate_property_from_fit (:385-391): exp(a0 + a1 L + a2 L^2 + a3 L^3); the T <= 0
    // guard is handled by the callers.
    if (zero) return R(0);
    R lp = (R)co[0] + (R)co[1] * L + (R)co[2] * L2 + (R)co[3] * L3;
    return qexp(lp);
}

// update_rho_from_EOS (:1894-1905) on the FP64 state, with the state division of the precision form
// Form.  In the FP64 form the gas constant of the mixture is multiplied out (rho = p / ((R sum Y_k / M_k) T):
// one division instead of three); the FP32 form keeps its three (les_f32_form.cuh says why).
template <typename Form>
__device__ __forceinline__ double eos_rho_state(const Consts& C, double T, const double Y[NSP], double fallback) {
    if constexpr (std::is_same<Form, float>::value) {
        double syw = cdv(Y[0], C.d_mwk[0]);
#pragma unroll
        for (int s = 1; s < NSP; s++) syw += cdv(Y[s], C.d_mwk[s]);
        if (syw > 1e-9 && T > 1.0)
            return sdiv<Form>(P_CONST, __dmul_rn(sdiv<Form>(R_UNIV, sdiv<Form>(1.0, syw)), T));
    } else {
        double syw = Y[0] * C.d_mwk[0].r;
#pragma unroll
        for (int s = 1; s < NSP; s++) syw = fma(Y[s], C.d_mwk[s].r, syw);
        if (syw > 1e-9 && T > 1.0) return sdiv<Form>(P_CONST, (R_UNIV * syw) * T);
    }
    return fallback;
}

// Mass fractions brought to the sum 1 where it is above `least` (:4447, :3152): one reciprocal, the
// quotients sharing it corrected with one fma each.
template <typename Form>
__device__ __forceinline__ bool renormalise(double* Y, double least) {
    double sy = 0.0;
#pragma unroll
    for (int s = 0; s < NSP; s++) sy += Y[s];
    if (!(sy > least)) return false;
    const double y = srecip<Form>(sy);
#pragma unroll
    for (int s = 0; s < NSP; s++) Y[s] = cquot(Y[s], sy, y);
    return true;
}

__device__ __forceinline__ bool off_faces(const Consts& C, int i, int j, int k) {
    return i >= 1 && i < C.nx - 1 && j >= 1 && j < C.ny - 1 && k >= 1 && k < C.nz - 1;
}
// A cell of a face or the one next to it, which the boundary conditions copy.
__device__ __forceinline__ bool beside_face(const Consts& C, int i, int j, int k) {
    return i < 2 || i >= C.nx - 2 || j < 2 || j >= C.ny - 2 || k < 2 || k >= C.nz - 2;
}

// Cell-local mixture properties of one fluid cell (attr == 3), general path: any temperature, any
// composition, any fits, by the reference's own rules term by term.  Called, not inlined: ordinary
// cells (cell_props_fast) never come here, and the instructions of this path in their way cost the
// pass instruction-cache misses.
template <typename R>
__device__ __noinline__ void cell_props_any(const Consts& C, R Tl, const R* Yf, R rhof, CellProps<R>* out) {
    const auto& K = kc<R>(C);
    R &mu_mix = out->mu_mix, &nu = out->nu, &aT = out->aT, &cp_out = out->cp, &lam_out = out->lam, &alpha = out->alpha;
    auto store_d = [&](const R* D) {
        for (int s = 0; s < NSP; s++) out->D[s] = D[s];
    };
    R X[NSP];
    R syw = R(0);
    bool tpos = Tl > R(0);
    R ym[NSP];
#pragma unroll
    for (int s = 0; s < NSP; s++) ym[s] = cdv(Yf[s], K.d_mwk[s]);
    if (tpos) {
#pragma unroll
        for (int s = 0; s < NSP; s++) syw += ym[s];
    }
    bool ok = tpos && !(syw < R(1e-9));
    // Cp (:1772-1786) -- independent of the mole fractions
    R Cp;
    if (!tpos) {
        Cp = R(1000.0);
    } else {
        R T2 = Tl * Tl, T3 = pow3_rn(Tl), T4 = pow4_rn(Tl);
        R cp = R(0);
#pragma unroll
        for (int s = 0; s < NSP; s++) {
            const auto* a = (Tl > (R)K.t_mid[s]) ? K.nasa_high[s] : K.nasa_low[s];
            R cpr = (R)a[0] + (R)a[1] * Tl + (R)a[2] * T2 + (R)a[3] * T3 + (R)a[4] * T4;
            R cpm = cpr * (R)R_UNIV;
            R cpk = (K.mwk[s] < R(1e-9)) ? R(1000.0) : cdv(cpm, K.d_mwk[s]);
            cp += Yf[s] * cpk;
        }
        Cp = fmax(R(100.0), cp);
    }
    cp_out = Cp;
    if (!ok) {
        nu = R(1.5e-5);
        mu_mix = R(1.8e-5);
        R D[NSP];
#pragma unroll
        for (int s = 0; s < NSP; s++) D[s] = R(1e-5);
        store_d(D);
        R lam = R(0.025);
        lam_out = lam;
        alpha = R(1.8e-5);
        aT = (rhof > R(1e-6) && Cp > R(1e-6)) ? qdiv(lam, rhof * Cp) : R(0);
        return;
    }
    // The FP32 form takes reciprocals once where the FP64 form (the reference's arithmetic)
    // divides per term.
    constexpr bool kF32 = std::is_same<R, float>::value;
    if constexpr (kF32) {
        const R isyw = qdiv(R(1.0), syw);
#pragma unroll
        for (int s = 0; s < NSP; s++) X[s] = ym[s] * isyw;
    } else {
        const R ysyw = qdiv(R(1.0), syw);
#pragma unroll
        for (int s = 0; s < NSP; s++) X[s] = mdiv(ym[s], syw, ysyw);
    }
    const R L = qlog(Tl);
    const R L2 = L * L;
    const R L3 = pow3_rn(L);
    {
        // Hirschfelder-Curtiss (:1716-1749): sx_a = sum over b != a (ascending b) of X_b / D_ab.
        // With a symmetric fit table each D_ab is evaluated once per unordered pair and both
        // sums take their term from it; the rows are visited in ascending order, so each sx_a
        // still receives its terms in ascending b.  1 / D_ab is taken directly as
        // exp(-P_ab(ln T)) * 1e4 (D_ab = exp(P_ab) * 1e-4), one exponential and no division: the
        // terms X_b / D_ab differ from the reference's quotients by at most ~2 ulp (the FP64
        // property pass 2.82 -> 2.53 ms per 256x128x128 step); the skip rule D_ab > 1e-12 reads
        // 1 / D_ab < 1e12.
        R sxa[NSP], D[NSP];
#pragma unroll
        for (int a = 0; a < NSP; a++) sxa[a] = R(0);
        if (C.dco_sym) {
#pragma unroll
            for (int a = 0; a < NSP; a++)
#pragma unroll
                for (int b = a + 1; b < NSP; b++) {
                    if (!(X[a] > R(1e-12) || X[b] > R(1e-12))) continue;
                    if (C.dco_zero[a][b]) continue;          // D_ab = 0 fails D_ab > 1e-12
                    const auto& co = K.dco[a][b];
                    const R lp = (R)co[0] + (R)co[1] * L + (R)co[2] * L2 + (R)co[3] * L3;
                    const R y = qexp(-lp) * R(1e4);
                    if (!(y < R(1e12))) continue;
                    if (X[b] > R(1e-12)) sxa[a] += X[b] * y;
                    if (X[a] > R(1e-12)) sxa[b] += X[a] * y;
                }
        } else {
#pragma unroll
            for (int a = 0; a < NSP; a++)
#pragma unroll
                for (int b = 0; b < NSP; b++) {
                    if (a == b || !(X[b] > R(1e-12))) continue;
                    const R v = fit_prop<R>(K.dco[a][b], C.dco_zero[a][b], L, L2, L3) * R(1e-4);
                    if (v > R(1e-12)) sxa[a] += qdiv(X[b], v);
                }
        }
#pragma unroll
        for (int a = 0; a < NSP; a++) {
            const R sx = sxa[a];
            R Dv;
            if (fabs(R(1.0) - X[a]) < R(1e-9)) {
                int o = (a != N2) ? N2 : O2;
                Dv = fit_prop<R>(K.dco[a][o], C.dco_zero[a][o], L, L2, L3) * R(1e-4);
            } else if (sx > R(1e-12)) {
                Dv = qdiv(R(1.0) - X[a], sx);
            } else {
                Dv = R(1e-5);
            }
            // pressure correction PATM / (p0 + P_f) (:1743-1746): P is identically zero in the
            // reference (it is never assigned a non-zero value), so the factor is exactly 1.
            D[a] = fmax(R(1e-9), fmin(R(1e-2), Dv));
        }
        store_d(D);
    }
    // pure-species viscosity and conductivity (:394-398, :431-437)
    // species with X < 1e-12 take no part in either mixing rule: their pure-species values
    // are not evaluated
    R muk[NSP];
#pragma unroll
    for (int s = 0; s < NSP; s++) {
        muk[s] = R(1.0);
        if (!(X[s] < R(1e-12))) muk[s] = fit_prop<R>(K.eta[s], C.eta_zero[s], L, L2, L3) * R(0.1);
    }
    // Wilke (:1530-1546) and Wassiljew (:1842-1863) share the same phi_ij, the same skip
    // rule and the same summation order, so one denominator per species serves both.
    // sqrt(mu_a / mu_b) is taken as sqrt(mu_a) * (1 / sqrt(mu_b)): 5 square roots and 5
    // reciprocals instead of 20 quotients and 20 square roots.  In FP64 this differs from the
    // reference's sqrt of the rounded quotient by at most 2 ulp (the FP64 property pass went
    // from 3.02 to 2.77 ms per 256x128x128 step); mu_a / mu_a stays exactly 1 for a positive
    // finite mu_a.
    R mu = R(0), lam = R(0);
    R rsmu[NSP];
#pragma unroll
    for (int s = 0; s < NSP; s++) {
        rsmu[s] = R(1.0);
        if (X[s] < R(1e-12)) continue;
        if constexpr (kF32) rsmu[s] = rsqrtf(muk[s]);
        else rsmu[s] = qdiv(R(1.0), qsqrt(muk[s]));
    }
#pragma unroll
    for (int a = 0; a < NSP; a++) {
        if (X[a] < R(1e-12)) continue;
        const R smu_a = qsqrt(muk[a]);
        R den = R(0);
#pragma unroll
        for (int b = 0; b < NSP; b++) {
            if (X[b] < R(1e-12)) continue;
            // as in the reference, a zero or infinite mu_a gives NaN on the diagonal too
            const R sr = (a == b && muk[a] > R(0) && muk[a] <= R(1e300)) ? R(1.0) : smu_a * rsmu[b];
            R t = R(1.0) + sr * (R)K.wpow[a][b];
            R ph = cdv(t * t, K.d_wden[a][b]);
            den += X[b] * ph;
        }
        if (den > R(1e-9)) {
            // the pure-species conductivity only where it is used
            const R lamk = fit_prop<R>(K.lam[a], C.lam_zero[a], L, L2, L3) * R(1e-5);
            if constexpr (kF32) {
                const R iden = qdiv(R(1.0), den);
                mu += (X[a] * muk[a]) * iden;
                lam += (X[a] * lamk) * iden;
            } else {
                const R yden = qdiv(R(1.0), den);
                mu += mdiv(X[a] * muk[a], den, yden);
                lam += mdiv(X[a] * lamk, den, yden);
            }
        }
    }
    mu_mix = fmax(R(1e-7), mu);
    R nuv = (rhof > R(1e-3)) ? qdiv(mu_mix, rhof) : R(1.5e-5);
    nu = fmax(R(1e-7), nuv);
    R lmix = fmax(R(1e-3), lam);
    lam_out = lmix;
    R q = R(0);
    bool qok = (rhof > R(1e-6) && Cp > R(1e-6));
    if (qok) q = qdiv(lmix, rhof * Cp);
    alpha = fmax(R(1e-7), qok ? q : R(1.8e-5));
    aT = q;
}

// The same for an ordinary cell: FIT_TMIN < T < FIT_TMAX, some mass, no pure species, fits that
// passed the host's check.  False where the cell is not one.  No branches but the choice of
// NASA range: species below the reference's X = 1e-12 take part with weight 0, which is what its
// skips amount to.  Against the general path per cell: 20 exponentials of 17 instructions
// instead of about 35 each (exp2_fit; the unit factors and 1/2 of the square roots are in the
// fits), no square roots, Wilke's denominators folded into two constants a pair, cp as one
// polynomial of the mixture, and reciprocals without the general division's checks.
// The diffusivities go to store_d as soon as they are known, so that they are not held across the
// mixing rules.
template <typename R, typename StoreD>
__device__ __forceinline__ bool cell_props_fast(const Consts& C, const double* tab, R Tl, const R* Yf, R rhof,
                                                const StoreD& store_d, CellProps<R>& o) {
    const auto& K = kc<R>(C);
    R X[NSP];
    R syw = R(0);
#pragma unroll
    for (int s = 0; s < NSP; s++) {
        X[s] = Yf[s] * K.d_mwk[s].r;
        syw += X[s];
    }
    if (!(C.fit_ok && Tl > R(FIT_TMIN) && Tl < R(FIT_TMAX) && syw >= R(1e-9) && syw < R(1e9) && rhof > R(1e-3) &&
          rhof < R(1e9)))
        return false;
    const R isyw = frcp(syw);
    bool pure = false;
#pragma unroll
    for (int s = 0; s < NSP; s++) {
        X[s] *= isyw;
        pure = pure || fabs(R(1.0) - X[s]) < R(1e-9);
    }
    if (pure) return false;
    const R L = qlog(Tl);
    auto fit = [&](const auto& c) { return exp2_fit(fma(fma(fma((R)c[3], L, (R)c[2]), L, (R)c[1]), L, (R)c[0]), tab); };
    R w[NSP];
#pragma unroll
    for (int s = 0; s < NSP; s++) w[s] = X[s] > R(1e-12) ? X[s] : R(0);
    {
        // Hirschfelder-Curtiss (:1716-1749), sums over b != a in ascending b; the pressure factor
        // PATM / (p0 + P_f) (:1743-1746) is exactly 1, P being identically zero in the reference
        R sx[NSP];
#pragma unroll
        for (int s = 0; s < NSP; s++) sx[s] = R(0);
        int p = 0;
#pragma unroll
        for (int a = 0; a < NSP; a++)
#pragma unroll
            for (int b = a + 1; b < NSP; b++, p++) {
                const R y = fit(K.f_idif[p]);
                sx[a] = fma(w[b], y, sx[a]);
                sx[b] = fma(w[a], y, sx[b]);
            }
#pragma unroll
        for (int s = 0; s < NSP; s++) {
            const R d = (R(1.0) - X[s]) * frcp(sx[s]);
            o.D[s] = fmax(R(1e-9), fmin(R(1e-2), sx[s] > R(1e-12) ? d : R(1e-5)));
        }
        store_d(o.D);
    }
    // cp (:1772-1786)
    R c[5];
#pragma unroll
    for (int q = 0; q < 5; q++) c[q] = R(0);
    if (Tl > K.t_split) {
#pragma unroll
        for (int s = 0; s < NSP; s++)
#pragma unroll
            for (int q = 0; q < 5; q++) c[q] = fma(Yf[s], (R)K.cp_high[s][q], c[q]);
    } else {
#pragma unroll
        for (int s = 0; s < NSP; s++)
#pragma unroll
            for (int q = 0; q < 5; q++) c[q] = fma(Yf[s], (R)K.cp_low[s][q], c[q]);
    }
    const R Cp = fmax(R(100.0), fma(fma(fma(fma(c[4], Tl, c[3]), Tl, c[2]), Tl, c[1]), Tl, c[0]));
    // Wilke (:1530-1546) and Wassiljew (:1842-1863): the same phi_ab, skip rule and order of
    // summation, so one denominator serves both; phi_ab = (w0 + w1 sqrt(mu_a / mu_b))^2, phi_aa = 1
    R smu[NSP], ismu[NSP];
#pragma unroll
    for (int s = 0; s < NSP; s++) {
        smu[s] = fit(K.f_smu[s]);
        ismu[s] = frcp(smu[s]);
    }
    R mu = R(0), lam = R(0);
#pragma unroll
    for (int a = 0; a < NSP; a++) {
        R den = w[a];
#pragma unroll
        for (int b = 0; b < NSP; b++) {
            if (b == a) continue;
            const R t = fma(smu[a] * ismu[b], (R)K.w1[a][b], (R)K.w0[a][b]);
            den = fma(w[b] * t, t, den);
        }
        const R q = den > R(1e-9) ? w[a] * frcp(den) : R(0);
        mu = fma(q * smu[a], smu[a], mu);
        lam = fma(q, fit(K.f_lam[a]), lam);
    }
    o.cp = Cp;
    o.mu_mix = fmax(R(1e-7), mu);
    o.lam = fmax(R(1e-3), lam);
    const R rc = rhof * Cp, irc = frcp(rc);
    o.nu = fmax(R(1e-7), cquot(o.mu_mix, rhof, Cp * irc));
    o.aT = cquot(o.lam, rc, irc);
    o.alpha = fmax(R(1e-7), o.aT);
    return true;
}

// ------------------------------------------------------------------ pass A: filter

// Block partials of one or more reductions into part[q * nblk + block]; true in the last block to
// arrive, whose threads may then reduce them and change what the blocks have read.  The block
// arrives only when all its threads have come here, so what they read before is read.
__device__ __forceinline__ bool last_block(double* part, unsigned nblk, unsigned bid, const double* v, int nv,
                                           unsigned* counter, int tid) {
    __shared__ bool last;
    __syncthreads();
    if (tid == 0) {
        for (int q = 0; q < nv; q++) part[(size_t)q * nblk + bid] = v[q];
        __threadfence();
        last = atomicAdd(counter, 1u) == nblk - 1;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// V consecutive values as 16-byte loads and stores.
template <typename T, int V>
__device__ __forceinline__ void ld_vec(const T* __restrict__ p, T (&v)[V]) {
    if constexpr (V == 1) {
        v[0] = __ldg(p);
    } else if constexpr (sizeof(T) == 8) {
        const double2 t = __ldg(reinterpret_cast<const double2*>(p));
        v[0] = t.x; v[1] = t.y;
    } else {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p));
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
}
template <int V>
__device__ __forceinline__ void st_vec(double* p, const double (&v)[V]) {
    if constexpr (V == 1) *p = v[0];
    else *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
}
template <int V>
__device__ __forceinline__ void st_vec(float* p, const float (&v)[V]) {
    if constexpr (V == 1) *p = v[0];
    else if constexpr (V == 2) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
    else *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
// V attribute bytes; id is a multiple of V.
template <int V>
__device__ __forceinline__ void ld_attr(const uint8_t* __restrict__ p, int (&a)[V]) {
    if constexpr (V == 1) {
        a[0] = __ldg(p);
    } else if constexpr (V == 2) {
        const uchar2 t = __ldg(reinterpret_cast<const uchar2*>(p));
        a[0] = t.x; a[1] = t.y;
    } else {
        const uchar4 t = __ldg(reinterpret_cast<const uchar4*>(p));
        a[0] = t.x; a[1] = t.y; a[2] = t.z; a[3] = t.w;
    }
}

// apply_box_filter (:1307-1470) of the 11 stage fields and the stage's <rho_f> (:2536-2550).  Bound
// by memory: 11 fields in and 11 out with nothing but sums between, so each block takes one field
// (blockIdx.z) and needs few registers, each thread V cells of a row in 16-byte accesses and
// marches through seg planes, keeping the planes before, at and after the current one.  One field a
// block also gives small grids 11 times the blocks.  V > 1 needs rows that are a multiple of V
// values; other grids take V = 1.  The mixture properties, which compute and need 7 of the 11
// fields, are in the next pass: in one kernel the filter's loads waited for registers that the
// properties held.  256x128x128, ms per step: filter and properties and, apart, strain took
// 1.63 + 0.60 (FP64) and 0.92 + 0.24 (FP32); the filter alone, a cell a thread and 11 fields a block,
// 0.76 and 0.58; in this form 0.59 and 0.36 (176 bytes a cell, 5.0 TB/s; seg = 4: 0.63, 16: 0.60,
// 1: 0.92), with properties and strain together at 1.11 and 0.505.  With V = 1 a thread has few bytes
// in flight, so it loads the plane after the next one ahead: 191x95x97 FP64 0.380 -> 0.336; with
// V > 1 the registers cost more than that gives (256x128x128 0.592 -> 0.607, FP32 0.365 -> 0.379).
template <int V, typename R, typename RI = R, bool BATCH = false>
__global__ void __launch_bounds__(NT)
    k_filter(LES_KERNEL_CONSTS, const uint8_t* __restrict__ attr, F11<RI> in, F11<R> F, double* __restrict__ part,
             Scalars* __restrict__ S, int seg, Batch B) {
    int q = blockIdx.z;
    if constexpr (BATCH) {
        const int m = blockIdx.z / NSTATE;
        q = blockIdx.z - m * NSTATE;
        const MemberTab& e = B.mt[m];
        shift_all(in, e.delta);
        shift_all(F, e.delta);
        attr = e.attr;
        part = e.part;
        S = e.S;
    }
    const RI* __restrict__ x = in.p[0];
    R* __restrict__ y = F.p[0];
#pragma unroll
    for (int s = 1; s < NSTATE; s++)
        if (q == s) { x = in.p[s]; y = F.p[s]; }
    const int nx = C.nx, ny = C.ny, nz = C.nz, nv = nz / V;
    const int tid = threadIdx.x, sI = ny * nz;
    const int pv = blockIdx.x * NT + tid;
    const int i0 = blockIdx.y * seg, i1 = min(i0 + seg, nx);
    constexpr bool AHEAD = V == 1;
    pdl_wait();
    double mass = 0.0;
    if (pv < ny * nv) {
        const int j = pv / nv, k = (pv - j * nv) * V;
        const bool row = j >= 1 && j < ny - 1;
        int id = i0 * sI + j * nz + k;
        RI lo[V], c[V], hi[V], ahead[V];
        ld_vec<RI, V>(x + id, c);
#pragma unroll
        for (int v = 0; v < V; v++) lo[v] = c[v];
        if (i0 > 0) ld_vec<RI, V>(x + id - sI, lo);
        if (AHEAD && i0 + 1 < nx) ld_vec<RI, V>(x + id + sI, hi);
        for (int i = i0; i < i1; i++, id += sI) {
            int a[V];
            ld_attr<V>(attr + id, a);
            if constexpr (AHEAD) {
                if (i + 1 < i1 && i + 2 < nx) ld_vec<RI, V>(x + id + 2 * sI, ahead);
            } else {
                if (i + 1 < nx) ld_vec<RI, V>(x + id + sI, hi);
            }
            R f[V];
            if (row && i >= 1 && i < nx - 1) {
                RI dn[V], up[V];
                ld_vec<RI, V>(x + id - nz, dn);
                ld_vec<RI, V>(x + id + nz, up);
                const RI left = k > 0 ? __ldg(x + id - 1) : RI(0), right = k + V < nz ? __ldg(x + id + V) : RI(0);
#pragma unroll
                for (int v = 0; v < V; v++) {
                    // FP64: (50 x + six neighbours) / 56 as x + (neighbours - 6 x) / 56: fewer roundings at
                    // the size of x, and a uniform field stays exactly what it is.  FP32: the sum
                    // itself, in the reference's order, as the picks of the G equation
                    // hang on its last bits.
                    const RI kl = v > 0 ? c[v > 0 ? v - 1 : 0] : left, kr = v < V - 1 ? c[v < V - 1 ? v + 1 : 0] : right;
                    const bool inner = a[v] == 3 && k + v >= 1 && k + v < nz - 1;
                    if constexpr (std::is_same<R, float>::value) {
                        const R sum = fma(R(FILTER_W), R(c[v]), R(lo[v]) + R(dn[v]) + R(kl));
                        f[v] = inner ? (sum + R(kr) + R(up[v]) + R(hi[v])) * R(1.0 / (FILTER_W + 6.0)) : R(c[v]);
                    } else {
                        const RI nb = lo[v] + dn[v] + kl + kr + up[v] + hi[v];
                        f[v] = R(inner ? fma(fma(RI(-6.0), c[v], nb), RI(1.0 / 56.0), c[v]) : c[v]);
                    }
                }
            } else {
#pragma unroll
                for (int v = 0; v < V; v++) f[v] = R(c[v]);
            }
            st_vec<V>(y + id, f);
            if (q == 5) {
#pragma unroll
                for (int v = 0; v < V; v++)
                    if (a[v] == 1 || a[v] == 2 || a[v] == 3 || a[v] == 5) mass += (((double)f[v] * C.dx) * C.dy) * C.dz;
            }
#pragma unroll
            for (int v = 0; v < V; v++) {
                lo[v] = c[v];
                c[v] = hi[v];
                if (AHEAD) hi[v] = ahead[v];
            }
        }
    }
    if (q != 5) return;
    // partial sums for <rho_f>; in a batched launch, over the member's own blocks
    __shared__ double sh[NT / 32];
    const unsigned nblk = gridDim.x * gridDim.y, bid = blockIdx.y * gridDim.x + blockIdx.x;
    const double bm = block_sum<NT>(mass, sh, tid);
    if (last_block(part, nblk, bid, &bm, 1, &S->counter[0], tid)) {
        double s = 0.0;
        // unrolled so that the partials' loads are in flight together; each thread still adds
        // its entries in ascending order, so the sum is unchanged
#pragma unroll 8
        for (unsigned b = tid; b < nblk; b += NT) s += __ldcg(&part[b]);
        s = block_sum<NT>(s, sh, tid);
        if (tid == 0) {
            S->rho_avg = (C.total_volume > 0) ? (s / C.total_volume) : 1.2;
            S->counter[0] = 0u;
        }
    }
}

// ------------------------------------------------------------------ pass B: properties, strain, nu_t, S_T

// keep: the last RHS evaluation of a step (or one on its own): mu, nu and |S| are written for
// inspection and the probe lines, which no other pass reads, and the nu/alpha maxima that feed the
// next dt are taken (:4401-4408).
template <typename R, bool BATCH = false, int NTB = NT>
__global__ void __launch_bounds__(NTB, lb_blocks(MinBlocks<R>::props, NTB))
    k_props(LES_KERNEL_CONSTS, const uint8_t* __restrict__ attr, F11<R> F, PropBuf<R> P, Scalars* __restrict__ S,
            int keep, Batch B) {
    const auto& K = kc<R>(C);
    __shared__ double tab[EXP_STEPS];
    int bz = blockIdx.z;
    ModelK<R> M;
    if constexpr (BATCH) {
        const int m = blockIdx.z / B.gz;
        bz = blockIdx.z - m * B.gz;
        const MemberTab& e = B.mt[m];
        shift_all(F, e.delta);
        shift_props(P, e.delta);
        attr = e.attr;
        S = e.S;
        M = member_model<R>(e);
    } else {
        M = model_of<R>(C);
    }
    const int nx = C.nx, ny = C.ny, nz = C.nz;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = bz * blockDim.z + threadIdx.z;
    const int tid = (threadIdx.z * blockDim.y + threadIdx.y) * blockDim.x + threadIdx.x;
    if constexpr (std::is_same<R, double>::value) {
        if (tid < EXP_STEPS) tab[tid] = C.exp_tab[tid];
        __syncthreads();
    }
    pdl_wait();
    const bool here = k < nz && j < ny && i < nx;
    const int id = here ? (int)cid(i, j, k, ny, nz) : 0;
    const bool interior = here && i >= 1 && i < nx - 1 && j >= 1 && j < ny - 1 && k >= 1 && k < nz - 1;
    const int a = here ? attr[id] : 0;
    // loaded beside the attribute, not after it: one trip to memory less
    const R T = F.p[3][id], rho = F.p[5][id], G = F.p[4][id];
    R Y[NSP];
#pragma unroll
    for (int s = 0; s < NSP; s++) Y[s] = F.p[6 + s][id];
    if (a == 3) {
        R num = R(0), div = R(0), nut = R(0), Smag = R(0);
        if (interior) {
            const int sI = ny * nz, sJ = nz;
            if constexpr (std::is_same<R, float>::value) {
                f32_strain(K, M, F, id, sI, sJ, G, Smag, nut, div, num);
            } else {
                const R* __restrict__ uf = F.p[0] + id;
                const R* __restrict__ vf = F.p[1] + id;
                const R* __restrict__ wf = F.p[2] + id;
                const R du_dx = (uf[sI] - uf[-sI]) * K.d_2dx.r, dv_dy = (vf[sJ] - vf[-sJ]) * K.d_2dy.r;
                const R dw_dz = (wf[1] - wf[-1]) * K.d_2dz.r, du_dy = (uf[sJ] - uf[-sJ]) * K.d_2dy.r;
                const R du_dz = (uf[1] - uf[-1]) * K.d_2dz.r, dv_dx = (vf[sI] - vf[-sI]) * K.d_2dx.r;
                const R dv_dz = (vf[1] - vf[-1]) * K.d_2dz.r, dw_dx = (wf[sI] - wf[-sI]) * K.d_2dx.r;
                const R dw_dy = (wf[sJ] - wf[-sJ]) * K.d_2dy.r;
                R S11 = du_dx, S22 = dv_dy, S33 = dw_dz;
                R S12 = R(0.5) * (du_dy + dv_dx), S13 = R(0.5) * (du_dz + dw_dx), S23 = R(0.5) * (dv_dz + dw_dy);
                const R off = fma(S23, S23, fma(S13, S13, S12 * S12));
                const R Sij = fma(R(2.0), off, fma(S33, S33, fma(S22, S22, S11 * S11)));
                Smag = qsqrt(R(2.0) * Sij);
                div = du_dx + dv_dy + dw_dz;
                R g = G;
                if (g < R(0.0)) g = R(0.0);
                if (g > R(1.0)) g = R(1.0);
                R cs = fma(M.cs_b - M.cs_u, g, M.cs_u);
                cs = fma(M.cs_boost * R(4.0) * g, R(1.0) - g, cs);
                const R dx = (R)K.dx;
                nut = (cs * dx) * (cs * dx) * Smag;
                num = fma(-div * div, R(1.0 / 3.0), Sij);
            }
        }
        CellProps<R> o;
        auto store_d = [&](const R* D) {
#pragma unroll
            for (int s = 0; s < NSP; s++) P.D[s][id] = D[s];
        };
        bool ordinary;
        if constexpr (std::is_same<R, float>::value) ordinary = f32_cell_props(C, T, Y, rho, store_d, o);
        else ordinary = cell_props_fast(C, tab, T, Y, rho, store_d, o);
        if (!ordinary) {
            CellProps<R> g;
            R Yf[NSP];
#pragma unroll
            for (int s = 0; s < NSP; s++) Yf[s] = Y[s];
            cell_props_any<R>(C, T, Yf, rho, &g);
            store_d(g.D);
            o = g;
        }
        P.aT[id] = o.aT;
        P.nu_t[id] = nut;
        P.mu_eff[id] = interior ? fma(rho, nut, o.mu_mix) : R(0);
        if (keep) {
            P.mu_mix[id] = o.mu_mix;
            P.nu[id] = o.nu;
            P.S_mag[id] = Smag;
            max_into(&S->numax, (double)o.nu);
            max_into(&S->alphamax, (double)o.alpha);
        }
        if (P.dbg_cp) { P.dbg_cp[id] = o.cp; P.dbg_lam[id] = o.lam; P.dbg_alpha[id] = o.alpha; }
        R ST = R(0);
        if constexpr (std::is_same<R, float>::value) {
            if (interior) ST = f32_flame_speed(K, num, div, o.nu);
        } else if (interior) {
            const R dx = (R)K.dx, nul = o.nu;
            // SSR-SGS turbulent flame speed (:1926-1957)
            const R X = (R)K.dx4 * num * frcp(nul * nul);
            R d_eta = R(1.0);
            if (!(X < R(SMALL))) {
                // X^(3/4) = sqrt(X) sqrt(sqrt(X)): two square roots instead of a power
                const R y = qsqrt(X), pX = y * qsqrt(y), arg = R(SSR_B) * pX;
                d_eta = R(SSR_A) * pX * (arg > R(1.0) ? qlog(arg) : R(0.0));
            }
            const R eta = qdiv(dx, d_eta + R(SMALL));
            R te = R(0.0);
            if (K.tau_sl > R(SMALL)) te = dx * fmax(R(0.0), div) * K.d_tau_sl.r;
            // The wrinkling ratio (8 exp(c / (8 eta)) eta / dx)^(2 - D3) is at most 1 where 8 eta >= dx and
            // the exponent is negative (c >= 0); without dilatation the speed is then S_L whatever its
            // value, and the exponential, the logarithm and the power are left out.
            R st = (R)K.s_l;
            if (!(te <= R(0.0) && K.ssr_exp <= R(0.0) && K.ssr_cdF >= R(0.0) && R(8.0) * eta >= dx)) {
                const R z = qdiv((R)K.ssr_cdF, fma(R(8.0), eta, R(SMALL)));
                const R wr = qexp((R)K.ssr_exp * (qlog(R(8.0) * eta * K.d_dx.r) + z));
                st = (R)K.s_l * fmax(R(0.0), wr + te);
            }
            ST = fmax((R)K.s_l, st);
        }
        P.ST[id] = ST;
    } else if (here) {
        P.nu_t[id] = R(0);
        P.ST[id] = interior ? (R)K.s_l : R(0);
        P.mu_eff[id] = R(0);
        if (keep) P.S_mag[id] = R(0);
        if (P.dbg_cp) {
            // property values of non-fluid cells are never read by the step; they are filled
            // only for inspection, with the reference's defaults
            P.mu_mix[id] = R(1.8e-5);
            P.nu[id] = R(1.5e-5);
#pragma unroll
            for (int s = 0; s < NSP; s++) P.D[s][id] = R(0);
            P.aT[id] = R(0);
            P.dbg_cp[id] = R(1000.0); P.dbg_lam[id] = R(0); P.dbg_alpha[id] = R(0);
        }
    }
}

// ------------------------------------------------------------------ pass C: right-hand sides

// TENO5 (:2190-2295) and the WENO5 gradient (:735-827) of one axis, in the differences between
// neighbouring cells.  With f, g the two differences of three consecutive values (a, b, c), the
// reference's smoothness differences are a - 2b + c = g - f and a - 4b + 3c = 3g - f (seen from
// the right end), a - c = -(f + g) (from the middle), 3a - 4b + c = g - 3f (from the left end).
template <typename R>
__device__ __forceinline__ R smooth(R s2, R b) { return fma(R(1.0 / 4.0) * b, b, s2); }   // s2 = 13/12 (g - f)^2

// 6 x (reconstructed value - its cell) from the three candidates q0, q1, q2 (:2212-2236): the
// smooth ones by their linear weights, or the smoothest where none is smooth.
template <typename R>
__device__ __forceinline__ R teno_pick(R is0, R is1, R is2, R q0, R q1, R q2) {
    const R w0 = is0 < R(TENO_CUT) ? R(0.1) : R(0.0), w1 = is1 < R(TENO_CUT) ? R(0.6) : R(0.0),
            w2 = is2 < R(TENO_CUT) ? R(0.3) : R(0.0);
    const R ws = w0 + w1 + w2;
    const R best = (is0 <= is1 && is0 <= is2) ? q0 : ((is1 <= is0 && is1 <= is2) ? q1 : q2);
    const R sum = fma(w2, q2, fma(w1, q1, w0 * q0));
    return ws > R(0.0) ? sum * frcp(ws > R(0.0) ? ws : R(1.0)) : best;
}

// Difference of the two reconstructed face values along the velocity, f1..f5 the differences of
// the six values from three upstream to two downstream: mirrored for a negative velocity the
// reference's two branches are this one expression, and the two faces share three stencils.
template <typename R>
__device__ __forceinline__ R teno_faces(R f1, R f2, R f3, R f4, R f5) {
    const R s1 = f2 - f1, s2 = f3 - f2, s3 = f4 - f3, s4 = f5 - f4;
    const R c = R(13.0 / 12.0);
    const R t1 = c * s1 * s1, t2 = c * s2 * s2, t3 = c * s3 * s3, t4 = c * s4 * s4;
    const R m = teno_pick<R>(smooth(t1, fma(R(3.0), f2, -f1)), smooth(t2, f2 + f3), smooth(t3, fma(R(-3.0), f3, f4)),
                             fma(R(5.0), f2, R(-2.0) * f1), fma(R(2.0), f3, f2), fma(R(4.0), f3, -f4));
    const R p = teno_pick<R>(smooth(t2, fma(R(3.0), f3, -f2)), smooth(t3, f3 + f4), smooth(t4, fma(R(-3.0), f4, f5)),
                             fma(R(5.0), f3, R(-2.0) * f2), fma(R(2.0), f4, f3), fma(R(4.0), f4, -f5));
    return fma(p - m, R(1.0 / 6.0), f3);
}

// The WENO5 gradient (:735-827, on the cells -2..+3 whatever the velocity) times the spacing, e1..e5 the
// differences of its six values.  The weights gamma_k / (eps + IS_k)^2 are brought to one
// denominator: one reciprocal per half instead of three quotients and three shares of their sum.
template <typename R>
__device__ __forceinline__ R weno_half(R i0, R i1, R i2, R g0, R g1, R g2, R q0, R q1, R q2) {
    const R eps = R(1.0e-6);
    const R a0 = eps + i0, a1 = eps + i1, a2 = eps + i2;
    const R e0 = a0 * a0, e1 = a1 * a1, e2 = a2 * a2;
    const R w0 = g0 * (e1 * e2), w1 = g1 * (e0 * e2), w2 = g2 * (e0 * e1);
    return fma(w2, q2, fma(w1, q1, w0 * q0)) * frcp(w0 + w1 + w2);
}
template <typename R>
__device__ __forceinline__ R weno_diff(R e1, R e2, R e3, R e4, R e5) {
    const R s1 = e2 - e1, s2 = e3 - e2, s3 = e4 - e3, s4 = e5 - e4;
    const R c = R(13.0 / 12.0);
    const R t1 = c * s1 * s1, t2 = c * s2 * s2, t3 = c * s3 * s3, t4 = c * s4 * s4;
    const R p = weno_half<R>(smooth(t2, fma(R(3.0), e3, -e2)), smooth(t3, e3 + e4), smooth(t4, fma(R(-3.0), e4, e5)),
                             R(0.3), R(0.6), R(0.1), fma(R(5.0), e3, R(-2.0) * e2), fma(R(2.0), e4, e3),
                             fma(R(4.0), e4, -e5));
    const R m = weno_half<R>(smooth(t1, fma(R(3.0), e2, -e1)), smooth(t2, e2 + e3), smooth(t3, fma(R(-3.0), e3, e4)),
                             R(0.1), R(0.6), R(0.3), fma(R(2.0), e2, e1), fma(R(4.0), e2, -e3),
                             fma(R(2.0), e4, fma(R(-5.0), e3, R(6.0) * e2)));
    return fma(p - m, R(1.0 / 6.0), e2 + e3);
}

// MUSCL-superbee (:2017-2028, :2058-2094).  Half the limited slope of a face,
// 0.5 * superbee(a / b) * b, with a the difference across the face behind and b across the face
// itself, as the reference defines it: b where |b| < SMALL (it sets r = 1e9, :2064), 0 where a
// and b differ in sign, otherwise the middle form of superbee without the quotient:
// superbee(a / b) |b| = min(2 min(|a|, |b|), max(|a|, |b|)).  Exact apart from the reference's
// rounding of (a / b) * b; a NaN in a alone gives b, as superbee(NaN) = 2 does.
__device__ __forceinline__ double half_slope(double a, double b) {
    const bool sm = fabs(a) < fabs(b);
    const double lo = sm ? a : b, hh = 0.5 * (sm ? b : a);
    double x = fabs(lo) >= fabs(hh) ? hh : lo;
    x = (a * b <= 0.0) ? 0.0 : x;
    return fabs(b) < SMALL ? b : x;
}

// One field around a cell, along each axis in the direction of the velocity there: the cell, its
// upstream and downstream neighbours and the cell two upstream.  Mirrored for a negative
// velocity, the reference's two branches are the same expression, so the flux difference needs
// no selects and four values per axis instead of five.
template <typename R>
struct Star {
    R c, up[3], dn[3], uu[3];
};

// What the advection-diffusion of every scalar of a cell shares.
template <typename R>
struct StarCoef {
    R av[3];            // |velocity| / spacing
    R gu[3], gd[3];     // (nu_t + nu_t of the neighbour) / (2 Sc_t) / spacing^2, up- and downstream face
    R lim;              // 1, or 0 in the band where the scheme is first-order upwind (:2043-2052)
};

// relax * (target - phi) - advection + div((g + D) grad phi) (:2037-2159, :2853-2865, :2932-2944):
// the face differences are formed once, and feed the limiter, the advection and the diffusion.
// Differences of neighbours instead of reconstructed face values keep the cancellation exact
// where the reference rounds face values first.  gr scales the shared SGS coefficients (1 for
// the mass fractions, Sc_t / Pr_t for the temperature).
template <typename R, bool UNIT>
__device__ __forceinline__ R star_rhs(const Star<R>& q, const StarCoef<R>& K, R gr, R D, const R (&ih2)[3], R src) {
    R k = src;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const R d1 = q.up[a] - q.uu[a], d2 = q.c - q.up[a], d3 = q.dn[a] - q.c;
        const R t = fma(K.lim, half_slope(d2, d3) - half_slope(d1, d2), d2);
        const R Dh = D * ih2[a];
        const R cu = UNIT ? K.gu[a] + Dh : fma(K.gu[a], gr, Dh);
        const R cd = UNIT ? K.gd[a] + Dh : fma(K.gd[a], gr, Dh);
        k = fma(-K.av[a], t, k);
        k = fma(cd, d3, k);
        k = fma(-cu, d2, k);
    }
    return k;
}

// C1: species (:2837-2904) and temperature (:2912-2962), then their RK4 bookkeeping.
// stage: 0,1,2 -> intermediate stage with coefficient 0.5/0.5/1.0, 3 -> final combine.
// Where the scalar pass reads its stencil fields (filtered T and Y_k, nu_t): global memory,
// or the shared-memory tile of the staged kernel (les_tma.cuh).  Offsets are 32-bit bytes: ten
// registers instead of twenty for the ten positions of a star (FP64 1.42 -> 1.37 ms per 256x128x128
// step).  A fluid cell of the first plane, which a caller's attribute map may hold, would be a negative offset
// away from its neighbour, 4 GiB behind the field in 32 bits: it reads itself (offsets counted from a plane
// ahead of the field instead: FP64 1.168 -> 1.211, FP32 1.128 -> 1.107).  Fields of 4 GiB less a
// plane do not fit 59 times (lesgpu_create refuses them).
template <typename R>
struct GSrc {
    const R* T;
    const R* Y[NSP];
    const R* nut;
    int id, s[3];                       // the cell, the strides
    unsigned c0, up[3], dn[3], uu[3];   // byte offsets of the cell and its neighbours
    __device__ __forceinline__ void orient(const bool (&pos)[3], bool far) {
        c0 = (unsigned)id * (unsigned)sizeof(R);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const unsigned b = (unsigned)s[a] * (unsigned)sizeof(R);
            const unsigned lo = !far && c0 < b ? c0 : c0 - b, hi = c0 + b;
            up[a] = pos[a] ? lo : hi;
            dn[a] = pos[a] ? hi : lo;
            uu[a] = far ? (pos[a] ? lo - b : hi + b) : up[a];    // the band's cells have no second neighbour
        }
    }
    static __device__ __forceinline__ R at(const R* p, unsigned o) {
        return *reinterpret_cast<const R*>(reinterpret_cast<const char*>(p) + o);
    }
    __device__ __forceinline__ void star(const R* p, Star<R>& q) const {
        q.c = at(p, c0);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            q.up[a] = at(p, up[a]);
            q.dn[a] = at(p, dn[a]);
            q.uu[a] = at(p, uu[a]);
        }
    }
    __device__ __forceinline__ void y(int sp, Star<R>& q) const { star(Y[sp], q); }
    __device__ __forceinline__ void t(Star<R>& q) const { star(T, q); }
    __device__ __forceinline__ void nu(R& c, R (&u)[3], R (&d)[3]) const {
        c = at(nut, c0);
#pragma unroll
        for (int a = 0; a < 3; a++) { u[a] = at(nut, up[a]); d[a] = at(nut, dn[a]); }
    }
};

template <typename R>
__device__ __forceinline__ GSrc<R> global_source(const F11<R>& F, const PropBuf<R>& P, int id, int ny, int nz) {
    GSrc<R> src;
    src.id = id;
    src.s[0] = ny * nz;
    src.s[1] = nz;
    src.s[2] = 1;
    src.T = F.p[3];
#pragma unroll
    for (int s = 0; s < NSP; s++) src.Y[s] = F.p[6 + s];
    src.nut = P.nu_t;
    return src;
}

// The RK stages as the scalar pass sees them: the first starts the running sum, the last ends it.
enum { RK_FIRST = 0, RK_MIDDLE = 1, RK_LAST = 2 };

// The dt inputs of the step have been read by now (the first stage's update has used dt), and the
// last stage's property and flow passes take them anew.
__device__ __forceinline__ void reset_maxima(Scalars* Sc) { Sc->umax = Sc->numax = Sc->alphamax = 0.0; }

// One cell of the scalar pass (the body shared by both read paths).
template <int PART, typename R, typename RS, typename Src, typename Hand>
__device__ __forceinline__ void rhs_scalar_cell(const Consts& C, const uint8_t* __restrict__ attr, const F11<R>& F,
                                                const PropBuf<R>& P, const F11<RS>& S0, const F11<R>& St,
                                                const AccBuf<R>& acc, const Hand& hand, const KDbg<R>& kd,
                                                Scalars* __restrict__ Sc, int stage, int i, int j, int k,
                                                Src& src, const R relax) {
    const auto& K = kc<R>(C);
    const int nx = C.nx, ny = C.ny, nz = C.nz;
    const size_t id = cid(i, j, k, ny, nz);
    const int a = attr[id];
    // loaded beside the attribute, not after it: one trip to memory less
    const R vel[3] = {F.p[0][id], F.p[1][id], F.p[2][id]};
    R g = F.p[4][id];

    if (a != 3) {
        // non-fluid cells: the temp state is Phi_n (:4444, :4454); rho_temp is only ever written on
        // outlet/fluid cells (:1893), so it stays 0 on inlet/wall/symmetry cells.  These values
        // are the same for all stages of a step.
        // Cells of the boundary faces get their final values in k_bc; the last stage brings any
        // other cell that is not fluid to what the reference's EOS sweep (:3130-3160) leaves there.
        RS Y0[NSP];
        const RS T0 = S0.p[3][id], r0 = S0.p[5][id];
#pragma unroll
        for (int s = 0; s < NSP; s++) Y0[s] = S0.p[6 + s][id];
        if (PART == RK_FIRST) {
            const RS r = eos_rho_state<R>(C, T0, Y0, r0);
            St.p[3][id] = R(T0);
#pragma unroll
            for (int s = 0; s < NSP; s++) St.p[6 + s][id] = R(Y0[s]);
            if (a == 2) St.p[5][id] = R(r);
        } else if (PART == RK_LAST && off_faces(C, i, j, k)) {
            hand(eos_rho_state<R>(C, T0, Y0, RS(1.2)));
            if ((a == 2 || a == 5) && !beside_face(C, i, j, k) && renormalise<R>(Y0, RS(1e-6))) {
#pragma unroll
                for (int s = 0; s < NSP; s++) S0.p[6 + s][id] = Y0[s];
            }
        }
        if (kd.p[0]) {
#pragma unroll
            for (int q = 0; q < NACC; q++) kd.p[q][id] = R(0);
        }
        return;
    }

    // the right-hand sides and running sums of T, Y0..Y4 in this order, fields 3 and 5..9 of acc
    R kv[1 + NSP];
    const bool band2 = (i < 2 || i >= nx - 2 || j < 2 || j >= ny - 2 || k < 2 || k >= nz - 2);
    if (g < R(0.0)) g = R(0.0);
    if (g > R(1.0)) g = R(1.0);
    const bool pos[3] = {vel[0] >= R(0.0), vel[1] >= R(0.0), vel[2] >= R(0.0)};
    src.orient(pos, !band2);
    // the targets of the nudging
    const R Tt = fma(g, (R)K.t_burnt_span, (R)K.t_in);
    auto target = [&](int s) {
        auto line = [&](R y, R slope) {
            if constexpr (std::is_same<R, float>::value) return fma(slope, g, y);
            else return y + slope * g;
        };
        if (s == C3H8) return (R)K.inletYk[C3H8] * (R(1.0) - g);
        if (s == O2) return fmax(R(0.0), line((R)K.inletYk[O2], -(R)K.cons_o2));
        if (s == CO2) return line((R)K.inletYk[CO2], (R)K.prod_co2);
        if (s == H2O) return line((R)K.inletYk[H2O], (R)K.prod_h2o);
        return (R)K.inletYk[N2];
    };
    if constexpr (std::is_same<R, float>::value) {
        float n0, nu[3], nd[3];
        src.nu(n0, nu, nd);
        Fl sp[3], sm[3], gp[3], gm[3];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            sp[q] = Fl(pos[q] ? nd[q] : nu[q]) + Fl(n0);
            sm[q] = Fl(pos[q] ? nu[q] : nd[q]) + Fl(n0);
            gp[q] = sp[q] * Fl(K.d_prt2.r);
            gm[q] = sm[q] * Fl(K.d_prt2.r);
        }
        Star<float> q;
        src.t(q);
        kv[0] = f32_scalar_rhs<true>(K, q, pos, band2, vel, gp, gm, ld_stream(P.aT + id), relax, Tt, 1.0f);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            gp[a] = sp[a] * Fl(K.d_sct2.r);
            gm[a] = sm[a] * Fl(K.d_sct2.r);
        }
#pragma unroll
        for (int s = 0; s < NSP; s++) {
            src.y(s, q);
            const Fl D = ld_stream(P.D[s] + id);
            if (s == C3H8) kv[1] = f32_scalar_rhs<true>(K, q, pos, band2, vel, gp, gm, D, relax, K.inletYk[s], 1.0f - g);
            else kv[1 + s] = f32_scalar_rhs<false>(K, q, pos, band2, vel, gp, gm, D, relax, target(s), 1.0f);
        }
    } else {
        const R ih2[3] = {K.d_dxx.r, K.d_dyy.r, K.d_dzz.r};
        StarCoef<R> co;
        co.lim = band2 ? R(0.0) : R(1.0);
        co.av[0] = fabs(vel[0]) * K.d_dx.r;
        co.av[1] = fabs(vel[1]) * K.d_dy.r;
        co.av[2] = fabs(vel[2]) * K.d_dz.r;
        {
            R n0, nu[3], nd[3];
            src.nu(n0, nu, nd);
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const R c = K.d_sct2.r * ih2[q];
                co.gu[q] = (nu[q] + n0) * c;
                co.gd[q] = (nd[q] + n0) * c;
            }
        }
        {
            Star<R> q;
            src.t(q);
            kv[0] = star_rhs<R, false>(q, co, K.d_sct2.c * K.d_prt2.r, ld_stream(P.aT + id), ih2, relax * (Tt - q.c));
        }
#pragma unroll
        for (int s = 0; s < NSP; s++) {
            Star<R> q;
            src.y(s, q);
            kv[1 + s] = star_rhs<R, true>(q, co, R(1.0), ld_stream(P.D[s] + id), ih2, relax * (target(s) - q.c));
        }
    }
    // ---- RK4 bookkeeping.  acc holds k1, k1 + 2k2, (k1 + 2k2) + 2k3: exactly the
    // left-to-right partial sums of k1 + 2.0*k2 + 2.0*k3 + k4 (:4520).  All loads come before the
    // first store: a store in between may alias them as far as the compiler knows, and each load
    // after it would wait for that store's operand, one trip to memory after another; for the
    // same reason the part of the step is a template parameter, not a branch.
    RS sn[2 + NSP];                     // T, Y0..Y4, rho
    R ac[1 + NSP];
#pragma unroll
    for (int q = 0; q < 1 + NSP; q++) {
        sn[q] = ld_stream(S0.p[q == 0 ? 3 : 5 + q] + id);
        ac[q] = PART != RK_FIRST ? ld_stream(acc.p[q == 0 ? 3 : 4 + q] + id) : R(0);
    }
    const RS rho_n = ld_stream(S0.p[5] + id);
    const double dt = Sc->dt;
    // The update itself runs in the state's type: in the FP32 form the right-hand sides are
    // FP32 and Phi_n, the stage update and the final combine FP64, so increments far below
    // the state's FP32 ulp are not rounded away step after step.
    const RS cdt = PART == RK_LAST ? (RS)(dt / 6.0) : (RS)((PART == RK_MIDDLE && stage == 2 ? 1.0 : 0.5) * dt);
    RS up[1 + NSP];
#pragma unroll
    for (int q = 0; q < 1 + NSP; q++) {
        const R incr = PART == RK_LAST ? ac[q] + kv[q] : kv[q];
        ac[q] = PART == RK_FIRST ? kv[q] : fma(R(2.0), kv[q], ac[q]);
        up[q] = fma(cdt, (RS)incr, sn[q]);
        up[q] = q == 0 ? fmax(RS(200.0), fmin(RS(3000.0), up[q])) : fmax(RS(0.0), fmin(RS(1.0), up[q]));
    }
    renormalise<R>(up + 1, RS(SMALL));
    RS rho = eos_rho_state<R>(C, up[0], up + 1, PART == RK_LAST ? RS(0.0) : rho_n);
    if (PART == RK_LAST) {
        // the EOS sweep after the boundary conditions (:3130-3160) finds this density again (and 1.2
        // where there is none, which the sign bit tells the flow pass, of zero and NaN too) and
        // renormalises once more
        if (rho == RS(0.0)) rho = -fabs(rho_n);
        if (!band2) renormalise<R>(up + 1, RS(1e-6));   // k_bc: beside a face, after the copies
    }
    if (kd.p[0]) {
#pragma unroll
        for (int q = 0; q < 1 + NSP; q++) kd.p[q == 0 ? 3 : 4 + q][id] = kv[q];
    }
    hand(rho);
    if (PART != RK_LAST) St.p[5][id] = R(rho);
#pragma unroll
    for (int q = 0; q < 1 + NSP; q++) {
        if (PART != RK_LAST) {
            st_stream(acc.p[q == 0 ? 3 : 4 + q] + id, ac[q]);
            St.p[q == 0 ? 3 : 5 + q][id] = R(up[q]);
        } else {
            S0.p[q == 0 ? 3 : 5 + q][id] = up[q];
        }
    }
}

// Has the L1 cache fetch the value at p: an asynchronous copy into shared memory that nobody reads,
// so that no register waits for it.
__device__ __forceinline__ void touch_line(double* scratch, const double* p) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(scratch)), "l"(p));
}

// The FP64 form waits for memory: 10 values of a star fill 20 of the 64 registers, so its 6 stars
// and diffusivities come one trip to memory after another (long scoreboard 10.6 of 15 stall
// cycles an issue, DRAM 39 %).  It therefore first has the cell's own values of them fetched
// into L1, where the threads around it find their neighbours.  Scalar pass per step, ms: 128x64x64
// 0.213 -> 0.201, 191x95x97 0.629 -> 0.595, 256x128x128 1.355 -> 1.186; with the stars alone 1.270,
// the diffusivities alone 1.300, Phi_n and the running sum as well 1.245, prefetch.global.L1 of the
// stars 1.30.  The FP32 form, whose stars take half the registers, gained nothing (0.818 -> 0.828).
template <int PART, typename R, typename RS = R, bool BATCH = false, int NTB = NT>
__global__ void __launch_bounds__(NTB, lb_blocks(MinBlocks<R>::scalar, NTB))
    k_rhs_scalar(LES_KERNEL_CONSTS, const uint8_t* __restrict__ attr, F11<R> F, PropBuf<R> P, F11<RS> S0, F11<R> St,
                 AccBuf<R> acc, RS* __restrict__ rn, KDbg<R> kd, Scalars* __restrict__ Sc, int stage, Batch B) {
    int bz = blockIdx.z;
    R relax;
    if constexpr (BATCH) {
        const int m = blockIdx.z / B.gz;
        bz = blockIdx.z - m * B.gz;
        const MemberTab& e = B.mt[m];
        shift_all(F, e.delta);
        shift_props(P, e.delta);
        shift_all(S0, e.delta);
        shift_all(St, e.delta);
        shift_all(acc, e.delta);
        rn = shifted(rn, e.delta);
#pragma unroll
        for (int q = 0; q < NACC; q++) kd.p[q] = nullptr;
        attr = e.attr;
        Sc = e.S;
        relax = member_model<R>(e).relax;
    } else {
        relax = (R)kc<R>(C).relax;
    }
    const int ny = C.ny, nz = C.nz;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = bz * blockDim.z + threadIdx.z;
    pdl_wait();
    if (k >= nz || j >= ny || i >= C.nx) return;
    const size_t id = cid(i, j, k, ny, nz);
    if (PART == RK_MIDDLE && id == 0) reset_maxima(Sc);
    constexpr bool TOUCH = std::is_same<R, double>::value;
    if constexpr (TOUCH) {
        __shared__ double scratch[NTB];
        double* mine = scratch + (threadIdx.z * blockDim.y + threadIdx.y) * blockDim.x + threadIdx.x;
        touch_line(mine, F.p[3] + id);
#pragma unroll
        for (int s = 0; s < NSP; s++) touch_line(mine, F.p[6 + s] + id);
        touch_line(mine, P.aT + id);
#pragma unroll
        for (int s = 0; s < NSP; s++) touch_line(mine, P.D[s] + id);
    }
    GSrc<R> src = global_source<R>(F, P, (int)id, ny, nz);
    auto hand = [&](RS rho) { st_stream(rn + id, rho); };
    rhs_scalar_cell<PART, R, RS>(C, attr, F, P, S0, St, acc, hand, kd, Sc, stage, i, j, k, src, relax);
    if constexpr (TOUCH) asm volatile("cp.async.wait_all;" ::: "memory");   // no copy outlives its block
}

// C2: momentum (:2552-2697) with calculate_convection_conservative (:683-727) and the G
// equation (:2706-2825), then the RK4 bookkeeping of u, v, w and G with the density the scalar
// pass left in rn.  Measured at 256x128x128, both passes together: handing the density over
// (8 bytes a cell) instead of four right-hand sides, with this pass updating what it computes,
// moves 48 bytes a cell less and takes the loads of half the update out of the scalar pass,
// which waits for memory, into this one, which computes.
// In FP64 everything is in differences across the six faces: a conservative flux m p with the face
// value p = p0 + d/2 (first-order upwind next to the boundary: p0 or p0 + d by the sign of m),
// so convection and diffusion of all three components are two coefficients a face.
// The right-hand sides of rho u, rho v, rho w and G of one fluid cell.
template <typename R>
__device__ __forceinline__ void flow_rhs(const Consts& C, const ModelK<R>& M, const F11<R>& F, const PropBuf<R>& P,
                                         const Scalars* __restrict__ Sc, int i, int j, int k, int id,
                                         const FlowCell<R>& c, R (&kv)[4]) {
    const auto& K = kc<R>(C);
    const int nx = C.nx, ny = C.ny, nz = C.nz;
    const R (&p0)[3] = c.p0;
    const R r0 = c.r0, G0 = c.G0, n0 = c.n0, mu = c.mu;
    const int st[3] = {ny * nz, nz, 1};
    const R ih[3] = {K.d_dx.r, K.d_dy.r, K.d_dz.r}, ih2[3] = {K.d_dxx.r, K.d_dyy.r, K.d_dzz.r};
    const bool band2 = (i < 2 || i >= nx - 2 || j < 2 || j >= ny - 2 || k < 2 || k >= nz - 2);
    const bool band3 = (i < 3 || i >= nx - 3 || j < 3 || j >= ny - 3 || k < 3 || k >= nz - 3);
    R km[3];
    {
        R out = R(0);
#pragma unroll
        for (int q = 0; q < 3; q++) km[q] = R(0);
#pragma unroll
        for (int x = 0; x < 3; x++) {
            const R* __restrict__ rho = F.p[5];
            const R* __restrict__ va = F.p[x];
            const R mp = (R(0.5) * (rho[id + st[x]] + r0)) * (R(0.5) * (va[id + st[x]] + p0[x]));
            const R mm = (R(0.5) * (rho[id - st[x]] + r0)) * (R(0.5) * (va[id - st[x]] + p0[x]));
            const R up = band2 ? (mp > R(0) ? R(0) : mp) : R(0.5) * mp;
            const R um = band2 ? (mm > R(0) ? mm : R(0)) : R(0.5) * mm;
            const R v = mu * ih2[x];
            const R cp = fma(-ih[x], up, v), cm = fma(ih[x], um, v);
            out = fma(ih[x], mp - mm, out);
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const R* __restrict__ ph = F.p[q];
                km[q] = fma(cp, ph[id + st[x]] - p0[q], km[q]);
                km[q] = fma(-cm, p0[q] - ph[id - st[x]], km[q]);
            }
        }
#pragma unroll
        for (int q = 0; q < 3; q++) km[q] = fma(-out, p0[q], km[q]);
    }
    R kG, grad[3], lap = R(0);
    {
        const R* __restrict__ G = F.p[4];
        R adv = R(0), sgs = R(0);
        R e3[3];
#pragma unroll
        for (int x = 0; x < 3; x++) {
            const bool pos = p0[x] >= R(0.0);
            const int o = pos ? -st[x] : st[x];
            const R U = G[id + o], Dn = G[id - o];
            const R f3 = G0 - U, f4 = Dn - G0;
            R d = f3;                                   // first-order upwind (:642-651)
            if (!band3) {
                const R UU = G[id + 2 * o], U3 = G[id + 3 * o], DD = G[id - 2 * o];
                d = teno_faces<R>(UU - U3, U - UU, f3, f4, DD - Dn);
            } else if (!band2) {
                // central faces (:652-677): the zero UW2 coefficient makes both upwind branches identical
                d = R(0.5) * (f3 + f4);
            }
            adv = fma(fabs(p0[x]) * ih[x], d, adv);
            const R gu = (P.nu_t[id + o] + n0) * K.d_sct2.r, gd = (P.nu_t[id - o] + n0) * K.d_sct2.r;
            sgs = fma(ih2[x], fma(gd, f4, -gu * f3), sgs);
            lap = fma(ih2[x], f4 - f3, lap);
            e3[x] = pos ? f3 + f4 : -(f3 + f4);
            grad[x] = R(0.5) * ih[x] * e3[x];
        }
        kG = sgs - adv;
    }
    R art = R(0), fo[3] = {R(0), R(0), R(0)};
    if (C.flame_accel && G0 > R(0.01) && G0 < R(0.99)) {
        const R df = G0 - M.accel_center;
        const R window = qexp(-(df * df) * M.d_w2.r);
        const R zp = (R)k * (R)K.dz;
        const R ramp = zp < R(RAMP_DIST) ? zp * K.d_ramp.r : R(1.0);
        // tip_mask is the literal 1.0 in the momentum source (:2638)
        const R cf = M.accel_strength * r0 * window * ramp;
        fo[0] = cf * R(0.05) * fmax(grad[0], R(0.0));
        fo[1] = cf * fmax(grad[1], R(0.0));
        fo[2] = cf * (zp - (R)K.inlet_center_z > R(0.0) ? fmax(grad[2], R(0.0)) : fmin(grad[2], R(0.0)));
        // tip_mask = 1 - exp(-r^2 / 0^2) is exactly 1 for every fluid cell (j >= 1)
        // because TIP_PROTECTION_RADIUS is 0.0 (:234, :2806-2807).
        if (G0 > R(0.1)) art = R(5.0) * (n0 + R(1.0e-5)) * window * lap;
    }
    const R lim = R(FORCE_LIMIT);
#pragma unroll
    for (int q = 0; q < 3; q++) {
        R f = fo[q];
        if (f > lim) f = lim;
        if (f < -lim) f = -lim;
        km[q] += f;
    }
    km[0] = fma(r0 - (R)Sc->rho_avg, R(G_GRAVITY), km[0]);
    if (Sc->t_loop >= C.weno_step && !band3) {
        const R* __restrict__ G = F.p[4];
#pragma unroll
        for (int x = 0; x < 3; x++) {
            const R q0 = G[id - 2 * st[x]], q1 = G[id - st[x]], q3 = G[id + st[x]], q4 = G[id + 2 * st[x]],
                    q5 = G[id + 3 * st[x]];
            grad[x] = ih[x] * weno_diff<R>(q1 - q0, G0 - q1, q3 - G0, q4 - q3, q5 - q4);
        }
    }
    const R gmag = qsqrt(fma(grad[2], grad[2], fma(grad[1], grad[1], grad[0] * grad[0])));
    if (P.grad_g) P.grad_g[id] = gmag;   // grad_G_magnitude_for_debug (:2783)
    kG = fma(P.ST[id], gmag, kG) + art;
    kv[0] = km[0]; kv[1] = km[1]; kv[2] = km[2]; kv[3] = kG;
}

// A cell that is not fluid, as in the scalar pass: its stage state is Phi_n, and the last stage
// leaves cells off the faces as the EOS sweep does.
template <int PART, typename R, typename RS>
__device__ __forceinline__ void flow_other(const Consts& C, int a, const F11<RS>& S0, const F11<R>& St,
                                           Scalars* __restrict__ Sc, int i, int j, int k, int id, const RS* left) {
    if (PART == RK_FIRST) {
#pragma unroll
        for (int q = 0; q < 5; q++)
            if (q != 3) St.p[q][id] = R(S0.p[q][id]);
    } else if (PART == RK_LAST && off_faces(C, i, j, k)) {
        S0.p[5][id] = *left;
        const RS u = S0.p[0][id], v = S0.p[1][id], w = S0.p[2][id];
        if (a == 1) max_into(&Sc->umax, sqrt(u * u + v * v + w * w));
    }
}

// The RK4 bookkeeping of a fluid cell (see rhs_scalar_cell) with the density that the scalar pass
// left; every load ahead of the first store.
template <int PART, typename R, typename RS>
__device__ __forceinline__ void flow_update(const F11<RS>& S0, const F11<R>& St, const AccBuf<R>& acc, const KDbg<R>& kd,
                                            Scalars* __restrict__ Sc, int stage, int id, const R (&kv)[4], RS left) {
    constexpr int qa[4] = {0, 1, 2, 4};
    RS sn[4];
    R ac[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        sn[q] = ld_stream(S0.p[qa[q]] + id);
        ac[q] = PART != RK_FIRST ? ld_stream(acc.p[qa[q]] + id) : R(0);
    }
    const RS rho_n = ld_stream(S0.p[5] + id);
    const RS rho = PART == RK_LAST ? fabs(left) : left;
    const double dt = Sc->dt;
    const RS cdt = PART == RK_LAST ? (RS)(dt / 6.0) : (RS)((PART == RK_MIDDLE && stage == 2 ? 1.0 : 0.5) * dt);
    const RS irho = srecip<R>(rho);
    RS out[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const R incr = PART == RK_LAST ? ac[q] + kv[q] : kv[q];
        ac[q] = PART == RK_FIRST ? kv[q] : fma(R(2.0), kv[q], ac[q]);
        if (q < 3) {
            // rhou = rho*u after the BC (:3146); the FP32 form has always rounded the other product
            const RS m = std::is_same<R, float>::value ? fma(rho_n, sn[q], __dmul_rn(cdt, (RS)incr))
                                                       : fma(cdt, (RS)incr, rho_n * sn[q]);
            out[q] = rho > RS(SMALL) ? cquot(m, rho, irho) : RS(0);
        } else {
            out[q] = fmax(RS(0.0), fmin(RS(1.0), fma(cdt, (RS)incr, sn[q])));
        }
    }
    if (kd.p[0]) {
#pragma unroll
        for (int q = 0; q < 4; q++) kd.p[qa[q]][id] = kv[q];
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        if (PART != RK_LAST) {
            st_stream(acc.p[qa[q]] + id, ac[q]);
            St.p[qa[q]][id] = R(out[q]);
        } else {
            S0.p[qa[q]][id] = out[q];
        }
    }
    if (PART == RK_LAST) {
        S0.p[5][id] = signbit(left) ? RS(1.2) : left;
        // |u| of the next dt (:1472-1485)
        max_into(&Sc->umax, sqrt(out[0] * out[0] + out[1] * out[1] + out[2] * out[2]));
    }
}

template <int PART, typename R, typename RS = R, bool BATCH = false, int NTB = NT>
__global__ void __launch_bounds__(NTB, lb_blocks(MinBlocks<R>::flow, NTB))
    k_rhs_flow(LES_KERNEL_CONSTS, const uint8_t* __restrict__ attr, F11<R> F, PropBuf<R> P, F11<RS> S0, F11<R> St,
               AccBuf<R> acc, RS* __restrict__ rn, KDbg<R> kd, Scalars* __restrict__ Sc, int stage, Batch B) {
    const auto& K = kc<R>(C);
    int bz = blockIdx.z;
    ModelK<R> M;
    if constexpr (BATCH) {
        const int m = blockIdx.z / B.gz;
        bz = blockIdx.z - m * B.gz;
        const MemberTab& e = B.mt[m];
        shift_all(F, e.delta);
        shift_props(P, e.delta);
        shift_all(S0, e.delta);
        shift_all(St, e.delta);
        shift_all(acc, e.delta);
        rn = shifted(rn, e.delta);
#pragma unroll
        for (int q = 0; q < NACC; q++) kd.p[q] = nullptr;
        attr = e.attr;
        Sc = e.S;
        M = member_model<R>(e);
    } else {
        M = model_of<R>(C);
    }
    const int nx = C.nx, ny = C.ny, nz = C.nz;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = bz * blockDim.z + threadIdx.z;
    pdl_wait();
    if (k >= nz || j >= ny || i >= nx) return;
    const int id = (int)cid(i, j, k, ny, nz);
    const int a = attr[id];
    // loaded beside the attribute, not after it: one trip to memory less
    FlowCell<R> c;
    c.load(F, P, id);
    if (a != 3) {
        flow_other<PART, R, RS>(C, a, S0, St, Sc, i, j, k, id, rn + id);
        return;
    }
    R kv[4];
    if constexpr (std::is_same<R, float>::value) f32_flow_rhs(C, M, F, P, Sc, i, j, k, id, c, kv);
    else flow_rhs<R>(C, M, F, P, Sc, i, j, k, id, c, kv);
    flow_update<PART, R, RS>(S0, St, acc, kd, Sc, stage, id, kv, ld_stream(rn + id));
}

// Both passes in one launch, for grids that do not fill the GPU several times over: the first half
// of a block's threads takes the scalar pass of its cells, the second half the flow pass, which
// needs the other's density only for its update; it is handed over through shared memory at a
// named barrier at which the scalar half arrives without waiting (2 blocks an SM; 1 and 3 were
// slower).  When it is used: both_passes, les_launch.cuh.
template <int PART, typename R, typename RS = R>
__global__ void __launch_bounds__(2 * NT, 2)
    k_rhs_both(LES_KERNEL_CONSTS, const uint8_t* __restrict__ attr, F11<R> F, PropBuf<R> P, F11<RS> S0, F11<R> St,
               AccBuf<R> acc, KDbg<R> kd, Scalars* __restrict__ Sc, int stage, int3 tile) {
    __shared__ RS rn[NT];
    const int t = threadIdx.x & (NT - 1);
    const int tk = t % tile.x, tj = (t / tile.x) % tile.y, ti = t / (tile.x * tile.y);
    const int nx = C.nx, ny = C.ny, nz = C.nz;
    const int k = blockIdx.x * tile.x + tk, j = blockIdx.y * tile.y + tj, i = blockIdx.z * tile.z + ti;
    const bool here = k < nz && j < ny && i < nx;
    const int id = here ? (int)cid(i, j, k, ny, nz) : 0;
    pdl_wait();
    if (threadIdx.x < NT) {
        if (here) {
            if (PART == RK_MIDDLE && id == 0) reset_maxima(Sc);
            GSrc<R> src = global_source<R>(F, P, id, ny, nz);
            auto hand = [&](RS rho) { rn[t] = rho; };
            rhs_scalar_cell<PART, R, RS>(C, attr, F, P, S0, St, acc, hand, kd, Sc, stage, i, j, k, src, (R)kc<R>(C).relax);
        }
        __syncwarp();
        asm volatile("barrier.cta.arrive 1, 512;" ::: "memory");
    } else {
        const int a = here ? attr[id] : 0;
        FlowCell<R> c;
        c.load(F, P, id);
        R kv[4];
        if (a == 3) {
            if constexpr (std::is_same<R, float>::value) f32_flow_rhs(C, model_of<R>(C), F, P, Sc, i, j, k, id, c, kv);
            else flow_rhs<R>(C, model_of<R>(C), F, P, Sc, i, j, k, id, c, kv);
        }
        __syncwarp();
        asm volatile("barrier.cta.sync 1, 512;" ::: "memory");
        if (a == 3) flow_update<PART, R, RS>(S0, St, acc, kd, Sc, stage, id, kv, rn[t]);
        else if (here) flow_other<PART, R, RS>(C, a, S0, St, Sc, i, j, k, id, &rn[t]);
    }
}

// ------------------------------------------------------------------ boundary conditions
// apply_boundary_conditions (:2967-3161): the i-faces (with the SEM + white-noise inflow), then for
// every interior i the j-faces, then the k-faces, then the equation of state and mass-fraction
// renormalisation.  Only the cells of the six faces and, in their mass fractions, the cells next to
// them change: the last stage's scalar and flow passes leave every other cell as the reference's EOS
// sweep over the grid does, and take the maximum of |u| over fluid cells, so no pass over the whole
// grid is needed here.  The cells next to a face are renormalised for the second time here, as the
// copies take their mass fractions before the sweep.

template <typename R>
__device__ __forceinline__ void copy_cell(F11<R>& S, size_t dst, size_t src) {
    R v[NSTATE];
#pragma unroll
    for (int q = 0; q < NSTATE; q++)
        if (q != 5) v[q] = S.p[q][src];
#pragma unroll
    for (int q = 0; q < NSTATE; q++)
        if (q != 5) S.p[q][dst] = v[q];
}
template <typename R>
__device__ __forceinline__ void ambient_cell(const Consts& C, F11<R>& S, size_t dst) {
    const auto& K = kc<R>(C);
    S.p[0][dst] = R(0); S.p[1][dst] = R(0); S.p[2][dst] = R(0);
    S.p[3][dst] = (R)K.t_amb; S.p[4][dst] = R(0);
#pragma unroll
    for (int s = 0; s < NSP; s++) S.p[6 + s][dst] = (R)K.ambientYk[s];
}

// The cell (0, j, k): inflow, open face or rim; the cell (nx-1, j, k): outlet.
template <typename R>
__device__ __forceinline__ void bc_first_plane(const Consts& C, const uint8_t* __restrict__ attr, F11<R>& S,
                                               const double* __restrict__ plane, const double* __restrict__ noise,
                                               const int* __restrict__ inlet_pos, int j, int k) {
    const auto& K = kc<R>(C);
    const int ny = C.ny, nz = C.nz;
    const size_t i0 = cid(0, j, k, ny, nz), i1 = cid(1, j, k, ny, nz);
    const int a0 = attr[i0];
    if (a0 == 1) {
        const size_t p = (size_t)j * nz + k;
        const size_t npl = (size_t)ny * nz;
        const int q = inlet_pos[p];
        const R amp = (R)K.noise_amp;
        R r1 = (R)noise[3 * q + 0], r2 = (R)noise[3 * q + 1], r3 = (R)noise[3 * q + 2];
        S.p[0][i0] = fmax(R(0.0), (R)K.u_in + (R)plane[p] + amp * r1);
        S.p[1][i0] = (R)plane[npl + p] + amp * r2;
        S.p[2][i0] = (R)plane[2 * npl + p] + amp * r3;
        S.p[3][i0] = (R)K.t_in;
        S.p[4][i0] = R(0);
#pragma unroll
        for (int s = 0; s < NSP; s++) S.p[6 + s][i0] = (R)K.inletYk[s];
    } else if (a0 == 4) {
        if (S.p[0][i1] < R(0)) ambient_cell<R>(C, S, i0);
        else copy_cell<R>(S, i0, i1);
    } else if (a0 == 6) {
        copy_cell<R>(S, i0, i1);
        S.p[0][i0] = R(0); S.p[1][i0] = R(0); S.p[2][i0] = R(0);
    }
}
template <typename R>
__device__ __forceinline__ void bc_last_plane(const Consts& C, const uint8_t* __restrict__ attr, F11<R>& S, int j, int k) {
    const size_t in = cid(C.nx - 1, j, k, C.ny, C.nz), im = cid(C.nx - 2, j, k, C.ny, C.nz);
    if (attr[in] == 2) copy_cell<R>(S, in, im);
}

// EOS + renormalisation (:3130-3160) of one cell, and |u| of an inlet or fluid cell for the next
// dt (:1472-1485).
template <typename R, typename Form>
__device__ __forceinline__ void bc_eos_cell(const Consts& C, const uint8_t* __restrict__ attr, F11<R>& S, size_t id,
                                            Scalars* __restrict__ Sc) {
    const int a = attr[id];
    R Y[NSP];
#pragma unroll
    for (int s = 0; s < NSP; s++) Y[s] = S.p[6 + s][id];
    const R T = S.p[3][id], u = S.p[0][id], v = S.p[1][id], w = S.p[2][id];
    S.p[5][id] = eos_rho_state<Form>(C, T, Y, R(1.2));
    if ((a == 3 || a == 2 || a == 5) && renormalise<Form>(Y, R(1e-6))) {
#pragma unroll
        for (int s = 0; s < NSP; s++) S.p[6 + s][id] = Y[s];
    }
    if (a == 1 || a == 3) max_into(&Sc->umax, sqrt(u * u + v * v + w * w));
}

// The second renormalisation (:3150-3159) of a cell next to a face.
template <typename R, typename Form>
__device__ __forceinline__ void bc_renormalise(const uint8_t* __restrict__ attr, F11<R>& S, size_t id) {
    const int a = attr[id];
    R Y[NSP];
#pragma unroll
    for (int s = 0; s < NSP; s++) Y[s] = S.p[6 + s][id];
    if ((a == 3 || a == 2 || a == 5) && renormalise<Form>(Y, R(1e-6))) {
#pragma unroll
        for (int s = 0; s < NSP; s++) S.p[6 + s][id] = Y[s];
    }
}

// The q-th of the 2 (ny + nz) - 4 cells around a plane.
__device__ __forceinline__ void ring_cell(int q, int ny, int nz, int& j, int& k) {
    if (q < 2 * nz) {
        j = q < nz ? 0 : ny - 1;
        k = q < nz ? q : q - nz;
    } else {
        q -= 2 * nz;
        j = 1 + (q >> 1);
        k = (q & 1) ? nz - 1 : 0;
    }
}

// One launch for all of it.  Block b < nx - 2 takes the faces around plane i = b + 1 in the
// reference's order, its own barriers between the steps; the blocks of the second and the last
// but one plane also take, first, the two outermost rings of planes 0 and nx - 1, which copy cells
// that the j- and k-faces then overwrite or copy too.  The remaining blocks take the other cells of planes
// 0 and nx - 1, each the only reader of the cell it copies.  A block writes to a cell next to a
// face only after the last copy of it, which is always its own.
template <typename R, typename Form = R>
__global__ void __launch_bounds__(NT) k_bc(LES_KERNEL_CONSTS, const uint8_t* __restrict__ attr, F11<R> S,
                                           const double* __restrict__ plane, const double* __restrict__ noise,
                                           const int* __restrict__ inlet_pos, Scalars* __restrict__ Sc) {
    const int nx = C.nx, ny = C.ny, nz = C.nz, tid = threadIdx.x;
    const int ring = 2 * (ny + nz) - 4, rings = 2 * ring - 8;
    int j, k;
    pdl_wait();
    if ((int)blockIdx.x >= nx - 2) {
        const int q = ((int)blockIdx.x - (nx - 2)) * NT + tid;
        if (q >= (ny - 2) * (nz - 2)) return;
        j = 1 + q / (nz - 2);
        k = 1 + q % (nz - 2);
        if (j == 1 || j == ny - 2 || k == 1 || k == nz - 2) return;
        bc_first_plane<R>(C, attr, S, plane, noise, inlet_pos, j, k);
        bc_last_plane<R>(C, attr, S, j, k);
        bc_eos_cell<R, Form>(C, attr, S, cid(0, j, k, ny, nz), Sc);
        bc_eos_cell<R, Form>(C, attr, S, cid(nx - 1, j, k, ny, nz), Sc);
        bc_renormalise<R, Form>(attr, S, cid(1, j, k, ny, nz));
        bc_renormalise<R, Form>(attr, S, cid(nx - 2, j, k, ny, nz));
        return;
    }
    const int i = (int)blockIdx.x + 1;
    auto cell = [&](int q) {                        // of the outermost ring, then of the one inside it
        if (q < ring) {
            ring_cell(q, ny, nz, j, k);
        } else {
            ring_cell(q - ring, ny - 2, nz - 2, j, k);
            j++;
            k++;
        }
    };
    if (i == 1 || i == nx - 2) {
        for (int q = tid; q < rings; q += NT) {
            cell(q);
            if (i == 1) bc_first_plane<R>(C, attr, S, plane, noise, inlet_pos, j, k);
            else bc_last_plane<R>(C, attr, S, j, k);
        }
        __syncthreads();
    }
    for (k = tid; k < nz; k += NT) {
        const size_t b = cid(i, 0, k, ny, nz), n1 = cid(i, 1, k, ny, nz);
        if (attr[b] == 5) {
            copy_cell<R>(S, b, n1);
            S.p[1][b] = R(0.0);
        }
        const size_t t = cid(i, ny - 1, k, ny, nz), tm = cid(i, ny - 2, k, ny, nz);
        if (attr[t] == 4) {
            if (S.p[1][tm] < R(0)) ambient_cell<R>(C, S, t);
            else copy_cell<R>(S, t, tm);
        }
    }
    __syncthreads();
    for (j = tid; j < ny; j += NT) {
        const size_t b = cid(i, j, 0, ny, nz), n1 = cid(i, j, 1, ny, nz);
        if (attr[b] == 4) {
            if (S.p[2][n1] > R(0)) ambient_cell<R>(C, S, b);
            else copy_cell<R>(S, b, n1);
        }
        const size_t t = cid(i, j, nz - 1, ny, nz), tm = cid(i, j, nz - 2, ny, nz);
        if (attr[t] == 4) {
            if (S.p[2][tm] < R(0)) ambient_cell<R>(C, S, t);
            else copy_cell<R>(S, t, tm);
        }
    }
    __syncthreads();
    for (int q = tid; q < rings; q += NT) {
        cell(q);
        if (q < ring) bc_eos_cell<R, Form>(C, attr, S, cid(i, j, k, ny, nz), Sc);
        else bc_renormalise<R, Form>(attr, S, cid(i, j, k, ny, nz));
        if (i == 1) bc_eos_cell<R, Form>(C, attr, S, cid(0, j, k, ny, nz), Sc);
        if (i == nx - 2) bc_eos_cell<R, Form>(C, attr, S, cid(nx - 1, j, k, ny, nz), Sc);
    }
}

// Max velocity over inlet/fluid cells without touching the state (after an upload).
template <typename R, typename Form = R>
__global__ void __launch_bounds__(NT) k_umax(LES_KERNEL_CONSTS, const uint8_t* __restrict__ attr, F11<R> S,
                                             double* __restrict__ part, Scalars* __restrict__ Sc) {
    __shared__ double sh[NT / 32];
    __shared__ bool last;
    const int ny = C.ny, nz = C.nz;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z * blockDim.z + threadIdx.z;
    const int tid = (threadIdx.z * blockDim.y + threadIdx.y) * blockDim.x + threadIdx.x;
    double vmax = 0.0;
    if (k < nz && j < ny && i < C.nx) {
        const size_t id = cid(i, j, k, ny, nz);
        const int a = attr[id];
        if (a == 1 || a == 3) {
            R u = S.p[0][id], v = S.p[1][id], w = S.p[2][id];
            vmax = (double)sqrt(u * u + v * v + w * w);
        }
    }
    const unsigned nblk = gridDim.x * gridDim.y * gridDim.z;
    const unsigned bid = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    double bm = block_max<NT>(vmax, sh, tid);
    if (tid == 0) {
        part[bid] = bm;
        __threadfence();
        unsigned t = atomicAdd(&Sc->counter[2], 1u);
        last = (t == nblk - 1);
    }
    __syncthreads();
    if (last) {
        __threadfence();
        double m = 0.0;
#pragma unroll 8
        for (unsigned q = tid; q < nblk; q += NT) m = fmax(m, __ldcg(&part[q]));
        m = block_max<NT>(m, sh, tid);
        if (tid == 0) {
            Sc->umax = m;
            Sc->counter[2] = 0u;
        }
    }
}

// ------------------------------------------------------------------ diagnostics

template <typename R, typename Form = R>
__global__ void __launch_bounds__(NT) k_monitor(LES_KERNEL_CONSTS, F11<R> S, double* __restrict__ part,
                                                Scalars* __restrict__ Sc, size_t n) {
    // write_monitor_log (:3884-3897)
    __shared__ double sh[NT / 32];
    __shared__ bool last;
    const int tid = threadIdx.x;
    double mass = 0.0, tmin = 1.0e9, tmax = -1.0e9, gmin = 1.0e9, gmax = -1.0e9, ymin = 1.0e9;
    for (size_t id = (size_t)blockIdx.x * NT + tid; id < n; id += (size_t)gridDim.x * NT) {
        double r = (double)S.p[5][id], T = (double)S.p[3][id], G = (double)S.p[4][id], Y = (double)S.p[6][id];
        mass += ((r * C.dx) * C.dy) * C.dz;
        tmin = fmin(tmin, T); tmax = fmax(tmax, T);
        gmin = fmin(gmin, G); gmax = fmax(gmax, G);
        ymin = fmin(ymin, Y);
    }
    const unsigned nblk = gridDim.x;
    double v[6];
    v[0] = block_sum<NT>(mass, sh, tid);
    v[1] = block_min<NT>(tmin, sh, tid);
    v[2] = block_max<NT>(tmax, sh, tid);
    v[3] = block_min<NT>(gmin, sh, tid);
    v[4] = block_max<NT>(gmax, sh, tid);
    v[5] = block_min<NT>(ymin, sh, tid);
    if (tid == 0) {
        for (int q = 0; q < 6; q++) part[q * nblk + blockIdx.x] = v[q];
        __threadfence();
        unsigned t = atomicAdd(&Sc->counter[3], 1u);
        last = (t == nblk - 1);
    }
    __syncthreads();
    if (last) {
        __threadfence();
        double acc[6] = {0.0, 1.0e9, -1.0e9, 1.0e9, -1.0e9, 1.0e9};
#pragma unroll 4
        for (unsigned q = tid; q < nblk; q += NT) {
            acc[0] += __ldcg(&part[q]);
            acc[1] = fmin(acc[1], __ldcg(&part[nblk + q]));
            acc[2] = fmax(acc[2], __ldcg(&part[2 * nblk + q]));
            acc[3] = fmin(acc[3], __ldcg(&part[3 * nblk + q]));
            acc[4] = fmax(acc[4], __ldcg(&part[4 * nblk + q]));
            acc[5] = fmin(acc[5], __ldcg(&part[5 * nblk + q]));
        }
        acc[0] = block_sum<NT>(acc[0], sh, tid);
        acc[1] = block_min<NT>(acc[1], sh, tid);
        acc[2] = block_max<NT>(acc[2], sh, tid);
        acc[3] = block_min<NT>(acc[3], sh, tid);
        acc[4] = block_max<NT>(acc[4], sh, tid);
        acc[5] = block_min<NT>(acc[5], sh, tid);
        if (tid == 0) {
            for (int q = 0; q < 6; q++) Sc->mon[q] = acc[q];
            Sc->counter[3] = 0u;
        }
    }
}

template <typename RS, typename R = RS>
__global__ void k_probe(LES_KERNEL_CONSTS, F11<RS> S, PropBuf<R> P, const int* __restrict__ st, int n, int kline,
                        double* __restrict__ out) {
    const int ny = C.ny, nz = C.nz;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int q = blockIdx.y;
    if (j >= ny || q >= n) return;
    const size_t id = cid(st[q], j, kline, ny, nz);
    double* o = out + ((size_t)q * ny + j) * 6;
    o[0] = (double)S.p[0][id];
    o[1] = (double)S.p[1][id];
    o[2] = (double)S.p[2][id];
    o[3] = (double)S.p[4][id];
    o[4] = (double)P.nu_t[id];
    o[5] = (double)P.S_mag[id];
}

// Host-driven steps: dt and t_loop come from the caller.
static __global__ void k_set_step(Scalars* __restrict__ Sc, double dt, int t_loop) {
    Sc->dt = dt;
    Sc->t_loop = t_loop;
}

// Device loop, last launch of a step: the probe lines of record_flame_region_data (:3403-3471)
// and dt/|u|max of this step go to history slot run_step, on steps with t_loop % 10 == 0 the
// monitor reductions (:3874-3918) too (other slots are left untouched), and the last block to
// finish advances the step counters.
template <typename RS, typename R = RS>
__global__ void __launch_bounds__(NT)
    k_loop_end(LES_KERNEL_CONSTS, F11<RS> S, PropBuf<R> P, double* __restrict__ part, Scalars* __restrict__ Sc,
               const int* __restrict__ st, int nst, int kline, size_t n, int cap, double* __restrict__ hprobe,
               double* __restrict__ hdt, double* __restrict__ humax, double* __restrict__ hmon) {
    __shared__ double sh[NT / 32];
    __shared__ int now[2];
    const int ny = C.ny, nz = C.nz, tid = threadIdx.x;
    pdl_wait();
    // The grid's last block advances these two: one thread reads them for its block, before the
    // block can be counted as arrived.
    if (tid == 0) {
        now[0] = Sc->run_step;
        now[1] = Sc->t_loop;
    }
    __syncthreads();
    const int slot = now[0];
    const bool monitor = now[1] % 10 == 0;              // uniform across the grid
    const unsigned nblk = gridDim.x;
    double v[6];
    if (slot >= 0 && slot < cap) {
        if (blockIdx.x == 0 && tid == 0) {
            hdt[slot] = Sc->dt;
            humax[slot] = Sc->umax_used;
        }
        for (int r = (int)blockIdx.x * NT + tid; r < nst * ny; r += (int)nblk * NT) {
            const int q = r / ny, j = r - q * ny;
            const size_t id = cid(st[q], j, kline, ny, nz);
            double* o = hprobe + (((size_t)slot * nst + q) * ny + j) * 6;
            const double a0 = (double)S.p[0][id], a1 = (double)S.p[1][id], a2 = (double)S.p[2][id],
                         a3 = (double)S.p[4][id], a4 = (double)P.nu_t[id], a5 = (double)P.S_mag[id];
            o[0] = a0; o[1] = a1; o[2] = a2; o[3] = a3; o[4] = a4; o[5] = a5;
        }
        if (monitor) {
            double mass = 0.0, tmin = 1.0e9, tmax = -1.0e9, gmin = 1.0e9, gmax = -1.0e9, ymin = 1.0e9;
            for (size_t id = (size_t)blockIdx.x * NT + tid; id < n; id += (size_t)nblk * NT) {
                double r = (double)S.p[5][id], T = (double)S.p[3][id], G = (double)S.p[4][id], Y = (double)S.p[6][id];
                mass += ((r * C.dx) * C.dy) * C.dz;
                tmin = fmin(tmin, T); tmax = fmax(tmax, T);
                gmin = fmin(gmin, G); gmax = fmax(gmax, G);
                ymin = fmin(ymin, Y);
            }
            v[0] = block_sum<NT>(mass, sh, tid);
            v[1] = block_min<NT>(tmin, sh, tid);
            v[2] = block_max<NT>(tmax, sh, tid);
            v[3] = block_min<NT>(gmin, sh, tid);
            v[4] = block_max<NT>(gmax, sh, tid);
            v[5] = block_min<NT>(ymin, sh, tid);
        }
    }
    if (!last_block(part, nblk, blockIdx.x, v, monitor && slot >= 0 && slot < cap ? 6 : 0, &Sc->counter[1], tid)) return;
    if (monitor && slot >= 0 && slot < cap) {
        double acc[6] = {0.0, 1.0e9, -1.0e9, 1.0e9, -1.0e9, 1.0e9};
#pragma unroll 4
        for (unsigned q = tid; q < nblk; q += NT) {
            acc[0] += __ldcg(&part[q]);
            acc[1] = fmin(acc[1], __ldcg(&part[nblk + q]));
            acc[2] = fmax(acc[2], __ldcg(&part[2 * nblk + q]));
            acc[3] = fmin(acc[3], __ldcg(&part[3 * nblk + q]));
            acc[4] = fmax(acc[4], __ldcg(&part[4 * nblk + q]));
            acc[5] = fmin(acc[5], __ldcg(&part[5 * nblk + q]));
        }
        acc[0] = block_sum<NT>(acc[0], sh, tid);
        acc[1] = block_min<NT>(acc[1], sh, tid);
        acc[2] = block_max<NT>(acc[2], sh, tid);
        acc[3] = block_min<NT>(acc[3], sh, tid);
        acc[4] = block_max<NT>(acc[4], sh, tid);
        acc[5] = block_min<NT>(acc[5], sh, tid);
        if (tid == 0)
            for (int q = 0; q < 6; q++) hmon[(size_t)slot * 6 + q] = acc[q];
    }
    if (tid == 0) {
        Sc->counter[1] = 0u;
        Sc->t_loop += 1;
        Sc->run_step += 1;
    }
}

// update_time_averages (:3166-3191) after the boundary conditions of steps with
// t_loop >= start (:4577-4579): first and second moments summed per cell in FP64.
template <typename RS, typename Form = RS>
__global__ void __launch_bounds__(NT) k_time_avg(F11<RS> S, AvgBuf A, Scalars* __restrict__ Sc, size_t n, int start) {
    if (Sc->t_loop < start) return;            // uniform across the grid
    for (size_t id = (size_t)blockIdx.x * NT + threadIdx.x; id < n; id += (size_t)gridDim.x * NT) {
        const double u = (double)S.p[0][id], v = (double)S.p[1][id], w = (double)S.p[2][id];
        const double G = (double)S.p[4][id];
        A.p[0][id] += u;
        A.p[1][id] += v;
        A.p[2][id] += w;
        A.p[9][id] += G;
        A.p[3][id] += u * u;
        A.p[4][id] += v * v;
        A.p[5][id] += w * w;
        A.p[6][id] += u * v;
        A.p[7][id] += u * w;
        A.p[8][id] += v * w;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) Sc->avg_steps += 1;
}

template <typename R, typename Form = R>
__global__ void k_check_finite(const R* __restrict__ x, size_t n, int* __restrict__ flag) {
    for (size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x; id < n; id += (size_t)gridDim.x * blockDim.x)
        if (!isfinite((double)x[id])) atomicExch(flag, 1);
}

}  // namespace les
