// les_launch.cuh -- stream-ordered launch sequence of one solver step, templated on the
// field type.  Included once per precision translation unit.
#pragma once

#include "les_ctx.h"
#include "les_kernels.cuh"
#include "les_tma.cuh"

namespace les {

// The state Phi_n is FP64 in both forms; R is the form's type of every other field.
using RS = double;

template <typename R>
static F11<R> f11(void* const* p) {
    F11<R> f;
    for (int q = 0; q < NSTATE; q++) f.p[q] = (R*)p[q];
    return f;
}

template <typename R>
static PropBuf<R> props(const DevCtx& c) {
    PropBuf<R> P;
    P.mu_mix = (R*)c.mu_mix;
    P.nu = (R*)c.nu;
    for (int s = 0; s < NSP; s++) P.D[s] = (R*)c.D[s];
    P.aT = (R*)c.aT;
    P.nu_t = (R*)c.nu_t;
    P.S_mag = (R*)c.S_mag;
    P.ST = (R*)c.ST;
    P.mu_eff = (R*)c.mu_eff;
    P.dbg_cp = c.debug ? (R*)c.dbg_cp : nullptr;
    P.dbg_lam = c.debug ? (R*)c.dbg_lam : nullptr;
    P.dbg_alpha = c.debug ? (R*)c.dbg_alpha : nullptr;
    P.grad_g = (R*)c.grad_g;
    return P;
}

static inline dim3 cell_block(const DevCtx& c, int cls) {
    const Shape t = kShapes[c.shape[cls]];
    return dim3((unsigned)t.bx, (unsigned)t.by, (unsigned)t.bz);
}
static inline dim3 cell_grid(const DevCtx& c, int cls) {
    const Shape t = kShapes[c.shape[cls]];
    return dim3((unsigned)((c.nz + t.bx - 1) / t.bx), (unsigned)((c.ny + t.by - 1) / t.by),
                (unsigned)((c.nx + t.bz - 1) / t.bz));
}

// A launch in a step's chain.  With `pdl` it may start while the launch before it in the stream
// drains (pdl_wait); without, it starts when everything before it is complete, as a launch does
// that follows an event of another stream.
template <typename... P, typename... A>
static inline void chain(bool pdl, void (*kernel)(P...), dim3 g, dim3 b, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = g;
    cfg.blockDim = b;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// The filter pass: 16-byte accesses where a row is a multiple of them, and as many planes per
// thread as leave every SM several blocks.
constexpr int FILTER_SEG = 8;
static inline int filter_vec(const DevCtx& c, size_t bytes) {
    const int v = (int)(16 / bytes);
    return c.nz % v == 0 ? v : 1;
}
static inline dim3 filter_grid(const DevCtx& c, size_t bytes, int& seg) {
    const int v = filter_vec(c, bytes);
    const unsigned gx = (unsigned)(((size_t)c.ny * (c.nz / v) + NT - 1) / NT);
    seg = FILTER_SEG;
    while (seg > 1 && (size_t)gx * ((c.nx + seg - 1) / seg) * NSTATE < 148 * 12) seg /= 2;
    return dim3(gx, (unsigned)((c.nx + seg - 1) / seg), NSTATE);
}
template <typename R, typename RI, bool BATCH>
static inline void launch_filter(bool pdl, const DevCtx& c, cudaStream_t st, const F11<RI>& in, const F11<R>& F, int members,
                                 const Batch& B) {
    constexpr int V = 16 / sizeof(RI);
    int seg;
    dim3 g = filter_grid(c, sizeof(RI), seg);
    g.z *= (unsigned)members;
    if (filter_vec(c, sizeof(RI)) == V)
        chain(pdl, k_filter<V, R, RI, BATCH>, g, NT, st, c.hC, c.attr, in, F, c.part, c.dS, seg, B);
    else
        chain(pdl, k_filter<1, R, RI, BATCH>, g, NT, st, c.hC, c.attr, in, F, c.part, c.dS, seg, B);
}
static inline size_t filter_blocks(const DevCtx& c) {
    int seg;
    const dim3 a = filter_grid(c, c.esz, seg), b = filter_grid(c, 8, seg);
    const size_t na = (size_t)a.x * a.y, nb = (size_t)b.x * b.y;
    return na > nb ? na : nb;
}

// The property, flow and scalar passes with the kernel instance of their tile's block size.
template <typename R, bool BATCH>
static inline void launch_props(bool pdl, const DevCtx& c, dim3 g, dim3 b, cudaStream_t st, const F11<R>& F, const PropBuf<R>& P,
                                int keep, const Batch& B) {
    if (b.x * b.y * b.z == 512) chain(pdl, k_props<R, BATCH, 512>, g, b, st, c.hC, c.attr, F, P, c.dS, keep, B);
    else chain(pdl, k_props<R, BATCH>, g, b, st, c.hC, c.attr, F, P, c.dS, keep, B);
}
template <int PART, typename R, bool BATCH>
static inline void launch_scalar_part(bool pdl, dim3 g, dim3 b, cudaStream_t st, const Consts& hC, const uint8_t* attr,
                                      const F11<R>& F, const PropBuf<R>& P, const F11<RS>& S, const F11<R>& St,
                                      const AccBuf<R>& acc, RS* rn, const KDbg<R>& kd, Scalars* dS,
                                      int stage, const Batch& B) {
    if (b.x * b.y * b.z == 512)
        chain(pdl, k_rhs_scalar<PART, R, RS, BATCH, 512>, g, b, st, hC, attr, F, P, S, St, acc, rn, kd, dS, stage, B);
    else
        chain(pdl, k_rhs_scalar<PART, R, RS, BATCH>, g, b, st, hC, attr, F, P, S, St, acc, rn, kd, dS, stage, B);
}
template <typename R, bool BATCH>
static inline void launch_scalar(bool pdl, dim3 g, dim3 b, cudaStream_t st, const Consts& hC, const uint8_t* attr,
                                 const F11<R>& F, const PropBuf<R>& P, const F11<RS>& S, const F11<R>& St,
                                 const AccBuf<R>& acc, RS* rn, const KDbg<R>& kd, Scalars* dS,
                                 int stage, const Batch& B) {
    if (stage == 0) launch_scalar_part<RK_FIRST, R, BATCH>(pdl, g, b, st, hC, attr, F, P, S, St, acc, rn, kd, dS, stage, B);
    else if (stage < 3) launch_scalar_part<RK_MIDDLE, R, BATCH>(pdl, g, b, st, hC, attr, F, P, S, St, acc, rn, kd, dS, stage, B);
    else launch_scalar_part<RK_LAST, R, BATCH>(pdl, g, b, st, hC, attr, F, P, S, St, acc, rn, kd, dS, stage, B);
}

template <int PART, typename R, bool BATCH>
static inline void launch_flow_part(bool pdl, dim3 g, dim3 b, cudaStream_t st, const Consts& hC, const uint8_t* attr,
                                      const F11<R>& F, const PropBuf<R>& P, const F11<RS>& S, const F11<R>& St,
                                      const AccBuf<R>& acc, RS* rn, const KDbg<R>& kd, Scalars* dS,
                                      int stage, const Batch& B) {
    if (b.x * b.y * b.z == 512)
        chain(pdl, k_rhs_flow<PART, R, RS, BATCH, 512>, g, b, st, hC, attr, F, P, S, St, acc, rn, kd, dS, stage, B);
    else
        chain(pdl, k_rhs_flow<PART, R, RS, BATCH>, g, b, st, hC, attr, F, P, S, St, acc, rn, kd, dS, stage, B);
}
template <typename R, bool BATCH>
static inline void launch_flow(bool pdl, dim3 g, dim3 b, cudaStream_t st, const Consts& hC, const uint8_t* attr,
                                 const F11<R>& F, const PropBuf<R>& P, const F11<RS>& S, const F11<R>& St,
                                 const AccBuf<R>& acc, RS* rn, const KDbg<R>& kd, Scalars* dS,
                                 int stage, const Batch& B) {
    if (stage == 0) launch_flow_part<RK_FIRST, R, BATCH>(pdl, g, b, st, hC, attr, F, P, S, St, acc, rn, kd, dS, stage, B);
    else if (stage < 3) launch_flow_part<RK_MIDDLE, R, BATCH>(pdl, g, b, st, hC, attr, F, P, S, St, acc, rn, kd, dS, stage, B);
    else launch_flow_part<RK_LAST, R, BATCH>(pdl, g, b, st, hC, attr, F, P, S, St, acc, rn, kd, dS, stage, B);
}

// The scalar and flow pass in one launch, where both_passes (les_ctx.h) has it so.
template <typename R>
static inline void launch_both(bool pdl, const DevCtx& c, cudaStream_t st, const F11<R>& F, const PropBuf<R>& P,
                               const F11<RS>& S, const F11<R>& St, const AccBuf<R>& acc, const KDbg<R>& kd, int stage) {
    const Shape t = kShapes[both_tile(c)];
    const int3 tile = make_int3(t.bx, t.by, t.bz);
    const dim3 g((unsigned)((c.nz + t.bx - 1) / t.bx), (unsigned)((c.ny + t.by - 1) / t.by), (unsigned)((c.nx + t.bz - 1) / t.bz));
    if (stage == 0) chain(pdl, k_rhs_both<RK_FIRST, R, RS>, g, 2 * NT, st, c.hC, c.attr, F, P, S, St, acc, kd, c.dS, stage, tile);
    else if (stage < 3) chain(pdl, k_rhs_both<RK_MIDDLE, R, RS>, g, 2 * NT, st, c.hC, c.attr, F, P, S, St, acc, kd, c.dS, stage, tile);
    else chain(pdl, k_rhs_both<RK_LAST, R, RS>, g, 2 * NT, st, c.hC, c.attr, F, P, S, St, acc, kd, c.dS, stage, tile);
}

// Every launch that writes per-block partials checks the buffer first: `per_block` values
// per block for `blocks` blocks must fit in c.part.
static inline bool part_fits(const DevCtx& c, size_t blocks, size_t per_block) {
    return blocks * per_block <= c.part_len;
}
static inline size_t cell_blocks(const DevCtx& c, int cls) {
    dim3 g = cell_grid(c, cls);
    return (size_t)g.x * g.y * g.z;
}

// The end of a step after the four RK stages: boundary conditions, EOS, time averages and,
// in the device loop, the step's history and counters.
template <typename R>
void step_tail(DevCtx& c, cudaStream_t st, bool device_mode, bool pdl) {
    F11<RS> S = f11<RS>(c.S);
    PropBuf<R> P = props<R>(c);
    const unsigned inner = (unsigned)(((size_t)(c.ny - 2) * (c.nz - 2) + NT - 1) / NT);
    chain(pdl, k_bc<RS, R>, (unsigned)(c.nx - 2) + inner, NT, st, c.hC, c.attr, S, c.plane, c.noise, c.inlet_pos, c.dS);
    if (c.avg) {
        AvgBuf A;
        for (int q = 0; q < NAVG; q++) A.p[q] = c.avg + (size_t)q * c.n;
        k_time_avg<RS, R><<<MON_BLOCKS, NT, 0, st>>>(S, A, c.dS, c.n, c.avg_start);
    }
    if (device_mode)
        chain(!c.timing && !c.avg, k_loop_end<RS, R>, MON_BLOCKS, NT, st, c.hC, S, P, c.part, c.dS, c.loop_st,
              c.loop_nst, c.loop_kline, c.n, c.loop_cap, c.hist_probe, c.hist_dt, c.hist_umax, c.hist_mon);
}

// One time step.  Host-driven (device_mode false): dt and t_loop come from the caller and
// the inflow from lesgpu_set_inflow.  Device loop (true): dt, the vortex update and the
// inflow noise are computed on the GPU first, and the step's history is recorded at the
// end; every launch then reads only device memory, so the sequence can be graph-captured.
template <typename R>
cudaError_t step_impl(DevCtx& c, double dt, int t_loop, bool device_mode) {
    cudaStream_t st = c.stream;
    if (!part_fits(c, filter_blocks(c), 1) || !part_fits(c, MON_BLOCKS, 6))
        return cudaErrorInvalidValue;
    const dim3 gB = cell_grid(c, SH_STRAIN), bB = cell_block(c, SH_STRAIN);
    const dim3 gC = cell_grid(c, SH_FLOW), bC = cell_block(c, SH_FLOW);
    const dim3 gD = cell_grid(c, SH_SCALAR), bD = cell_block(c, SH_SCALAR);
    F11<RS> S = f11<RS>(c.S);
    F11<R> St = f11<R>(c.St), F = f11<R>(c.F);
    PropBuf<R> P = props<R>(c);
    AccBuf<R> acc;
    for (int q = 0; q < NACC; q++) acc.p[q] = (R*)c.acc[q];
    KDbg<R> kd;
    for (int q = 0; q < NACC; q++) kd.p[q] = c.debug ? (R*)c.kd[q] : nullptr;
    KDbg<R> knone;
    for (int q = 0; q < NACC; q++) knone.p[q] = nullptr;
    RS* rn = (RS*)c.rn;

    int tm = tmark_begin(c, 0);
    // The head of a step runs on a side stream: dt and the draws of the device loop beside the
    // first stage's filter and properties, which need neither, the SEM inflow plane (:943-1075)
    // beside the four RK stages, as only the boundary conditions read it.  With kernel timing
    // on it runs in line so that its events bracket it alone.
    const bool overlap = !c.timing && c.side;
    cudaStream_t hs = overlap ? c.side : st;
    if (!device_mode) k_set_step<<<1, 1, 0, st>>>(c.dS, dt, t_loop);
    if (overlap) {
        cudaEventRecord(c.ev_fork, st);
        cudaStreamWaitEvent(hs, c.ev_fork, 0);
    }
    if (device_mode) {
        loop_pre(c, hs);
        if (overlap) cudaEventRecord(c.ev_dt, hs);
    }
    sem_inflow(c, hs);
    if (overlap) cudaEventRecord(c.ev_join, hs);
    tmark_end(c, tm);
    const bool pdl = !c.timing;
    // four RK4 stages (:4428-4544)
    for (int s = 0; s < 4; s++) {
        tm = tmark_begin(c, 1);
        if (s == 0) launch_filter<R, RS, false>(false, c, st, S, F, 1, Batch{});
        else launch_filter<R, R, false>(pdl, c, st, St, F, 1, Batch{});
        tmark_end(c, tm);
        tm = tmark_begin(c, 2);
        launch_props<R, false>(pdl, c, gB, bB, st, F, P, s == 3 ? 1 : 0, Batch{});
        tmark_end(c, tm);
        if (s == 0 && device_mode && overlap) cudaStreamWaitEvent(st, c.ev_dt, 0);
        // the k-arrays of the first stage are kept for inspection when requested
        const KDbg<R>& kds = (s == 0) ? kd : knone;
        if (both_passes(c)) {   // (kernel timing brackets the two apart)
            launch_both<R>(pdl && !(s == 0 && device_mode && overlap), c, st, F, P, S, St, acc, kds, s);
            continue;
        }
        tm = tmark_begin(c, 5);
        if (c.scalar_tma && c.tma_ok) launch_scalar_tma<R, RS>(c, st, F, P, S, St, acc, rn, kds, s);
        else launch_scalar<R, false>(pdl && !(s == 0 && device_mode && overlap), gD, bD, st, c.hC, c.attr, F, P, S, St, acc, rn, kds, c.dS, s, Batch{});
        tmark_end(c, tm);
        tm = tmark_begin(c, 3);
        launch_flow<R, false>(pdl, gC, bC, st, c.hC, c.attr, F, P, S, St, acc, rn, kds, c.dS, s, Batch{});
        tmark_end(c, tm);
    }
    // apply_boundary_conditions (:2967-3161)
    if (overlap) cudaStreamWaitEvent(st, c.ev_join, 0);
    tm = tmark_begin(c, 4);
    step_tail<R>(c, st, device_mode, pdl && !overlap);
    tmark_end(c, tm);
    tmark_flush(c);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ batched members
// Several members of one grid shape and precision, stepped together: each member's step head
// (dt, vortex and noise draws, SEM plane) and tail (boundary conditions, history) on its own
// stream as above, and the four RK stages of all of them in one launch per pass, whose grid is
// the first member's grid repeated along z once per member.  Every block reads its member's
// arena offset, attribute map, reductions and model constants from the member table (les_common.cuh,
// MemberTab); the tiles are the first member's.

template <typename R>
cudaError_t batch_head(DevCtx& c) {
    loop_pre(c, c.stream);
    sem_inflow(c, c.stream);
    return cudaGetLastError();
}

template <typename R>
cudaError_t batch_tail(DevCtx& c) {
    step_tail<R>(c, c.stream, true, false);
    return cudaGetLastError();
}

template <typename R>
cudaError_t batch_stages(DevCtx& c0, const MemberTab* mt, int nmem, cudaStream_t st) {
    if (nmem < 1 || !part_fits(c0, filter_blocks(c0), 1)) return cudaErrorInvalidValue;
    auto grid = [&](int cls, Batch& b) {
        dim3 g = cell_grid(c0, cls);
        b.mt = mt;
        b.gz = (int)g.z;
        g.z *= (unsigned)nmem;
        return g;
    };
    Batch BB, BC, BD;
    const dim3 gB = grid(SH_STRAIN, BB), bB = cell_block(c0, SH_STRAIN);
    const dim3 gC = grid(SH_FLOW, BC), bC = cell_block(c0, SH_FLOW);
    const dim3 gD = grid(SH_SCALAR, BD), bD = cell_block(c0, SH_SCALAR);
    if (gB.z > 65535u || (unsigned)nmem * NSTATE > 65535u || gC.z > 65535u || gD.z > 65535u) return cudaErrorInvalidConfiguration;
    F11<RS> S = f11<RS>(c0.S);
    F11<R> St = f11<R>(c0.St), F = f11<R>(c0.F);
    PropBuf<R> P = props<R>(c0);
    AccBuf<R> acc;
    for (int q = 0; q < NACC; q++) acc.p[q] = (R*)c0.acc[q];
    KDbg<R> knone;
    for (int q = 0; q < NACC; q++) knone.p[q] = nullptr;
    RS* rn = (RS*)c0.rn;
    for (int s = 0; s < 4; s++) {
        if (s == 0) launch_filter<R, RS, true>(false, c0, st, S, F, nmem, Batch{mt, 0});
        else launch_filter<R, R, true>(true, c0, st, St, F, nmem, Batch{mt, 0});
        launch_props<R, true>(true, c0, gB, bB, st, F, P, s == 3 ? 1 : 0, BB);
        launch_scalar<R, true>(true, gD, bD, st, c0.hC, c0.attr, F, P, S, St, acc, rn, knone, c0.dS, s, BD);
        launch_flow<R, true>(true, gC, bC, st, c0.hC, c0.attr, F, P, S, St, acc, rn, knone, c0.dS, s, BC);
    }
    return cudaGetLastError();
}

// Stage-1 right-hand side at the current state with the inspection buffers filled (when
// debug buffers exist); the state itself is not advanced (dt = 0 leaves the stage state
// equal to Phi_n).  The four kernels are bracketed by the kernel-timing marks, which the
// tile autotuner reads; with `one_launch` the scalar and flow pass are one, under the flow pass's mark.
template <typename R>
cudaError_t rhs_only_impl(DevCtx& c, int t_loop, bool one_launch) {
    cudaStream_t st = c.stream;
    if (!part_fits(c, filter_blocks(c), 1)) return cudaErrorInvalidValue;
    F11<RS> S = f11<RS>(c.S);
    F11<R> St = f11<R>(c.St), F = f11<R>(c.F);
    PropBuf<R> P = props<R>(c);
    AccBuf<R> acc;
    for (int q = 0; q < NACC; q++) acc.p[q] = (R*)c.acc[q];
    KDbg<R> kd;
    for (int q = 0; q < NACC; q++) kd.p[q] = (R*)c.kd[q];
    RS* rn = (RS*)c.rn;
    k_set_step<<<1, 1, 0, st>>>(c.dS, 0.0, t_loop);
    // the nu and alpha maxima become this state's (the property pass raises them)
    static_assert(offsetof(Scalars, alphamax) == offsetof(Scalars, numax) + sizeof(double), "cleared together");
    cudaMemsetAsync(&c.dS->numax, 0, 2 * sizeof(double), st);
    int tm = tmark_begin(c, 1);
    launch_filter<R, RS, false>(false, c, st, S, F, 1, Batch{});
    tmark_end(c, tm);
    tm = tmark_begin(c, 2);
    launch_props<R, false>(false, c, cell_grid(c, SH_STRAIN), cell_block(c, SH_STRAIN), st, F, P, 1, Batch{});
    tmark_end(c, tm);
    if (one_launch) {
        tm = tmark_begin(c, 3);
        launch_both<R>(false, c, st, F, P, S, St, acc, kd, 0);
        tmark_end(c, tm);
        tmark_flush(c);
        return cudaGetLastError();
    }
    tm = tmark_begin(c, 5);
    if (c.scalar_tma && c.tma_ok)
        launch_scalar_tma<R, RS>(c, st, F, P, S, St, acc, rn, kd, 0);
    else
        launch_scalar<R, false>(false, cell_grid(c, SH_SCALAR), cell_block(c, SH_SCALAR), st, c.hC, c.attr, F, P, S, St,
                                acc, rn, kd, c.dS, 0, Batch{});
    tmark_end(c, tm);
    tm = tmark_begin(c, 3);
    launch_flow<R, false>(false, cell_grid(c, SH_FLOW), cell_block(c, SH_FLOW), st, c.hC, c.attr, F, P, S, St, acc, rn, kd,
                          c.dS, 0, Batch{});
    tmark_end(c, tm);
    tmark_flush(c);
    return cudaGetLastError();
}

template <typename R>
cudaError_t umax_impl(DevCtx& c) {
    if (!part_fits(c, cell_blocks(c, SH_EOS), 1)) return cudaErrorInvalidValue;
    k_umax<RS, R><<<cell_grid(c, SH_EOS), cell_block(c, SH_EOS), 0, c.stream>>>(c.hC, c.attr, f11<RS>(c.S), c.part,
                                                                               c.dS);
    return cudaGetLastError();
}

template <typename R>
cudaError_t monitor_impl(DevCtx& c) {
    const int nb = MON_BLOCKS;
    if (!part_fits(c, nb, 6)) return cudaErrorInvalidValue;
    k_monitor<RS, R><<<nb, NT, 0, c.stream>>>(c.hC, f11<RS>(c.S), c.part, c.dS, c.n);
    return cudaGetLastError();
}

template <typename R>
cudaError_t probe_impl(DevCtx& c, int n, int kline) {
    const int tpb = 64;
    k_probe<RS, R><<<dim3((c.ny + tpb - 1) / tpb, n), tpb, 0, c.stream>>>(c.hC, f11<RS>(c.S), props<R>(c), c.probe_st,
                                                                          n, kline, c.probe_out);
    return cudaGetLastError();
}

template <typename R>
cudaError_t check_impl(DevCtx& c, int field) {
    cudaMemsetAsync(c.flag, 0, sizeof(int), c.stream);
    if (field < NSTATE) k_check_finite<RS, R><<<592, 256, 0, c.stream>>>((const RS*)c.S[field], c.n, c.flag);
    else k_check_finite<R, R><<<592, 256, 0, c.stream>>>((const R*)c.nu_t, c.n, c.flag);
    return cudaGetLastError();
}

}  // namespace les
