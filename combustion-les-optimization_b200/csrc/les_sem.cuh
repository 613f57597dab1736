// les_sem.cuh -- synthetic-eddy inflow plane kernels.  Compiled only into the FP64 unit
// (no FMA contraction) and shared by both precision forms: the plane is always FP64.
#pragma once

#include "les_common.cuh"

namespace les {

// ------------------------------------------------------------------ SEM inflow plane

// generate_inlet_turbulence_SEM plane sum (:965-1003).  Few vortices reach a cell, but the cell's
// value is the reference's serial sum in vortex order: a warp takes a cell, its lanes test 32
// vortices at a time (the root and the quotient of each, which is where the time goes), and the
// contributions found are added one after another in lane order, the same roundings as the
// serial loop.  One thread a cell waited for 2000 roots in turn (60x20x40,
// 2000 vortices, eight host-driven steps: 3004 -> 1926 us; plane and normalisation at 256x128x128, 800
// vortices, with the chunked sums below: 0.21 -> 0.05 ms a step).
constexpr int SEM_WARPS = 4;
__global__ void __launch_bounds__(32 * SEM_WARPS)
    k_sem_plane(const Consts* __restrict__ C, const int* __restrict__ inlet_list, int n_inlet,
                const double* __restrict__ vort, int nv, double* __restrict__ plane) {
    const int q = blockIdx.x * SEM_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (q >= n_inlet) return;
    const int ny = C->ny, nz = C->nz, p = inlet_list[q];
    const int j = p / nz, k = p % nz;
    const double y = j * C->dy, z = k * C->dz;
    double su = 0.0, svv = 0.0, sw = 0.0;
    for (int base = 0; base < nv; base += 32) {
        const int v = base + lane;
        double cu = 0.0, cv = 0.0, cw = 0.0;
        bool in = false;
        if (v < nv) {
            const double* V = vort + 7 * (size_t)v;
            const double ddx = 0.0 - V[0], ddy = y - V[1], ddz = z - V[2], rad = V[3];
            const double dist = sqrt(ddx * ddx + ddy * ddy + ddz * ddz);
            in = dist < rad;
            if (in) {
                const double infl = 1.0 - (dist / rad);
                cu = V[4] * infl;
                cv = V[5] * infl;
                cw = V[6] * infl;
            }
        }
        for (unsigned m = __ballot_sync(0xffffffffu, in); m != 0u; m &= m - 1u) {
            const int l = __ffs((int)m) - 1;
            su += __shfl_sync(0xffffffffu, cu, l);
            svv += __shfl_sync(0xffffffffu, cv, l);
            sw += __shfl_sync(0xffffffffu, cw, l);
        }
    }
    if (lane == 0) {
        const size_t npl = (size_t)ny * nz;
        plane[p] = su;
        plane[npl + p] = svv;
        plane[2 * npl + p] = sw;
    }
}

// Mean removal and rms rescale (:1005-1074).  The running sums are serial, in the reference's
// (j, k) order, so the plane is bit-identical to the reference's: one thread a component adds, from
// shared memory that the block fills a chunk at a time, so that only the additions are in turn.
constexpr int SEM_CHUNK = 1024;
__global__ void __launch_bounds__(256)
    k_sem_normalize(const Consts* __restrict__ C, const int* __restrict__ inlet_list, int n_inlet,
                    double* __restrict__ plane, Scalars* __restrict__ Sc) {
    __shared__ double buf[3][SEM_CHUNK];
    __shared__ double tot[3];
    const size_t npl = (size_t)C->ny * C->nz;
    const int t = threadIdx.x;
    if (n_inlet <= 0) return;
    double s = 0.0;
    for (int base = 0; base < n_inlet; base += SEM_CHUNK) {
        const int m = min(SEM_CHUNK, n_inlet - base);
        __syncthreads();
        for (int q = t; q < m; q += blockDim.x) {
            const int p = inlet_list[base + q];
            buf[0][q] = plane[p];
            buf[1][q] = plane[npl + p];
            buf[2][q] = plane[2 * npl + p];
        }
        __syncthreads();
        if (t < 3)
#pragma unroll 16
            for (int q = 0; q < m; q++) s += buf[t][q];
    }
    if (t < 3) {
        tot[t] = s / n_inlet;
        Sc->sem[t] = s;
        s = 0.0;
    }
    for (int base = 0; base < n_inlet; base += SEM_CHUNK) {
        const int m = min(SEM_CHUNK, n_inlet - base);
        __syncthreads();
        for (int q = t; q < m; q += blockDim.x) {
            const int p = inlet_list[base + q];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const double x = plane[c * npl + p] - tot[c];
                plane[c * npl + p] = x;
                buf[c][q] = x * x;
            }
        }
        __syncthreads();
        if (t < 3)
#pragma unroll 16
            for (int q = 0; q < m; q++) s += buf[t][q];
    }
    __syncthreads();
    if (t < 3) {
        const double rms = sqrt(s / n_inlet);
        tot[t] = (rms > SMALL) ? C->ti_rms / rms : 0.0;
        Sc->sem[3 + t] = rms;
    }
    __syncthreads();
    for (int q = t; q < n_inlet; q += blockDim.x) {
        const int p = inlet_list[q];
        plane[p] *= tot[0];
        plane[npl + p] *= tot[1];
        plane[2 * npl + p] *= tot[2];
    }
}

}  // namespace les
