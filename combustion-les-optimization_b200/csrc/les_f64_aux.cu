// les_f64_aux.cu -- the parts of a step that both precision forms share and that must give
// the host's bits: the SEM inflow plane (bit-identical to the reference's plane for the same
// vortices), the device-loop dt and rand() draws (bit-identical to the host-driven loop), and
// the division self-check.  Always built with -fmad=false, whatever the stage kernels use.
#include <math.h>
#include <string.h>
#include <vector>

#include "les_ctx.h"
#include "les_sem.cuh"
#include "les_devloop.cuh"

namespace les {

cudaError_t sem_inflow(DevCtx& c, cudaStream_t st) {
    if (c.n_inlet <= 0) return cudaSuccess;
    k_sem_plane<<<(c.n_inlet + SEM_WARPS - 1) / SEM_WARPS, 32 * SEM_WARPS, 0, st>>>(c.dC, c.inlet_list, c.n_inlet,
                                                                                     c.vort, c.nv, c.plane);
    k_sem_normalize<<<1, 256, 0, st>>>(c.dC, c.inlet_list, c.n_inlet, c.plane, c.dS);
    return cudaGetLastError();
}

// Checks cdv() against IEEE division: n pseudo-random dividends spanning 2^-60..2^60 for
// each divisor; counts quotients whose bit patterns differ.
__global__ void k_selfcheck_div(const DC* __restrict__ ds, int nd, size_t n, unsigned long long seed,
                                unsigned long long* __restrict__ bad) {
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    unsigned long long local = 0;
    for (int d = 0; d < nd; d++) {
        const DC dc = ds[d];
        for (size_t q = tid; q < n; q += stride) {
            unsigned long long z = seed + q * 0x9E3779B97F4A7C15ull + (unsigned long long)d * 0xD1B54A32D192ED03ull;
            z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
            z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
            z ^= z >> 31;
            unsigned long long e = (unsigned long long)(1023 - 60 + (int)((z >> 52) % 121));
            unsigned long long bits = (z & 0x000FFFFFFFFFFFFFull) | (e << 52) | ((z >> 63) << 63);
            double x = __longlong_as_double((long long)bits);
            if (__double_as_longlong(x / dc.c) != __double_as_longlong(cdv(x, dc))) local++;
        }
    }
    if (local) atomicAdd(bad, local);
}

int selfcheck_division(const double* divisors, int nd, size_t n, unsigned long long seed, unsigned long long* bad) {
    DC* dd = nullptr;
    unsigned long long* db = nullptr;
    std::vector<DC> h(nd);
    for (int q = 0; q < nd; q++) { h[q].c = divisors[q]; h[q].r = 1.0 / divisors[q]; }
    if (cudaMalloc(&dd, nd * sizeof(DC)) != cudaSuccess) return -3;
    if (cudaMalloc(&db, sizeof(unsigned long long)) != cudaSuccess) { cudaFree(dd); return -3; }
    cudaMemcpy(dd, h.data(), nd * sizeof(DC), cudaMemcpyHostToDevice);
    cudaMemset(db, 0, sizeof(unsigned long long));
    k_selfcheck_div<<<1184, 256>>>(dd, nd, n, seed, db);
    cudaError_t e = cudaMemcpy(bad, db, sizeof(unsigned long long), cudaMemcpyDeviceToHost);
    cudaFree(dd);
    cudaFree(db);
    return e == cudaSuccess ? 0 : -2;
}

// frcp, exp2_fit, cquot and qdiv_normal against CUDA's own functions (lesgpu_selfcheck_math).
__device__ __forceinline__ double last_places(double x, double want) {
    return scalbn(fabs(x - want), 52 - ilogb(want));
}
__global__ void k_selfcheck_math(const double* __restrict__ tab, size_t n, unsigned long long seed, double* __restrict__ err,
                                 unsigned long long* __restrict__ bad) {
    __shared__ double t16[EXP_STEPS];
    if (threadIdx.x < EXP_STEPS) t16[threadIdx.x] = tab[threadIdx.x];
    __syncthreads();
    double e[3] = {0.0, 0.0, 0.0};
    unsigned long long differ = 0;
    auto mix = [](unsigned long long z) {
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    };
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x) {
        const unsigned long long z = mix(seed + q * 0x9E3779B97F4A7C15ull), y = mix(z + 0xD1B54A32D192ED03ull);
        const double x = __longlong_as_double((long long)((z & 0x000FFFFFFFFFFFFFull) | ((923ull + (z >> 52) % 201) << 52)));
        const double a = __longlong_as_double((long long)((y & 0x000FFFFFFFFFFFFFull) | ((923ull + (y >> 52) % 201) << 52)));
        const double r = frcp(x), t = ((double)(long long)y * 0x1p-63) * 15999.0;
        e[0] = fmax(e[0], last_places(r, 1.0 / x));
        e[1] = fmax(e[1], last_places(exp2_fit(t, t16), exp2(t * (1.0 / EXP_STEPS))));
        e[2] = fmax(e[2], last_places(cquot(a, x, r), a / x));
        const float fa = __uint_as_float((unsigned)y), fb = __uint_as_float((unsigned)z);
        if (isfinite(fa) && fabsf(fb) >= 1.17549435e-38f &&
            __float_as_uint(qdiv_normal(fa, fb)) != __float_as_uint(qdiv(fa, fb)))
            differ++;
    }
    for (int q = 0; q < 3; q++)
        atomicMax(reinterpret_cast<unsigned long long*>(err + q), (unsigned long long)__double_as_longlong(e[q]));
    if (differ) atomicAdd(bad, differ);
}

int selfcheck_math(size_t n, unsigned long long seed, double out[4]) {
    double h[EXP_STEPS + 4] = {};
    for (int j = 0; j < EXP_STEPS; j++) h[j] = (double)exp2l((long double)j / EXP_STEPS);
    double* d = nullptr;
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess) return -3;
    cudaMemcpy(d, h, sizeof(h), cudaMemcpyHostToDevice);
    k_selfcheck_math<<<1184, 256>>>(d, n, seed, d + EXP_STEPS, reinterpret_cast<unsigned long long*>(d + EXP_STEPS + 3));
    cudaError_t e = cudaMemcpy(out, d + EXP_STEPS, 4 * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(d);
    unsigned long long differ;
    memcpy(&differ, out + 3, sizeof(differ));
    out[3] = (double)differ;
    return e == cudaSuccess ? 0 : -2;
}

cudaError_t loop_pre(DevCtx& c, cudaStream_t st) {
    k_loop_pre<<<1, LOOP_THREADS, 0, st>>>(c.dC, c.dS, (LoopState*)c.dL, c.J, c.jrows, c.vort, c.nv, c.noise,
                                                 c.n_inlet, c.lp_lbox, c.lp_ly, c.lp_lz, c.lp_uin, c.lp_ti, c.lp_ell,
                                                 c.lp_cfl, c.lp_cfld, c.lp_dx);
    return cudaGetLastError();
}

}  // namespace les
