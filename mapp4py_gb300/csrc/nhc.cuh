// Nose-Hoover chain of the particle thermostat on the device
// (ThermostatNHC::operator(), thermostat.cpp:47-143) and its use by
// MDNVT::run (md_nvt.cpp:409-438): one half = chain(T/T0), then
// mvv *= fac^2, T *= fac^2.
#pragma once

#include "system.h"

namespace mappg {

// The chain is one thread's serial work at the end of each MD step, so its
// cost is the latency of dependent FP64 operations, 65 clocks each on GB300
// (a division 670, an exp 1,100): no divisions; near 0, where a chain lives,
// short polynomials; the branch on the argument's size from its bits; and
// for the default chain (Chain3) everything that does not wait for the
// temperature formed ahead of it.  A half took 6.1-7.1 thousand clocks with
// divisions, exp and the variables in memory, 3.1 (closing) and 4.5 (opening) so; 100 steps of 4,000
// mixed atoms, with the reductions around it, 7.2 -> 5.4 ms.

// |x| < 1/64, from the exponent bits
__host__ __device__ __forceinline__ bool nhc_small(double x) {
#ifdef __CUDA_ARCH__
    return (__double2hiint(x) & 0x7fffffff) < 0x3f900000;
#else
    return fabs(x) < 0.015625;
#endif
}

static __host__ __device__ __noinline__ double nhc_exp_far(double x) { return exp(x); }
static __host__ __device__ __noinline__ double nhc_f_far(double x) { return (exp(x) - 1.0) / x; }

// (e^x - 1)/x, the reference's series near 0
__host__ __device__ __forceinline__ double nhc_f(double x) {
    if (!nhc_small(x)) return nhc_f_far(x);
    return (1.0 + 0.5 * x) + (x * x) * (1.0 / 6.0 + (1.0 / 24.0) * x);
}

// e^x: Taylor's series to x^7 below 1/64, where the rest is below 1e-19
__host__ __device__ __forceinline__ double nhc_exp(double x) {
    if (!nhc_small(x)) return nhc_exp_far(x);
    const double x2 = x * x;
    const double b = 0.5 + (1.0 / 6.0) * x, c = 1.0 / 24.0 + (1.0 / 120.0) * x, d = 1.0 / 720.0 + (1.0 / 5040.0) * x;
    return 1.0 + (x + x2 * (b + x2 * (c + x2 * d)));
}

// ThermostatNHC::operator() with the chain variables in e[0..L-1]; LT is L
// where it is known when compiled (the variables then live in registers)
template <int LT, class Eta>
__host__ __device__ __forceinline__ double nhc_chain(const NhcParams& P, Eta& e, double T_r) {
    const int L = LT ? LT : P.L;
    double rescale = 1.0, prev_fac, tmp;
    if (L == 1) {
        for (int it = 0; it < P.niters; it++) {
            e[0] += P.ddt2 * P.freq_sq * (T_r - 1.0);
            prev_fac = nhc_exp(-P.ddt * e[0]);
            rescale *= prev_fac;
            T_r *= prev_fac * prev_fac;
            e[0] += P.ddt2 * P.freq_sq * (T_r - 1.0);
        }
        return rescale;
    }
    const double h = P.ddt2, w = P.freq_sq;
    for (int it = 0; it < P.niters; it++) {
        e[L - 1] += h * (e[L - 2] * e[L - 2] - w);
        prev_fac = -e[L - 1];
#pragma unroll
        for (int ich = L - 2; ich > 0; ich--) {
            const double g = h * (prev_fac * e[ich] + (e[ich - 1] * e[ich - 1] - w));
            e[ich] += nhc_f(prev_fac * h) * g;
            prev_fac = -e[ich];
        }
        const double g0 = h * (prev_fac * e[0] + w * (T_r - 1.0));
        const double f0 = nhc_f(prev_fac * h);  // of e[1], which the closing update uses too
        e[0] += f0 * g0;
        tmp = nhc_exp(-P.ddt * e[0]);
        rescale *= tmp;
        T_r *= tmp * tmp;
        e[0] += f0 * (h * (prev_fac * e[0] + (T_r - 1.0) * w));
        prev_fac = P.ndof * e[0] * e[0] - w;
#pragma unroll
        for (int ich = 1; ich < L - 1; ich++) {
            e[ich] += nhc_f(-e[ich + 1] * h) * (h * (-e[ich + 1] * e[ich] + prev_fac));
            prev_fac = e[ich] * e[ich] - w;
        }
        e[L - 1] += h * prev_fac;
    }
    return rescale;
}

static __host__ __device__ __noinline__ double nhc_any(const NhcParams& P, double* eta, double T_r) {
    return nhc_chain<0>(P, eta, T_r);
}

__host__ __device__ inline double nhc_step(const NhcParams& P, double* eta, double T_r) {
    if (P.L != 3) return nhc_any(P, eta, T_r);
    double e[3] = {eta[0], eta[1], eta[2]};  // the default length
    const double r = nhc_chain<3>(P, e, T_r);
    for (int k = 0; k < 3; k++) eta[k] = e[k];
    return r;
}

#ifdef __CUDACC__
// nhc_step of a chain of three links and one iteration in two parts: pre()
// updates what does not need the temperature, post(T_r) the rest.  ok() is
// false if an argument left the range of the polynomials (the caller then
// takes nhc_step)
struct Chain3 {
    double h, w, e0, e1, e2, f1, f0;
    bool in_range;
    static __device__ __forceinline__ double f(double x) {
        return fma(x * x, fma(1.0 / 24.0, x, 1.0 / 6.0), fma(0.5, x, 1.0));
    }
    __device__ __forceinline__ void pre(const NhcParams& P, const double* eta) {
        h = P.ddt2;
        w = P.freq_sq;
        e0 = eta[0];
        e1 = eta[1];
        e2 = fma(h, fma(e1, e1, -w), eta[2]);
        const double x = -e2 * h, g = h * fma(-e2, e1, fma(e0, e0, -w));
        f1 = f(x);  // of e2, for both updates of e1
        e1 = fma(f1, g, e1);
        const double y = -e1 * h;
        f0 = f(y);  // of e1, for both updates of e0
        in_range = nhc_small(x) && nhc_small(y);
    }
    __device__ __forceinline__ double post(const NhcParams& P, double T_r) {
        e0 = fma(f0, h * fma(-e1, e0, w * (T_r - 1.0)), e0);
        const double x = -P.ddt * e0, x2 = x * x;
        const double b = fma(1.0 / 6.0, x, 0.5), c = fma(1.0 / 120.0, x, 1.0 / 24.0), d = fma(1.0 / 5040.0, x, 1.0 / 720.0);
        const double fac = 1.0 + fma(x2, fma(x2, fma(x2, d, c), b), x);  // e^x
        in_range = in_range && nhc_small(x);
        const double f2 = fac * fac;
        e0 = fma(f0, h * fma(-e1, e0, w * fma(T_r, f2, -1.0)), e0);
        e1 = fma(f1, h * fma(-e2, e1, fma(P.ndof_d * e0, e0, -w)), e1);
        e2 = fma(h, fma(e1, e1, -w), e2);
        return fac;
    }
};
#endif

template <class State>
__device__ inline double thermo_half(const NhcParams& P, State* sc) {
    double fac = nhc_step(P, sc->eta, sc->T_part * P.T_inv);
    double f2 = fac * fac;
    for (int k = 0; k < 6; k++) sc->mvv[k] *= f2;
    sc->T_part *= f2;
    return fac;
}

// thermo row: pe, T, mvv[6], virial[6]
__device__ inline void write_thermo_row(double* thermo, const DevScalars* sc, long long row) {
    if (!thermo) return;
    double* r = thermo + 14 * row;
    r[0] = sc->energy;
    r[1] = sc->T_part;
    for (int k = 0; k < 6; k++) r[2 + k] = sc->mvv[k];
    for (int k = 0; k < 6; k++) r[8 + k] = sc->virial[k];
}

}  // namespace mappg
