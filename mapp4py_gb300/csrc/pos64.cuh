// What the FP64 kernels share: positions with their periodic images, the
// shift and cutoff tables of a block, the embedding function.
#pragma once

#include "eam_common.cuh"

namespace mappg {

// atom i's position and the bin-edge flags that turn a bin step into an image
struct Pos64 {
    double x, y, z;
    int lo[3], hi[3];
    __device__ __forceinline__ void load(const EamArgs& a, int i) { load(a, i, a.nb); }
    // nb: the bins of the atom's cell
    __device__ __forceinline__ void load(const EamArgs& a, int i, const int* nb) {
        x = a.x[i];
        y = a.x[a.n + i];
        z = a.x[2 * a.n + i];
        int bc = a.binc[i];
        int b[3] = {bc & 1023, (bc >> 10) & 1023, (bc >> 20) & 1023};
#pragma unroll
        for (int d = 0; d < 3; d++) {
            lo[d] = b[d] == 0;
            hi[d] = b[d] == nb[d] - 1;
        }
    }
    // dx = x_i - (x_j + n*H)
    __device__ __forceinline__ void delta(const EamArgs& a, const double (*sh)[3], int e, double& dx, double& dy,
                                          double& dz) const {
        const int j = entry_j(e);
        const int d0 = entry_step(e, 0), d1 = entry_step(e, 1), d2 = entry_step(e, 2);
        int n0 = (d0 < 0 && lo[0]) ? -1 : ((d0 > 0 && hi[0]) ? 1 : 0);
        int n1 = (d1 < 0 && lo[1]) ? -1 : ((d1 > 0 && hi[1]) ? 1 : 0);
        int n2 = (d2 < 0 && lo[2]) ? -1 : ((d2 > 0 && hi[2]) ? 1 : 0);
        double xj = __ldg(a.x + j), yj = __ldg(a.x + a.n + j), zj = __ldg(a.x + 2 * a.n + j);
        // most pairs of a large cell reach no image: three FP64 additions less
        if ((n0 | n1 | n2) != 0) {
            const double* s = sh[(n0 + 1) + 3 * (n1 + 1) + 9 * (n2 + 1)];
            xj += s[0];
            yj += s[1];
            zj += s[2];
        }
        dx = x - xj;
        dy = y - yj;
        dz = z - zj;
    }
};

// cubic value and derivative (per knot) by Horner's scheme and its synthetic
// division
__device__ __forceinline__ void spl_both(const Dbl4& c, double p, double& v, double& d) {
    const double b2 = fma(c.w, p, c.z), b1 = fma(b2, p, c.y);
    v = fma(b1, p, c.x);
    d = fma(fma(c.w, p, b2), p, b1);
}

// m = min(floor(q), nr-2), p = min(q - m, 1) of q = r/dr: the integer part of
// a double below 2^20 is the top of its mantissa, cut out and shifted down by
// integer instructions (an FP64 conversion each way holds the FP64 pipe)
__device__ __forceinline__ int knot64_fast(double r, double dr_inv, int mmax, double& p) {
    const double q = r * dr_inv;
    const int hi = __double2hiint(q), ex = (hi >> 20) - 1023;  // q >= 0
    if (ex >= 20) {  // beyond any table
        p = 1.0;
        return mmax;
    }
    const int keep = ex < 0 ? 0 : hi & ~(0xfffff >> ex);
    int m = ex < 0 ? 0 : ((hi & 0xfffff) | 0x100000) >> (20 - ex);
    p = q - __hiloint2double(keep, 0);
    if (m > mmax) {
        m = mmax;
        p = 1.0;
    }
    return m;
}

// 1/sqrt(x): the FP32 reciprocal root of x as a start (its bits converted by
// integer instructions: an FP64 conversion holds the FP64 pipe like an
// addition), then one step of Halley's method, y + y e (1/2 + 3/8 e) with
// e = 1 - x y^2 (|e| < 2^-21, so the next term is below 2^-64).  y^2 of an FP32
// y has 48 bits, so e is as good as exact and the last rounding is the only
// error: measured 0.5000 ulp at most over 78 million x in 1..41, CUDA's rsqrt
// 0.5075 (with e from the rounded x y it was 0.996)
__device__ __forceinline__ double rsqrt_halley(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned f = __float_as_uint(rsqrtf(__uint_as_float(((hi - 0x38000000u) << 3) | (lo >> 29))));
    const double y = __hiloint2double((int)((f >> 3) + 0x38000000u), (int)(f << 29));
    const double e = fma(-x, y * y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// the same where FP32 can start it, else the library's
__device__ __forceinline__ double recip_root(double x) {
    const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
    return bits - 0x3a00000000000000ull < 0x0a00000000000000ull ? rsqrt_halley(x) : rsqrt(x);
}

// sqrt(x) from y = 1/sqrt(x) to an ulp: x y and one step of Newton's method
// for the root, r + (x - r^2) y/2.  The fma leaves the residual exact, so what
// is rounded last lies within 2^-100 of the root: the correctly rounded root
// wherever that decides, in two operations (y/2 and the test for zero are
// integer instructions).  Without the step one density in six came out an ulp off
__device__ __forceinline__ double root_from(double x, double y) {
    const double r = x * y, h = __hiloint2double(__double2hiint(y) - 0x100000, __double2loint(y));
    const double s = fma(fma(-r, r, x), h, r);
    return __double_as_longlong(x) == 0 ? 0.0 : s;
}

// x < y of two non-negative doubles by their bits (NaN is not below)
__device__ __forceinline__ bool below(double x, double y) {
    return (unsigned long long)__double_as_longlong(x) < (unsigned long long)__double_as_longlong(y);
}

struct Smem64 {
    double sh[27][3];
    double cut_sq[kMaxElem * kMaxElem];
    // batch: the shifts n*H of one cell (called by the whole block, after fill)
    __device__ void fill_cell(const CellGeo& g) {
        const double* h = g.h6;  // rows of H: (h0,0,0), (h1,h3,0), (h2,h4,h5)
        for (int t = threadIdx.x; t < 27; t += blockDim.x) {
            const int n0 = t % 3 - 1, n1 = (t / 3) % 3 - 1, n2 = t / 9 - 1;
            sh[t][0] = n0 * h[0] + n1 * h[1] + n2 * h[2];
            sh[t][1] = n1 * h[3] + n2 * h[4];
            sh[t][2] = n2 * h[5];
        }
        __syncthreads();
    }
    __device__ void fill(const EamArgs& a) {
        for (int t = threadIdx.x; t < 27; t += blockDim.x) {
            sh[t][0] = a.shift[t][0];
            sh[t][1] = a.shift[t][1];
            sh[t][2] = a.shift[t][2];
        }
        for (int t = threadIdx.x; t < a.ne * a.ne; t += blockDim.x) cut_sq[t] = a.cut_sq[t];
        __syncthreads();
    }
};

// F(rho), F'(rho) with the reference's extrapolation above rho_max
__device__ __forceinline__ void embed64(const EamArgs& a, int ei, double rho, double& Fv, double& dFv) {
    double p = rho * a.drho_inv;
    int m = p < (double)(a.nrho - 2) ? (int)p : a.nrho - 2;
    if (m < 0) m = 0;
    p -= (double)m;
    p = fmin(p, 1.0);
    Dbl4 c = ldg4(a.F64 + (size_t)ei * a.nrho + m);
    dFv = ((3.0 * c.w * p + 2.0 * c.z) * p + c.y) * a.drho_inv;
    Fv = ((c.w * p + c.z) * p + c.y) * p + c.x;
    if (rho > a.rho_max) Fv += dFv * (rho - a.rho_max);
}

}  // namespace mappg
