// What the FP64 kernels share: positions with their periodic images, the
// shift and cutoff tables of a block, the embedding function.
#pragma once

#include "eam_common.cuh"

namespace mappg {

// atom i's position and the bin-edge flags that turn a bin step into an image
struct Pos64 {
    double x, y, z;
    int lo[3], hi[3];
    __device__ __forceinline__ void load(const EamArgs& a, int i) {
        x = a.x[i];
        y = a.x[a.n + i];
        z = a.x[2 * a.n + i];
        int bc = a.binc[i];
        int b[3] = {bc & 1023, (bc >> 10) & 1023, (bc >> 20) & 1023};
#pragma unroll
        for (int d = 0; d < 3; d++) {
            lo[d] = b[d] == 0;
            hi[d] = b[d] == a.nb[d] - 1;
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

struct Smem64 {
    double sh[27][3];
    double cut_sq[kMaxElem * kMaxElem];
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
