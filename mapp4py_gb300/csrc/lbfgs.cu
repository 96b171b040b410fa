// L-BFGS minimization with back-tracking line search on the device:
// md.min_lbfgs(m,e_tol,max_dx,ls=ls_bt(c,rho,min_alpha)).run(atoms,nsteps).
//
// The iteration is MinLBFGS::__run (min_l-bfgs.h:113-219) over the line-
// search object MinMDHandler<false,true> (min_cg.h:215-309) and
// LineSearchBackTrack::min (ls.h:711-769):
//   x0 = x; h = f0 = f; two-loop recursion over the m most recent (s, y);
//   f.h < 0 -> h = f, history dropped; Armijo back-tracking from
//   alpha = min(max_dx/max|h|, 1); force call; stop on the energy tolerance,
//   on max|F| < f_tol (added), or on the iteration limit; history update
//   s0 = alpha*h, y0 = f0 - f, rho0 = 1/(s0.y0), gamma = s0.y0/(y0.y0).
// All vectors live on the device in the system's SoA layout.  The recursion
// keeps its scalars on the device: each kernel reads the coefficient it
// needs, applies its update and reduces the next dot product in the same
// pass, so the host only reads the line-search energies and f.h.  Dot
// products are FP64 with a fixed reduction order.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "eam_common.cuh"
#include "linesearch.h"

namespace mappg {

void sys_build(mappg_sys* s);
void lb_update(mappg_sys* s);

// device scalars of the recursion (one block of doubles)
struct LbScal {
    double dot[2 * 64 + 8];  // dot products, one slot per use
    double rho[64];
    double alpha[64];
    double gamma;
    double fh, hh, hmax, fmax;
    double tau;    // scale of the learned diagonal, (s.y)/(y.P.y)
    double dxmax;  // max |x - x_build| component (list validity of line-search trials)
    unsigned long long dxbits;  // the same by k_lb_dxmax (bits of a non-negative double)
};

constexpr int kLbU = 4;  // components a thread of the vector kernels loads at a time

// One step of the two-loop recursion, by MODE, then dot = s.h for the next
// one (s null: none).  Coefficients are read from the device:
//   kLbStart   h = f, and the iteration's start x0 = x, f0 = f
//   kLbFirst   alpha_i = -rho_i*dot_in, stored; h += alpha_i*y
//   kLbLast    kLbFirst, then the initial inverse Hessian (kLbH0)
//   kLbH0      h *= gamma; with P, the learned diagonal, h *= tau*P
//              elementwise (tau: its scale from the newest pair)
//   kLbSecond  h += (-alpha_i - rho_i*dot_in)*y
// A step is launch, the vectors' traffic and the last block's sum; the start
// and the scaling had launches of their own before (9.5 us each for 759,000
// components).
enum LbMode { kLbStart, kLbFirst, kLbLast, kLbH0, kLbSecond };
struct LbVec {
    int N;
    const double *x, *f;
    double *xs, *f0, *h;
    const double* P;
};
template <int MODE>
__global__ void __launch_bounds__(256) k_lb_step(LbVec a, const double* __restrict__ y, const double* __restrict__ s,
                                                 LbScal* L, int idx, int dot_in, int dot_out, double* partials,
                                                 unsigned* counter) {
    dep_wait();
    const int N = a.N;
    double coef = 0.0;
    if (MODE == kLbFirst || MODE == kLbLast) {
        coef = -L->rho[idx] * L->dot[dot_in];
        if (blockIdx.x == 0 && threadIdx.x == 0) L->alpha[idx] = coef;
    } else if (MODE == kLbSecond) {
        coef = -L->alpha[idx] - L->rho[idx] * L->dot[dot_in];
    }
    constexpr bool AXPY = MODE == kLbFirst || MODE == kLbLast || MODE == kLbSecond;
    constexpr bool H0 = MODE == kLbLast || MODE == kLbH0;
    const double gamma = H0 ? L->gamma : 0.0, tau = H0 ? L->tau : 0.0;
    double acc = 0.0;
    // kLbU components in flight per thread: their loads are issued together
    // (a thread has ~10 components in all, so the pass is load latency);
    // the products are added in component order
    const int stride = gridDim.x * blockDim.x;
    for (int q0 = blockIdx.x * blockDim.x + threadIdx.x; q0 < N; q0 += kLbU * stride) {
        double hv[kLbU], yv[kLbU], sv[kLbU], xv[kLbU];
#pragma unroll
        for (int u = 0; u < kLbU; u++) {
            const int q = q0 + u * stride;
            const bool in = q < N;
            hv[u] = in ? (MODE == kLbStart ? a.f[q] : a.h[q]) : 0.0;
            yv[u] = in && AXPY ? y[q] : 0.0;
            sv[u] = in && s ? s[q] : 0.0;
            xv[u] = !in ? 0.0 : MODE == kLbStart ? a.x[q] : H0 && a.P ? a.P[q] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kLbU; u++) {
            const int q = q0 + u * stride;
            if (q >= N) break;
            if (MODE == kLbStart) {
                a.xs[q] = xv[u];
                a.f0[q] = hv[u];
            }
            if (AXPY) hv[u] = hv[u] + coef * yv[u];
            if (H0) hv[u] = a.P ? hv[u] * (tau * xv[u]) : hv[u] * gamma;
            a.h[q] = hv[u];
            if (s) acc += sv[u] * hv[u];
        }
    }
    if (!s) return;
    double v[1] = {acc};
    __shared__ double t[1];
    if (block_partials<1, true>(v, partials, 0, counter)) {
        final_sums_ordered<1>(partials, gridDim.x, t);
        if (threadIdx.x == 0) {
            L->dot[dot_out] = t[0];
            *counter = 0;
        }
    }
}

// dots f.h, h.h and max|h| (line-search preparation) and max|f|; with x
// and xb (the neighbour list's build positions) also max|x - xb| over
// components
__global__ void __launch_bounds__(256) k_lb_prep(int N, const double* __restrict__ f, const double* __restrict__ h,
                                                 const double* __restrict__ x, const double* __restrict__ xb,
                                                 LbScal* L, double* partials, unsigned* counter) {
    dep_wait();
    double v[2] = {0.0, 0.0};
    unsigned long long mx[4] = {0, 0, 0, 0};  // bits of the maxima (integer compares; FP64 ones are slow here)
    const int stride = gridDim.x * blockDim.x;
    for (int q0 = blockIdx.x * blockDim.x + threadIdx.x; q0 < N; q0 += kLbU * stride) {
        double hv[kLbU], fv[kLbU], dx[kLbU];
#pragma unroll
        for (int u = 0; u < kLbU; u++) {
            const int q = q0 + u * stride;
            const bool in = q < N;
            hv[u] = in ? h[q] : 0.0;
            fv[u] = in ? f[q] : 0.0;
            dx[u] = in && x ? x[q] - xb[q] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kLbU; u++) {
            v[0] += fv[u] * hv[u];
            v[1] += hv[u] * hv[u];
            mx[0] = RedMaxBits()(mx[0], bits_of_abs(hv[u]));
            mx[1] = RedMaxBits()(mx[1], bits_of_abs(fv[u]));
            mx[2] = RedMaxBits()(mx[2], bits_of_abs(dx[u]));
        }
    }
    // maxima into slots 2,3,4 of the partial row that takes the sums
    __shared__ unsigned long long redm[32][4];
    __shared__ double tot[2];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const unsigned long long m = warp_reduce(mx, RedMaxBits());
    if (lane % 8 == 0) redm[w][lane / 8] = m;
    __syncthreads();
    if (threadIdx.x < 3) {
        unsigned long long r = 0;
        for (int q = 0; q < nw; q++) r = RedMaxBits()(r, redm[q][threadIdx.x]);
        partials[blockIdx.x * kRedSlots + 2 + threadIdx.x] = __longlong_as_double((long long)r);
    }
    if (block_partials<2, true>(v, partials, 0, counter)) {
        final_sums_ordered<2>(partials, gridDim.x, tot);
        unsigned long long b[4] = {0, 0, 0, 0};
        for (int bb = threadIdx.x; bb < (int)gridDim.x; bb += blockDim.x)
#pragma unroll
            for (int k = 0; k < 3; k++)
                b[k] = RedMaxBits()(b[k], (unsigned long long)__double_as_longlong(
                                              __ldcg(partials + bb * kRedSlots + 2 + k)));
        const unsigned long long t = warp_reduce(b, RedMaxBits());
        if (lane % 8 == 0) redm[w][lane / 8] = t;
        __syncthreads();
        if (threadIdx.x == 0) {
            double m3[3];
            for (int k = 0; k < 3; k++) {
                unsigned long long r = 0;
                for (int q = 0; q < nw; q++) r = RedMaxBits()(r, redm[q][k]);
                m3[k] = __longlong_as_double((long long)r);
            }
            L->fh = tot[0];
            L->hh = tot[1];
            L->hmax = m3[0];
            L->fmax = m3[1];
            L->dxmax = m3[2];
            *counter = 0;
        }
    }
}

// max|f| alone, into L->fmax (set to zero before): what the tolerance after
// a force call needs of k_lb_prep (21 us for 759,000 components, 5 this way)
__global__ void __launch_bounds__(256) k_lb_fmax(int N, const double* __restrict__ f, LbScal* L) {
    dep_wait();
    unsigned long long m = 0;
    const int stride = gridDim.x * blockDim.x;
    for (int q0 = blockIdx.x * blockDim.x + threadIdx.x; q0 < N; q0 += kLbU * stride) {
        double fv[kLbU];
#pragma unroll
        for (int u = 0; u < kLbU; u++) fv[u] = q0 + u * stride < N ? f[q0 + u * stride] : 0.0;
#pragma unroll
        for (int u = 0; u < kLbU; u++) m = RedMaxBits()(m, bits_of_abs(fv[u]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = RedMaxBits()(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ unsigned long long red[8];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 8) {
        m = red[threadIdx.x];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) m = RedMaxBits()(m, __shfl_xor_sync(0xffu, m, o));
        if (threadIdx.x == 0) atomicMax((unsigned long long*)&L->fmax, m);
    }
}

// max |x - xb| over components into *out (the bits of a non-negative double
// order as the values do, so an integer maximum of the bits is the maximum)
__global__ void k_lb_dxmax(int N, const double* __restrict__ x, const double* __restrict__ xb,
                           unsigned long long* out) {
    dep_wait();
    double m = 0.0;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < N; q += gridDim.x * blockDim.x)
        m = fmax(m, fabs(x[q] - xb[q]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

// the search direction as one float4 per atom (Cartesian) for k_de32
__global__ void k_lb_h32(int n, const double* __restrict__ h, float4* __restrict__ h32) {
    dep_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        h32[i] = make_float4((float)h[i], (float)h[n + i], (float)h[2 * n + i], 0.f);
}

// x = x0 + alpha*h  (MinMDHandler::F, min_cg.h:260-267)
__global__ void k_lb_trial(int N, double* __restrict__ x, const double* __restrict__ x0, const double* __restrict__ h,
                           double alpha) {
    dep_wait();
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < N; q += gridDim.x * blockDim.x)
        x[q] = x0[q] + alpha * h[q];
}

// s0 = alpha*h, y0 = f0 - f; dots s0.y0, y0.y0 -> rho0, gamma (and y0.P.y0
// -> tau with a learned diagonal).  A pair without positive curvature
// (s0.y0 <= 0, e.g. a step that underflowed to zero) gets rho0 = 0, so it
// takes no part in the recursion, and leaves gamma as it was; the
// reference would divide by it.
__global__ void __launch_bounds__(256) k_lb_hist(int N, double* __restrict__ s0, double* __restrict__ y0,
                                                 const double* __restrict__ h, const double* __restrict__ f0,
                                                 const double* __restrict__ f, const double* __restrict__ P,
                                                 double alpha, LbScal* L, double* partials, unsigned* counter) {
    dep_wait();
    double v[3] = {0.0, 0.0, 0.0};
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < N; q += gridDim.x * blockDim.x) {
        double sv = alpha * h[q];
        double yv = f0[q] - f[q];
        s0[q] = sv;
        y0[q] = yv;
        v[0] += sv * yv;
        v[1] += yv * yv;
        if (P) v[2] += yv * yv * P[q];
    }
    __shared__ double t[3];
    if (block_partials<3, true>(v, partials, 0, counter)) {
        final_sums_ordered<3>(partials, gridDim.x, t);
        if (threadIdx.x == 0) {
            if (t[0] > 0.0 && t[1] > 0.0) {
                L->gamma = t[0] / t[1];
                L->rho[0] = 1.0 / t[0];
                if (t[2] > 0.0) L->tau = t[0] / t[2];
            } else {
                L->rho[0] = 0.0;
            }
            *counter = 0;
        }
    }
}

__global__ void k_lb_shift_rho(LbScal* L, int m) {
    dep_wait();
    for (int i = m - 1; i > 0; i--) L->rho[i] = L->rho[i - 1];
}

// x0 = x, f0 = f: the start of an iteration of the conjugate gradients
__global__ void k_lb_start(int N, const double* __restrict__ x, const double* __restrict__ f, double* __restrict__ xs,
                           double* __restrict__ f0) {
    dep_wait();
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < N; q += gridDim.x * blockDim.x) {
        xs[q] = x[q];
        f0[q] = f[q];
    }
}

void launch_energy64(mappg_sys* s);  // eam.cu
void launch_de32(mappg_sys* s, double alpha);  // eam32.cu

// what the host reads of a pass: the device scalars with the capacity flag
// of the list check before it, and the vector kernels' results
struct LbRead {
    DevScalars sc;
    double prep[6];  // f.h, h.h, max|h|, max|f|, tau, max|x - x_build|
};
static_assert(sizeof(LbRead) <= 4096, "the landing place holds 4 KB");

static LbRead* lb_read(mappg_sys* s, const LbScal* L) {
    LbRead* r = (LbRead*)sys_landing(s);
    MAPPG_CUDA(cudaMemcpyAsync(&r->sc, s->sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, s->stream));
    if (L) MAPPG_CUDA(cudaMemcpyAsync(r->prep, &L->fh, sizeof(r->prep), cudaMemcpyDeviceToHost, s->stream));
    MAPPG_CUDA(cudaStreamSynchronize(s->stream));
    return r;
}

__global__ void k_clear_rebuild(DevScalars* sc) {
    dep_wait();
    sc->rebuild = 0;
}

// skin test and (gated) rebuild; the caller reads sc->overflow with what it
// runs next: a relaxation can crowd atoms beyond the rows' capacity, and a
// rebuild that ran out of room is redone with wider rows (sys_build)
static void lb_update_launch(mappg_sys* s) {
    launch_dep(s->stream, k_clear_rebuild, 1, 1, 0, s->sc);
    launch_skin_test(s);
    launch_rebuild_chain(s);
    // positions moved without a rebuild: refresh the mixed kernels' frame
    if (s->precision == MAPPG_MIXED) launch_shadow(s);
    MAPPG_CUDA(cudaGetLastError());
}

void lb_update(mappg_sys* s) {
    lb_update_launch(s);
    if (lb_read(s, nullptr)->sc.overflow) sys_build(s);
}

// list check, then the energy by `launch`, one read for both
template <class F>
static double lb_checked_energy(mappg_sys* s, F launch) {
    lb_update_launch(s);
    launch(s);
    const LbRead* r = lb_read(s, nullptr);
    if (r->sc.overflow) {
        sys_build(s);
        launch(s);
        r = lb_read(s, nullptr);
    }
    return r->sc.energy;
}

static double lb_energy(mappg_sys* s) {
    // mixed systems compare FP64 line-search energies, so FP32 rounding of
    // the pair terms does not decide the Armijo test near convergence
    return lb_checked_energy(s, s->precision == MAPPG_MIXED ? launch_energy64 : launch_energy);
}

static void lb_force(mappg_sys* s, double* pe) {
    launch_force(s);
    sync_forces64(s);
    *pe = lb_read(s, nullptr)->sc.energy;
}

// The caller's function after an iteration's force call, where the
// reference writes its periodic export (ExportHandler::print, min.h:216-220)
void iteration_hook(mappg_sys* s, int istep) {
    if (!s->hook || s->hook_every <= 0 || (istep + 1) % s->hook_every != 0) return;
    MAPPG_CUDA(cudaStreamSynchronize(s->stream));
    if (s->hook(s->hook_user, (long long)istep + 1) != 0)
        throw Error{MAPPG_ERR_ARG, "the iteration hook stopped the run"};
}

// The minimizers' line-search function (MinMDHandler::F and F_reset,
// min_cg.h:260-276): a trial moves x to x0 + alpha h and evaluates the
// energy; reset restores x0.  Trial energies by mode:
//   E64      the FP64 energy (FP64 systems; mixed systems on FP64 forces)
//   DELTA    e0 + dE, dE from the energy-difference pass (launch_de32) on
//            x0's rows and frame positions; no skin test or rebuild (the
//            caller has checked that every trial stays within the skin)
//   E32DIFF  e0 + (E32(trial) - E32(x0)) with the skin test and rebuilds:
//            searches whose first step is too long for DELTA, where the
//            energy changes are large next to the FP32 rounding
struct TrialLine {
    enum Mode { E64, DELTA, E32DIFF };
    mappg_sys* s;
    int N, grid;
    const double* xs;  // x0
    const double* h;
    long long* n_en;
    LbScal* L;
    Mode mode = E64;
    double e0 = 0.0;     // energy of x0 (DELTA, E32DIFF)
    double e0_32 = 0.0;  // FP32 energy of x0 (E32DIFF)
    double hmax = 0.0;   // max |h_c| of the direction
    double F(double a) {
        // an E32DIFF search whose trials have become short goes over to
        // energy differences (FP32 differences would drown in rounding)
        if (mode == E32DIFF && 1.7320508075688772 * a * hmax < 0.25 * s->skin) to_delta(a);
        launch_dep(s->stream, k_lb_trial, grid, 256, 0, N, s->x, xs, h, a);
        (*n_en)++;
        if (mode == E64) return lb_energy(s);
        if (mode == DELTA) {
            launch_de32(s, a);
            return e0 + lb_read(s, nullptr)->sc.de;
        }
        return e0 + (energy32(s) - e0_32);
    }
    void reset() {
        MAPPG_CUDA(cudaMemcpyAsync(s->x, xs, sizeof(double) * N, cudaMemcpyDeviceToDevice, s->stream));
        if (mode != DELTA) lb_update(s);
    }
    // back at x0 with a list around it; DELTA when the trial of step a then
    // stays within half the skin
    void to_delta(double a) {
        MAPPG_CUDA(cudaMemcpyAsync(s->x, xs, sizeof(double) * N, cudaMemcpyDeviceToDevice, s->stream));
        lb_update(s);
        MAPPG_CUDA(cudaMemsetAsync(&L->dxbits, 0, sizeof(unsigned long long), s->stream));
        launch_dep(s->stream, k_lb_dxmax, grid, 256, 0, N, s->x, s->x0, &L->dxbits);
        unsigned long long bits = 0;
        MAPPG_CUDA(cudaMemcpyAsync(&bits, &L->dxbits, sizeof(bits), cudaMemcpyDeviceToHost, s->stream));
        MAPPG_CUDA(cudaStreamSynchronize(s->stream));
        double dx;
        memcpy(&dx, &bits, sizeof(dx));
        if (1.7320508075688772 * (a * hmax + dx) < 0.5 * s->skin) mode = DELTA;
    }
    // skin test, gated rebuild, then the FP32 energy
    static double energy32(mappg_sys* s) { return lb_checked_energy(s, launch_energy); }
};

// grid of the FP64 vector kernels with grid-wide sums: two blocks per SM, so
// that each thread adds up N / (2 x SMs x 256) components (~10 for 250,000
// atoms) before the block and last-block reductions, whose FP64 shuffle
// trees would otherwise cost more than the components themselves (the order
// stays fixed for a given N)
static int lb_grid(mappg_sys* s, int N) { return std::max(1, std::min((N + 255) / 256, 2 * s->sm_count)); }

// a mixed-precision search that fails may be FP32 force noise, not a minimum
static bool ls_failed(int err) { return err == LS_MIN_ALPHA || err == B_F_DOWNHILL; }

void lbfgs_run(mappg_sys* s, int m, double e_tol, double max_dx, double f_tol, const LsParams& ls, int nsteps,
               double* stats, const double* P, long long* n_fallback) {
    if (m < 0 || m > 64) throw Error{MAPPG_ERR_ARG, "m must be in 0..64"};
    if (!(max_dx > 0.0)) throw Error{MAPPG_ERR_ARG, "max_dx must be positive"};
    if (!(e_tol >= 0.0)) throw Error{MAPPG_ERR_ARG, "e_tol must be >= 0"};
    if (nsteps < 0) throw Error{MAPPG_ERR_ARG, "nsteps must be >= 0"};
    const int N = 3 * s->n;
    const int grid = lb_grid(s, N);
    const bool mixed = s->precision == MAPPG_MIXED;
    Work work(s);
    work.reserve((3 + 2 * (size_t)m) * Work::room<double>(N) + Work::room<LbScal>(1) + Work::room<unsigned>(4) +
                 (mixed ? Work::room<float4>(s->n) : 0));
    double* f0 = work.take<double>(N);
    double* h = work.take<double>(N);
    double* xs = work.take<double>(N);
    std::vector<double*> sv(m), yv(m);
    for (int i = 0; i < m; i++) {
        sv[i] = work.take<double>(N);
        yv[i] = work.take<double>(N);
    }
    LbScal* L = work.take<LbScal>(1);
    unsigned* counter = work.take<unsigned>(4);
    MAPPG_CUDA(cudaMemsetAsync(L, 0, sizeof(LbScal), s->stream));
    MAPPG_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned) * 4, s->stream));
    const double one = 1.0;  // gamma starts at 1 (min_l-bfgs.h:140), as does tau
    MAPPG_CUDA(cudaMemcpyAsync(&L->gamma, &one, sizeof(double), cudaMemcpyHostToDevice, s->stream));
    MAPPG_CUDA(cudaMemcpyAsync(&L->tau, &one, sizeof(double), cudaMemcpyHostToDevice, s->stream));
    // a mixed relaxation that stalls above f_tol (its FP32 forces no longer
    // point downhill on the FP64 energy) goes on with FP64 forces
    struct Promote {
        mappg_sys* s;
        ~Promote() { s->force64 = false; }
    } promote{s};
    cudaStream_t st = s->stream;
    double* part = s->partials;
    // mixed systems: line-search trials inside the skin take energy
    // differences (TrialLine delta mode), which need x0's FP64 density and
    // the direction as float4
    struct KeepRho {
        mappg_sys* s;
        ~KeepRho() {
            s->keep_rho64 = false;
            s->h32 = nullptr;
        }
    } keep_rho{s};
    if (mixed) {
        s->keep_rho64 = true;
        s->h32 = work.take<float4>(s->n);
    }

    // NewDynamicMD::init then the opening force call
    sys_build(s);
    long long n_en = 0, n_fc = 1;
    double e_curr, pe_force;
    lb_force(s, &pe_force);
    // the line search's reference energy is an FP64 energy in both modes
    e_curr = s->precision == MAPPG_MIXED ? lb_energy(s) : pe_force;
    double e_prev, alpha_m = 0.0;
    int k = 0;
    int err = nsteps == 0 ? MIN_F_MAX_ITER : LS_S;
    double dxmax = 0.0;
    auto read_prep = [&](double* fh, double* hh, double* hmax, double* fmax_) {
        launch_dep(st, k_lb_prep, grid, 256, 0, N, s->f, h, s->x, s->x0, L, part, counter);
        const LbRead* r = lb_read(s, L);
        *fh = r->prep[0];
        *hh = r->prep[1];
        *hmax = r->prep[2];
        *fmax_ = r->prep[3];
        dxmax = r->prep[5];
        return r;
    };
    double fh, hh, hmax, fmaxv;
    auto read_fmax = [&]() -> const LbRead* {
        MAPPG_CUDA(cudaMemsetAsync(&L->fmax, 0, sizeof(double), st));
        launch_dep(st, k_lb_fmax, grid, 256, 0, N, s->f, L);
        const LbRead* r = lb_read(s, L);
        fmaxv = r->prep[3];
        return r;
    };
    if (err == LS_S && f_tol > 0.0) {
        MAPPG_CUDA(cudaMemcpyAsync(h, s->f, sizeof(double) * N, cudaMemcpyDeviceToDevice, st));
        read_prep(&fh, &hh, &hmax, &fmaxv);
        if (fmaxv < f_tol) err = MIN_S_FTOL;
    }
    // the two-loop recursion (min_l-bfgs.h:148-170) with the initial inverse
    // Hessian gamma*I, or diag(P) when a learned preconditioner is given
    auto two_loop = [&](bool diag) {
        const LbVec V = {N, s->x, s->f, xs, f0, h, diag ? P : nullptr};
        auto step = [&](auto kern, const double* y, const double* next, int i, int in, int out) {
            launch_dep(st, kern, grid, 256, 0, V, y, next, L, i, in, out, part, counter);
        };
        step(k_lb_step<kLbStart>, nullptr, k > 0 ? sv[0] : nullptr, 0, 0, 0);
        // first loop: alpha_i = -rho_i (s_i.h); h += alpha_i y_i; its last
        // step applies H0 and takes the second loop's first dot, y_{k-1}.h
        for (int i = 0; i + 1 < k; i++) step(k_lb_step<kLbFirst>, yv[i], sv[i + 1], i, i, i + 1);
        if (k > 0)
            step(k_lb_step<kLbLast>, yv[k - 1], yv[k - 1], k - 1, k - 1, 64);
        else
            step(k_lb_step<kLbH0>, nullptr, nullptr, 0, 0, 64);
        for (int i = k - 1; i > -1; i--)
            step(k_lb_step<kLbSecond>, sv[i], i > 0 ? yv[i - 1] : nullptr, i, 64 + (k - 1 - i), 64 + (k - i));
        MAPPG_CUDA(cudaGetLastError());
    };
    TrialLine line{s, N, grid, xs, h, &n_en, L};
    LineSearch<TrialLine> search(ls, line);
    int istep = 0;
    for (; err == LS_S; istep++) {
        if (P && s->precond_every > 0 && istep > 0 && istep % s->precond_every == 0) s->precond_refresh();
        two_loop(P != nullptr);
        e_prev = e_curr;
        read_prep(&fh, &hh, &hmax, &fmaxv);
        if (P && fh < 0.0) {
            // a non-descent preconditioned direction: plain L-BFGS instead
            if (n_fallback) (*n_fallback)++;
            two_loop(false);
            read_prep(&fh, &hh, &hmax, &fmaxv);
        }
        if (fh < 0.0) {
            MAPPG_CUDA(cudaMemcpyAsync(h, s->f, sizeof(double) * N, cudaMemcpyDeviceToDevice, st));
            k = 0;
            read_prep(&fh, &hh, &hmax, &fmaxv);
        }
        // ls->min(&handler, e_curr, alpha_m, 0) (min_l-bfgs.h:173)
        double dfa = -fh, max_a;
        int lerr = LS_S;
        if (hh == 0.0) {
            max_a = 0.0;
            dfa = 0.0;
        } else if (dfa >= 0.0) {
            max_a = 0.0;
            dfa = 1.0;
        } else {
            max_a = fabs(max_dx / hmax);
        }
        // mixed: trials that keep every atom within half the skin of the
        // list's build positions (the first, largest trial moves an atom by
        // at most sqrt(3) alpha max|h_c|) take energy differences on x0's
        // list; longer searches take differences of FP32 energies
        line.mode = TrialLine::E64;
        if (mixed && !s->force64 && dfa < 0.0 && max_a > 0.0) {
            line.e0 = e_curr;
            line.hmax = hmax;
            launch_dep(st, k_lb_h32, grid_for(s, s->n, 256), 256, 0, s->n, h, s->h32);
            MAPPG_CUDA(cudaGetLastError());
            const double a1 = std::min(max_a, 1.0);
            if (1.7320508075688772 * (a1 * hmax + dxmax) < 0.5 * s->skin) {
                line.mode = TrialLine::DELTA;
            } else {
                // the FP32 energy of x0 is the last force call's: the same
                // pair terms and compensated sums as the trials' energy pass
                line.mode = TrialLine::E32DIFF;
                line.e0_32 = pe_force;
            }
        }
        if (dfa == 0.0)
            lerr = LS_F_GRAD0;
        else if (max_a == 0.0)
            lerr = LS_MIN_ALPHA;
        else if (dfa >= 0.0)
            lerr = LS_F_DOWNHILL;
        else
            lerr = search.min(dfa, max_a, e_curr, alpha_m, 0);
        err = lerr;
        // after a DELTA search: the accepted (or restored) positions' skin
        // test, and the FP32 frame positions the force call reads
        const bool moved = line.mode == TrialLine::DELTA;
        if (moved) lb_update_launch(s);
        if (moved && err != LS_S && lb_read(s, nullptr)->sc.overflow) sys_build(s);
        if (ls_failed(err) && s->precision == MAPPG_MIXED && !s->force64 && f_tol > 0.0) {
            s->force64 = true;
            lb_force(s, &pe_force);
            n_fc++;
            e_curr = lb_energy(s);
            k = 0;
            MAPPG_CUDA(cudaMemcpyAsync(&L->gamma, &one, sizeof(double), cudaMemcpyHostToDevice, st));
            MAPPG_CUDA(cudaMemcpyAsync(&L->tau, &one, sizeof(double), cudaMemcpyHostToDevice, st));
            err = LS_S;
            istep--;
            continue;
        }
        if (err != LS_S) {
            istep--;
            continue;
        }
        // handler.force_calc(): forces and atoms->pe; e_curr stays the line
        // search's energy, as in min_l-bfgs.h:181-188.  max|F| and the energy
        // come back in one read, with the capacity flag of the list check
        // (max|F| after the caller's function where there is one: it may
        // change the system)
        auto force = [&] {
            launch_force(s);
            sync_forces64(s);
            return f_tol > 0.0 && !s->hook ? read_fmax() : lb_read(s, nullptr);
        };
        const LbRead* r = force();
        if (moved && r->sc.overflow) {
            sys_build(s);
            r = force();
        }
        pe_force = r->sc.energy;
        n_fc++;
        iteration_hook(s, istep);
        if (e_prev - e_curr < e_tol) err = MIN_S_TOLERANCE;
        if (f_tol > 0.0 && s->hook) read_fmax();
        if (f_tol > 0.0 && fmaxv < f_tol) err = MIN_S_FTOL;
        if (istep + 1 == nsteps) err = MIN_F_MAX_ITER;
        if (err) continue;
        if (m) {
            if (k != m) k++;
            double* ts = sv[k - 1];
            double* ty = yv[k - 1];
            for (int i = k - 1; i > 0; i--) {
                sv[i] = sv[i - 1];
                yv[i] = yv[i - 1];
            }
            sv[0] = ts;
            yv[0] = ty;
            launch_dep(st, k_lb_shift_rho, 1, 1, 0, L, m);
            launch_dep(st, k_lb_hist, grid, 256, 0, N, sv[0], yv[0], h, f0, s->f, P, alpha_m, L, part, counter);
            MAPPG_CUDA(cudaGetLastError());
        } else {
            // gamma = alpha_m (h.f0 - h.f)/(f.f + f0.f0 - 2 f.f0) on the host
            std::vector<double> hv(N), fv(N), f0v(N);
            MAPPG_CUDA(cudaMemcpyAsync(hv.data(), h, sizeof(double) * N, cudaMemcpyDeviceToHost, st));
            MAPPG_CUDA(cudaMemcpyAsync(fv.data(), s->f, sizeof(double) * N, cudaMemcpyDeviceToHost, st));
            MAPPG_CUDA(cudaMemcpyAsync(f0v.data(), f0, sizeof(double) * N, cudaMemcpyDeviceToHost, st));
            MAPPG_CUDA(cudaStreamSynchronize(st));
            double hf0 = 0, hf = 0, ff = 0, f0f0 = 0, ff0 = 0;
            for (int q = 0; q < N; q++) {
                hf0 += hv[q] * f0v[q];
                hf += hv[q] * fv[q];
                ff += fv[q] * fv[q];
                f0f0 += f0v[q] * f0v[q];
                ff0 += fv[q] * f0v[q];
            }
            double g = alpha_m * (hf0 - hf) / (ff + f0f0 - 2.0 * ff0);
            MAPPG_CUDA(cudaMemcpyAsync(&L->gamma, &g, sizeof(double), cudaMemcpyHostToDevice, st));
        }
    }
    if (f_tol <= 0.0 || err != MIN_S_FTOL) {
        MAPPG_CUDA(cudaMemcpyAsync(h, s->f, sizeof(double) * N, cudaMemcpyDeviceToDevice, st));
        read_prep(&fh, &hh, &hmax, &fmaxv);
    }
    DevScalars hs;
    MAPPG_CUDA(cudaMemcpyAsync(&hs, s->sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, st));
    MAPPG_CUDA(cudaStreamSynchronize(st));
    if (hs.overflow) throw Error{MAPPG_ERR_NBR, "neighbour list capacity exceeded during minimization"};
    if (hs.bad) throw Error{MAPPG_ERR_NAN, "non-finite value during minimization"};
    if (stats) {
        stats[0] = istep;
        stats[1] = pe_force;
        stats[2] = fmaxv;
        stats[3] = err;
        stats[4] = (double)n_en;
        stats[5] = (double)n_fc;
    }
}

}  // namespace mappg

// ------------------------------------------------------------------ MinCG
// md.min_cg(e_tol,max_dx,ls=ls_bt(...)).run(atoms,nsteps): MinCG::__run
// (min_cg.h:454-536), Polak-Ribiere directions h = ratio h + f with ratio =
// (f.f - f.f0)/(f0.f0), over LineSearchBackTrack::min with init_flag 1
// (ls.h:711-769: the first trial step is capped by -prev/dfa, prev being
// the previous step's decrease -dfa*alpha; LineSearch::reset, ls.h:42,
// starts prev at -1).  Same vectors and kernels as the L-BFGS driver.
namespace mappg {

// f.f and f.f0 into L->dot[0], L->dot[1]
__global__ void __launch_bounds__(256) k_cg_dots(int N, const double* __restrict__ f, const double* __restrict__ f0,
                                                 LbScal* L, double* partials, unsigned* counter) {
    dep_wait();
    double v[2] = {0.0, 0.0};
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < N; q += gridDim.x * blockDim.x) {
        v[0] += f[q] * f[q];
        v[1] += f[q] * f0[q];
    }
    __shared__ double t[2];
    if (block_partials<2, true>(v, partials, 0, counter)) {
        final_sums_ordered<2>(partials, gridDim.x, t);
        if (threadIdx.x == 0) {
            L->dot[0] = t[0];
            L->dot[1] = t[1];
            *counter = 0;
        }
    }
}

__global__ void k_cg_dir(int N, double* __restrict__ h, const double* __restrict__ f, double ratio) {
    dep_wait();
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < N; q += gridDim.x * blockDim.x) h[q] = ratio * h[q] + f[q];
}

void cg_run(mappg_sys* s, double e_tol, double max_dx, double f_tol, const LsParams& ls, int nsteps, double* stats) {
    if (!(max_dx > 0.0)) throw Error{MAPPG_ERR_ARG, "max_dx must be positive"};
    if (!(e_tol >= 0.0)) throw Error{MAPPG_ERR_ARG, "e_tol must be >= 0"};
    if (nsteps < 0) throw Error{MAPPG_ERR_ARG, "nsteps must be >= 0"};
    const int N = 3 * s->n;
    const int grid = lb_grid(s, N);
    Work work(s);
    work.reserve(3 * Work::room<double>(N) + Work::room<LbScal>(1) + Work::room<unsigned>(4));
    double* f0 = work.take<double>(N);
    double* h = work.take<double>(N);
    double* xs = work.take<double>(N);
    LbScal* L = work.take<LbScal>(1);
    unsigned* counter = work.take<unsigned>(4);
    cudaStream_t st = s->stream;
    MAPPG_CUDA(cudaMemsetAsync(L, 0, sizeof(LbScal), st));
    MAPPG_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned) * 4, st));
    double* part = s->partials;
    double dxmax = 0.0;
    auto read_prep = [&](double* fh, double* hh, double* hmax, double* fmax_) {
        launch_dep(st, k_lb_prep, grid, 256, 0, N, s->f, h, s->x, s->x0, L, part, counter);
        const LbRead* r = lb_read(s, L);
        *fh = r->prep[0];
        *hh = r->prep[1];
        *hmax = r->prep[2];
        *fmax_ = r->prep[3];
        dxmax = r->prep[5];
    };
    sys_build(s);
    long long n_en = 0, n_fc = 1;
    double pe_force;
    lb_force(s, &pe_force);
    double e_curr = s->precision == MAPPG_MIXED ? lb_energy(s) : pe_force, e_prev;
    int err = nsteps == 0 ? MIN_F_MAX_ITER : LS_S;
    double fh, hh, hmax, fmaxv;
    MAPPG_CUDA(cudaMemcpyAsync(h, s->f, sizeof(double) * N, cudaMemcpyDeviceToDevice, st));
    read_prep(&fh, &hh, &hmax, &fmaxv);
    if (err == LS_S && f_tol > 0.0 && fmaxv < f_tol) err = MIN_S_FTOL;
    double f0_f0 = fh;  // f.f with h = f
    TrialLine line{s, N, grid, xs, h, &n_en, L};
    LineSearch<TrialLine> search(ls, line);  // prev_val starts at -1 (LineSearch::reset)
    double alpha = 0.0;
    struct Promote {
        mappg_sys* s;
        ~Promote() { s->force64 = false; }
    } promote{s};
    int istep = 0;
    for (; err == LS_S; istep++) {
        if (f0_f0 == 0.0) {
            err = LS_F_GRAD0;
            continue;
        }
        launch_dep(st, k_lb_start, grid_for(s, N, 256), 256, 0, N, s->x, s->f, xs, f0);
        e_prev = e_curr;
        read_prep(&fh, &hh, &hmax, &fmaxv);
        if (fh < 0.0) {
            MAPPG_CUDA(cudaMemcpyAsync(h, s->f, sizeof(double) * N, cudaMemcpyDeviceToDevice, st));
            read_prep(&fh, &hh, &hmax, &fmaxv);
            fh = f0_f0;
        }
        double dfa = -fh, max_a;
        int lerr = LS_S;
        if (hh == 0.0) {
            max_a = 0.0;
            dfa = 0.0;
        } else if (dfa >= 0.0) {
            max_a = 0.0;
            dfa = 1.0;
        } else {
            max_a = fabs(max_dx / hmax);
        }
        if (dfa == 0.0)
            lerr = LS_F_GRAD0;
        else if (max_a == 0.0)
            lerr = LS_MIN_ALPHA;
        else if (dfa >= 0.0)
            lerr = LS_F_DOWNHILL;
        else
            lerr = search.min(dfa, max_a, e_curr, alpha, 1);  // init_flag 1 (min_cg.h:504)
        err = lerr;
        if (ls_failed(err) && s->precision == MAPPG_MIXED && !s->force64 && f_tol > 0.0) {
            // stalled on FP32 forces above f_tol: restart from x0 with FP64 forces
            s->force64 = true;
            lb_force(s, &pe_force);
            n_fc++;
            e_curr = lb_energy(s);
            MAPPG_CUDA(cudaMemcpyAsync(h, s->f, sizeof(double) * N, cudaMemcpyDeviceToDevice, st));
            read_prep(&fh, &hh, &hmax, &fmaxv);
            f0_f0 = fh;
            search.prev_val = -1.0;
            err = LS_S;
            istep--;
            continue;
        }
        if (err != LS_S) {
            istep--;
            continue;
        }
        lb_force(s, &pe_force);
        n_fc++;
        iteration_hook(s, istep);
        if (e_prev - e_curr < e_tol) err = MIN_S_TOLERANCE;
        if (f_tol > 0.0) {
            read_prep(&fh, &hh, &hmax, &fmaxv);
            if (fmaxv < f_tol) err = MIN_S_FTOL;
        }
        if (istep + 1 == nsteps) err = MIN_F_MAX_ITER;
        if (err) continue;
        launch_dep(st, k_cg_dots, grid, 256, 0, N, s->f, f0, L, part, counter);
        MAPPG_CUDA(cudaGetLastError());
        double dd[2];
        MAPPG_CUDA(cudaMemcpyAsync(dd, &L->dot[0], sizeof(dd), cudaMemcpyDeviceToHost, st));
        MAPPG_CUDA(cudaStreamSynchronize(st));
        const double ratio = (dd[0] - dd[1]) / f0_f0;
        launch_dep(st, k_cg_dir, grid, 256, 0, N, h, s->f, ratio);
        MAPPG_CUDA(cudaGetLastError());
        f0_f0 = dd[0];
    }
    MAPPG_CUDA(cudaMemcpyAsync(h, s->f, sizeof(double) * N, cudaMemcpyDeviceToDevice, st));
    read_prep(&fh, &hh, &hmax, &fmaxv);
    DevScalars hs;
    MAPPG_CUDA(cudaMemcpyAsync(&hs, s->sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, st));
    MAPPG_CUDA(cudaStreamSynchronize(st));
    if (hs.overflow) throw Error{MAPPG_ERR_NBR, "neighbour list capacity exceeded during minimization"};
    if (hs.bad) throw Error{MAPPG_ERR_NAN, "non-finite value during minimization"};
    if (stats) {
        stats[0] = istep;
        stats[1] = pe_force;
        stats[2] = fmaxv;
        stats[3] = err;
        stats[4] = (double)n_en;
        stats[5] = (double)n_fc;
    }
}

}  // namespace mappg

// ------------------------------------------------------------------ C entry
namespace mappg {
void sys_upload(mappg_sys* s, const double* host, double* dev);  // system.cu
}

// The energy change E(x + alpha h) - E(x) of a mixed-precision system as its
// minimizers' line searches take it (k_de32), without moving the atoms.
extern "C" int mappg_sys_energy_delta(mappg_sys* s, const double* h, double alpha, double* de) {
    using namespace mappg;
    try {
        if (!s || !h || !de) throw Error{MAPPG_ERR_ARG, "null argument"};
        if (s->precision != MAPPG_MIXED) throw Error{MAPPG_ERR_ARG, "energy differences are for mixed-precision systems"};
        if (s->ncell > 1) throw Error{MAPPG_ERR_UNSUPP, "energy differences run per single cell"};
        if (!s->built) sys_build(s);
        const int n = s->n;
        double* hd = nullptr;
        float4* h32 = nullptr;
        LbScal* L = nullptr;
        unsigned* counter = nullptr;
        // released on every return, including a failed allocation or launch
        struct Free {
            double*& a;
            float4*& b;
            LbScal*& l;
            unsigned*& c;
            mappg_sys* s;
            ~Free() {
                if (a) cudaFree(a);
                if (b) cudaFree(b);
                if (l) cudaFree(l);
                if (c) cudaFree(c);
                s->h32 = nullptr;
                s->keep_rho64 = false;
            }
        } fr{hd, h32, L, counter, s};
        MAPPG_CUDA(cudaMalloc(&hd, sizeof(double) * 3 * (size_t)n));
        MAPPG_CUDA(cudaMalloc(&h32, sizeof(float4) * (size_t)n));
        // the list must hold every pair inside the cutoff at x and at x + alpha h
        double hmax = 0.0;
        for (size_t q = 0; q < 3 * (size_t)n; q++) hmax = std::max(hmax, std::fabs(h[q]));
        lb_update(s);
        sys_upload(s, h, hd);
        const int N = 3 * n, grid = grid_for(s, N, 256);
        MAPPG_CUDA(cudaMalloc(&L, sizeof(LbScal)));
        MAPPG_CUDA(cudaMalloc(&counter, sizeof(unsigned)));
        MAPPG_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned), s->stream));
        launch_dep(s->stream, k_lb_prep, grid, 256, 0, N, hd, hd, s->x, s->x0, L, s->partials, counter);
        MAPPG_CUDA(cudaGetLastError());
        double dxmax = 0.0;
        MAPPG_CUDA(cudaMemcpyAsync(&dxmax, &L->dxmax, sizeof(double), cudaMemcpyDeviceToHost, s->stream));
        MAPPG_CUDA(cudaStreamSynchronize(s->stream));
        if (!(1.7320508075688772 * (std::fabs(alpha) * hmax + dxmax) < 0.5 * s->skin))
            throw Error{MAPPG_ERR_ARG, "alpha*h moves atoms beyond the neighbour list's skin"};
        s->keep_rho64 = true;
        s->h32 = h32;
        launch_force(s);  // density of x kept in FP64, F'(rho) and forces of x
        launch_dep(s->stream, k_lb_h32, grid_for(s, n, 256), 256, 0, n, hd, h32);
        launch_de32(s, alpha);
        MAPPG_CUDA(cudaMemcpyAsync(de, &s->sc->de, sizeof(double), cudaMemcpyDeviceToHost, s->stream));
        MAPPG_CUDA(cudaStreamSynchronize(s->stream));
        return MAPPG_OK;
    } catch (const Error& e) {
        set_error(e.msg);
        return e.code;
    } catch (const std::exception& e) {
        set_error(e.what());
        return MAPPG_ERR_ARG;
    }
}
