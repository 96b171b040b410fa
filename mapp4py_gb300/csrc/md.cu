// NVT molecular dynamics on the device: md.nvt(T,dt).run(atoms,nsteps).
//
// One step of MDNVT::run (md_nvt.cpp:409-438) is a fixed kernel sequence,
// captured once into a CUDA graph and replayed.
//
// FP64 path (the reference's operation order without fused multiply-adds,
// f*(dt2/m) for its f*dt2/m, so the trajectory follows the oracle to rounding;
// three FP64 divisions an atom cost more than the rest of a kick):
//   k_kick_drift64   v = v*fac_x_d + f*dt2/m; x += v*dt; sum of v*dt
//                    (update_x_d__x, md_nvt.cpp:70-102); fac_x_d holds the
//                    opening thermostat half, chain(T/T0)
//   k_com_skin64     x -= mean displacement; skin test (DynamicMD::decide,
//                    dynamic_md.cpp:90-105) opens the rebuild gate
//   rebuild chain    (system.cu) only when the gate is open
//   density, force   (pair64.cu, or eam.cu over full rows)
//   k_kick2_64       v += f*dt2/m, kinetic tensor (update_x_d,
//                    md_nvt.cpp:106-128), the force call's energy and virial
//                    from its partial sums, closing thermostat half, thermo
//                    row, and the next step's opening half
//
// Mixed path (FP64 state, fewer FP64 instructions; GB300 runs FP64 at a
// small fraction of FP32):
//   k_integrate32    the pending closing kick of the previous step and this
//                    step's kick as one, v <- A v + B f dt/2m (A = fc*fo,
//                    B = 1 + fc*fo; A = fo, B = 1 on the first), fo the
//                    opening half; x += v dt (FP64), v32 = (float)v, the frame
//                    position p32 from x, the FP32 skin test and the
//                    displacement sums; the mean displacement is accumulated
//                    in sc->drift (k_close32) and removed from x at the next rebuild and
//                    at the end of the run (a uniform shift leaves forces and
//                    energies unchanged)
//   rebuild chain, k_density32, k_force32
//   k_close32        kinetic tensor of v + f dt/2m, the force call's energy and
//                    virial from its partial sums, closing half, thermo row,
//                    the next step's opening half
// Velocity scaling stays lazy as in the reference: the chain's factor is
// folded into the next kick and applied at the end of the run
// (update_x_d_final, md_nvt.cpp:51-56).
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "eam_common.cuh"
#include "nhc.cuh"

namespace mappg {

void launch_cells_done(mappg_sys* s, const EamArgs& a, int what);  // eam32.cu
void lb_update(mappg_sys* s);                                       // lbfgs.cu

struct MdArgs {
    int n;
    double* x;
    double* v;
    const double* f;
    const float* f32;
    float* v32;
    const double* x0;
    const uint8_t* elem;
    const int* binc;
    float4* p32;
    const float4* p0;
    const uint8_t* dof;    // x_dof bits (null: every component free)
    int com_on[3];         // the mean displacement is removed along c (no frozen atom along c)
    double masses[kMaxElem];
    double dtm[kMaxElem];  // dt2/m
    float dtm32[kMaxElem];
    float m32[kMaxElem];   // masses as floats (the kinetic tensors' FP32 products)
    double dt, dt2, n_inv, skin_sq;
    int drift_rows;        // mixed: blocks of k_integrate32
    const double* pass_part;  // the force call's partial sums, where its totals
    PassRows pass;            // are left to the closing kernel (else pass.force = 0)
    float dt32, skin_sq32;
    double bs[6];          // x -> scaled frame
    Frame fr;
    double* partials;
    double* thermo;  // rows of 14 or null (a batch: rows of ncell x (pe, T))
    long long nsteps;
    NhcParams nhc;
    DevScalars* sc;
    // batch of cells
    int ncell, nchunk;
    const CellGeo* cells;
    const int* cell_of;
    const int* chunk_begin;
    const int* chunk_cell;
    const int* cell_chunk;
    double* chunk_part;
    double* chunk_disp;
    CellMd* cmd;
    uint8_t* cell_reb;  // per cell: an atom moved beyond skin/2 (rebuild that cell)
};

// NHC parameters of one cell of a batch: its own target and dof
__device__ __forceinline__ NhcParams cell_nhc(const NhcParams& P0, const CellMd* m) {
    NhcParams P = P0;
    P.T = m->T;
    P.T_inv = 1.0 / m->T;
    P.ndof = (int)m->ndof;
    P.ndof_kB = m->ndof_kB;
    return P;
}

// pre_init (md_nvt.cpp:256-340): kinetic tensor and temperature of the
// incoming velocities
__global__ void k_mvv_init(MdArgs a) {
    dep_wait();
    double d[6] = {0, 0, 0, 0, 0, 0};
    const int n = a.n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double m = a.masses[a.elem[i]];
        double v0 = a.v[i], v1 = a.v[n + i], v2 = a.v[2 * n + i];
        if (a.dof) {
            const unsigned b = a.dof[i];
            if (!(b & 1u)) v0 = 0.0;
            if (!(b & 2u)) v1 = 0.0;
            if (!(b & 4u)) v2 = 0.0;
        }
        d[0] += __dmul_rn(__dmul_rn(v0, v0), m);
        d[1] += __dmul_rn(__dmul_rn(v0, v1), m);
        d[2] += __dmul_rn(__dmul_rn(v0, v2), m);
        d[3] += __dmul_rn(__dmul_rn(v1, v1), m);
        d[4] += __dmul_rn(__dmul_rn(v1, v2), m);
        d[5] += __dmul_rn(__dmul_rn(v2, v2), m);
    }
    __shared__ double t[6];
    if (block_partials<6>(d, a.partials, 0, &a.sc->counter[3])) {
        final_sums<6>(a.partials, gridDim.x, t);
        if (threadIdx.x == 0) {
            for (int k = 0; k < 6; k++) a.sc->mvv[k] = t[k];
            a.sc->T_part = (t[0] + (t[3] + t[5])) * a.nhc.ndof_kB_inv;
            a.sc->counter[3] = 0;
            a.sc->step = 0;
        }
    }
}

// What the last block of a step's closing kernel does with the kinetic
// tensor mvv of the step (MDNVT::run, md_nvt.cpp:427-432, then 409-412 of the
// next step): the closing half of the thermostat, the thermo row, and the
// next step's opening half, taken ahead by the thread that has just closed
// this one.  The chain state before that opening half stays in sc->eta (the
// run may end here, and exports read it), the one after it in sc->eta_next.
// The device scalars it needs are read at the start of the kernel (load),
// and a thread that waits for the block to be counted in forms what the chain
// can without the temperature (pre): the serial part is the chain's latency.
struct CloseStep {
    double eta[kMaxChain], ev[7], T, fac;
    long long step;
    Chain3 c;
    __device__ __forceinline__ static bool three(const MdArgs& a) { return a.nhc.L == 3 && a.nhc.niters == 1; }
    __device__ __forceinline__ void load(const DevScalars* sc) {
        const int t = threadIdx.x;
        if (t < kMaxChain) eta[t] = sc->eta_next[t];
        if (t >= kMaxChain && t < kMaxChain + 7) ev[t - kMaxChain] = t == kMaxChain ? sc->energy : sc->virial[t - kMaxChain - 1];
        if (t == 31) step = sc->step;
    }
    __device__ __forceinline__ void pre(const MdArgs& a) {
        if (three(a)) c.pre(a.nhc, eta);
    }
    // one half on eta (one thread); c.pre is done
    __device__ __forceinline__ double half(const MdArgs& a, double T_r) {
        if (three(a)) {
            const double f = c.post(a.nhc, T_r);
            if (c.in_range) {
                eta[0] = c.e0;
                eta[1] = c.e1;
                eta[2] = c.e2;
                return f;
            }
        }
        return nhc_any(a.nhc, eta, T_r);
    }
    // whole last block: the energy and virial of the step's force call, where
    // its passes left them as partial sums
    __device__ __forceinline__ void totals(const MdArgs& a) {
        if (!a.pass.force) return;
        pass_totals(a.pass_part, a.pass, ev);
        if (threadIdx.x < 7) (threadIdx.x ? a.sc->virial[threadIdx.x - 1] : a.sc->energy) = ev[threadIdx.x];
    }
    // first warp of the block; returns the closing factor
    __device__ __forceinline__ double close(const MdArgs& a, const double* mvv) {
        const int lane = threadIdx.x;
        DevScalars* sc = a.sc;
        if (lane == 0) {
            T = (mvv[0] + (mvv[3] + mvv[5])) * a.nhc.ndof_kB_inv;
            fac = half(a, T * a.nhc.T_inv);
            T *= fac * fac;
        }
        __syncwarp();
        const double f2 = fac * fac;
        const long long st = step + 1;
        if (lane < kMaxChain) sc->eta[lane] = eta[lane];
        if (a.thermo && st <= a.nsteps && lane < 14)
            a.thermo[14 * st + lane] = lane == 0   ? ev[0]
                                       : lane == 1 ? T
                                       : lane < 8  ? mvv[lane - 2] * f2
                                                   : ev[lane - 7];
        if (lane == 0) {
            sc->step = st;
            if (!(isfinite(ev[0]) && isfinite(T))) sc->bad = 1;
        }
        __syncwarp();
        return fac;
    }
    // lane 0: the opening factor of the next step, whose list check starts anew
    __device__ __forceinline__ double open(const MdArgs& a) {
        pre(a);
        const double fo = half(a, T * a.nhc.T_inv);
        for (int k = 0; k < a.nhc.L; k++) a.sc->eta_next[k] = eta[k];
        a.sc->rebuild = 0;
        return fo;
    }
};

// block_partials of a kernel that ends a step: a thread of the second warp
// does S.pre while the first counts the block in
template <int K, class T>
__device__ __forceinline__ bool close_partials(const T (&v)[K], const MdArgs& a, unsigned* counter, CloseStep& S) {
    const double t = block_sums<K>(v);
    if (threadIdx.x < K) a.partials[blockIdx.x * kRedSlots + threadIdx.x] = t;
    if (threadIdx.x == 32) S.pre(a);
    return last_block(counter);
}

// run start (one block): no displacement sums yet (a list build before the
// first step reads them), thermo row 0, no pending velocity scale or kick, the
// first step's opening half
__global__ void k_run_begin(MdArgs a) {
    dep_wait();
    for (int q = threadIdx.x; q < 3 * a.drift_rows; q += blockDim.x) a.partials[(q / 3) * kRedSlots + 8 + q % 3] = 0.0;
    if (threadIdx.x != 0) return;
    DevScalars* sc = a.sc;
    write_thermo_row(a.thermo, sc, 0);
    double eta[kMaxChain];
    for (int k = 0; k < a.nhc.L; k++) eta[k] = sc->eta[k];
    const double fo = nhc_step(a.nhc, eta, sc->T_part * a.nhc.T_inv);
    for (int k = 0; k < a.nhc.L; k++) sc->eta_next[k] = eta[k];
    sc->fac_x_d = 1.0;
    sc->fac_next = fo;
    sc->pending_kick = 0;
    sc->kickA = fo;
    sc->kickB = 1.0;
    sc->rebuild = 0;
}

// ------------------------------------------------------------------ FP64 path
__global__ void __launch_bounds__(256) k_kick_drift64(MdArgs a) {
    dep_wait();
    const int n = a.n;
    const double fac = a.sc->fac_next;
    double dsum[3] = {0, 0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        // all loads before the first store, which they could not pass
        const int e = a.elem[i];
        const unsigned b = a.dof ? a.dof[i] : 7u;
        double vv[3], ff[3], xx[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            vv[c] = a.v[c * n + i];
            ff[c] = a.f[c * n + i];
            xx[c] = a.x[c * n + i];
        }
        const double dtm = a.dtm[e];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            // a frozen component keeps its velocity and still drifts
            // (update_x_d__x_w_dof, md_nvt.cpp:144-180)
            if ((b >> c) & 1u) vv[c] = __dadd_rn(__dmul_rn(vv[c], fac), __dmul_rn(ff[c], dtm));
            double dx = __dmul_rn(vv[c], a.dt);
            dsum[c] = __dadd_rn(dsum[c], dx);
            a.v[c * n + i] = vv[c];
            a.x[c * n + i] = __dadd_rn(xx[c], dx);
        }
    }
    __shared__ double t[3];
    if (block_partials<3>(dsum, a.partials, 0, &a.sc->counter[4])) {
        final_sums<3>(a.partials, gridDim.x, t);
        if (threadIdx.x == 0) {
            for (int c = 0; c < 3; c++) a.sc->com[c] = a.com_on[c] ? t[c] * a.n_inv : 0.0;
            a.sc->counter[4] = 0;
        }
    }
}

__global__ void __launch_bounds__(256) k_com_skin64(MdArgs a) {
    dep_wait();
    const int n = a.n;
    const double c0 = a.sc->com[0], c1 = a.sc->com[1], c2 = a.sc->com[2];
    int moved = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double b0 = a.x0[i], b1 = a.x0[n + i], b2 = a.x0[2 * n + i];  // before the stores
        double x0 = __dsub_rn(a.x[i], c0), x1 = __dsub_rn(a.x[n + i], c1), x2 = __dsub_rn(a.x[2 * n + i], c2);
        a.x[i] = x0;
        a.x[n + i] = x1;
        a.x[2 * n + i] = x2;
        double d0 = __dsub_rn(b0, x0), d1 = __dsub_rn(b1, x1), d2 = __dsub_rn(b2, x2);
        double r = __dadd_rn(__dmul_rn(d0, d0), __dadd_rn(__dmul_rn(d1, d1), __dmul_rn(d2, d2)));
        moved |= r > a.skin_sq;
    }
    if (__syncthreads_or(moved) && threadIdx.x == 0) a.sc->rebuild = 1;
}

__global__ void __launch_bounds__(256) k_kick2_64(MdArgs a) {
    dep_wait();
    const int n = a.n;
    __shared__ CloseStep S;
    S.load(a.sc);
    double d[6] = {0, 0, 0, 0, 0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int e = a.elem[i];
        const double m = a.masses[e];
        const unsigned b = a.dof ? a.dof[i] : 7u;
        const double dtm = a.dtm[e];
        double vv[3], ff[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {  // before the stores
            vv[c] = a.v[c * n + i];
            ff[c] = a.f[c * n + i];
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            // update_x_d_w_dof (md_nvt.cpp:184-215): frozen components are
            // neither kicked nor counted in the kinetic tensor
            if ((b >> c) & 1u) {
                vv[c] = __dadd_rn(vv[c], __dmul_rn(ff[c], dtm));
                a.v[c * n + i] = vv[c];
            } else {
                vv[c] = 0.0;
            }
        }
        d[0] += __dmul_rn(__dmul_rn(vv[0], vv[0]), m);
        d[1] += __dmul_rn(__dmul_rn(vv[0], vv[1]), m);
        d[2] += __dmul_rn(__dmul_rn(vv[0], vv[2]), m);
        d[3] += __dmul_rn(__dmul_rn(vv[1], vv[1]), m);
        d[4] += __dmul_rn(__dmul_rn(vv[1], vv[2]), m);
        d[5] += __dmul_rn(__dmul_rn(vv[2], vv[2]), m);
    }
    __shared__ double t[6];
    if (close_partials<6>(d, a, &a.sc->counter[5], S)) {
        S.totals(a);
        final_sums<6>(a.partials, gridDim.x, t);
        if (threadIdx.x < 32) {
            const double fac = S.close(a, t);
            if (threadIdx.x == 0) {
                a.sc->fac_x_d = fac;
                a.sc->fac_next = fac * S.open(a);
                a.sc->counter[5] = 0;
            }
        }
    }
}

__global__ void k_run_end64(MdArgs a) {
    dep_wait();
    const int n = a.n;
    const double fac = a.sc->fac_x_d;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 3 * n; i += gridDim.x * blockDim.x)
        if (!a.dof || ((a.dof[i % n] >> (i / n)) & 1u)) a.v[i] = __dmul_rn(a.v[i], fac);
}

// ------------------------------------------------------------------ mixed path
template <bool ORTHO>
__global__ void __launch_bounds__(256) k_integrate32(MdArgs a) {
    dep_wait();
    const int n = a.n;
    const double A = a.sc->kickA;
    const float B = (float)a.sc->kickB;
    float dsum0 = 0.f, dsum1 = 0.f, dsum2 = 0.f;
    int moved = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        // all loads before the first store, which they could not pass
        const int e = a.elem[i], bc = a.binc[i];
        const unsigned b = a.dof ? a.dof[i] : 7u;
        const float4 q = a.p0[i];
        double xv[3], vv[3];
        float vf[3], ff[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            vv[c] = a.v[c * n + i];
            xv[c] = a.x[c * n + i];
            ff[c] = a.f32[c * n + i];
        }
        const float kf = a.dtm32[e] * B;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            // a frozen component (atoms.x_dof) keeps its velocity and drifts
            if ((b >> c) & 1u) vv[c] = fma(vv[c], A, (double)(ff[c] * kf));
            xv[c] = fma(vv[c], a.dt, xv[c]);
            a.v[c * n + i] = vv[c];
            a.x[c * n + i] = xv[c];
            vf[c] = (float)vv[c];
            a.v32[c * n + i] = vf[c];
        }
        dsum0 = fmaf(vf[0], a.dt32, dsum0);
        dsum1 = fmaf(vf[1], a.dt32, dsum1);
        dsum2 = fmaf(vf[2], a.dt32, dsum2);
        // frame position and the skin test against the position at the build
        // the scaled frame; for an orthorhombic box one product per axis
        const double u0 = ORTHO ? a.bs[0] * xv[0] : a.bs[0] * xv[0] + (a.bs[1] * xv[1] + a.bs[2] * xv[2]);
        const double u1 = ORTHO ? a.bs[3] * xv[1] : a.bs[3] * xv[1] + a.bs[4] * xv[2];
        const double u2 = a.bs[5] * xv[2];
        float4 p;
        p.x = (float)(u0 - (double)(8 * (bc & 1023)));
        p.y = (float)(u1 - (double)(8 * ((bc >> 10) & 1023)));
        p.z = (float)(u2 - (double)(8 * ((bc >> 20) & 1023)));
        p.w = 0.f;
        a.p32[i] = p;
        const float da = p.x - q.x, db = p.y - q.y, dc = p.z - q.z;
        float cx, cy, cz;
        if (ORTHO) {
            cx = da * a.fr.G[0][0];
            cy = db * a.fr.G[1][1];
            cz = dc * a.fr.G[2][2];
        } else {
            cx = da * a.fr.G[0][0] + db * a.fr.G[1][0] + dc * a.fr.G[2][0];
            cy = db * a.fr.G[1][1] + dc * a.fr.G[2][1];
            cz = dc * a.fr.G[2][2];
        }
        moved |= fmaf(cx, cx, fmaf(cy, cy, cz * cz)) > a.skin_sq32;
    }
    if (__syncthreads_or(moved) && threadIdx.x == 0) a.sc->rebuild = 1;
    // the block's displacement sum; k_close32 adds the blocks' up, and a
    // rebuild or the run's last export before that (drift_now)
    const float dv[3] = {a.com_on[0] ? dsum0 : 0.f, a.com_on[1] ? dsum1 : 0.f, a.com_on[2] ? dsum2 : 0.f};
    const double t = block_sums<3>(dv);
    if (threadIdx.x < 3) a.partials[blockIdx.x * kRedSlots + 8 + threadIdx.x] = t;
}

// update_x_d (md_nvt.cpp:106-128) and the closing half of the thermostat
// (md_nvt.cpp:427-432) of a mixed step: kinetic tensor of the half-kicked
// velocity v + f dt/2m (FP32 terms, FP64 sums), then in the last block the
// mean displacement of the step and what CloseStep does
__global__ void __launch_bounds__(256) k_close32(MdArgs a) {
    dep_wait();
    const int n = a.n;
    __shared__ CloseStep S;
    S.load(a.sc);
    float k0 = 0.f, k1 = 0.f, k2 = 0.f, k3 = 0.f, k4 = 0.f, k5 = 0.f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int e = a.elem[i];
        const float dtm = a.dtm32[e], m = a.m32[e];
        float vx = fmaf(a.f32[i], dtm, a.v32[i]);
        float vy = fmaf(a.f32[n + i], dtm, a.v32[n + i]);
        float vz = fmaf(a.f32[2 * n + i], dtm, a.v32[2 * n + i]);
        if (a.dof) {  // frozen components leave the kinetic tensor
            const unsigned b = a.dof[i];
            if (!(b & 1u)) vx = 0.f;
            if (!(b & 2u)) vy = 0.f;
            if (!(b & 4u)) vz = 0.f;
        }
        const float mx = m * vx, my = m * vy, mz = m * vz;
        k0 = fmaf(mx, vx, k0);
        k1 = fmaf(mx, vy, k1);
        k2 = fmaf(mx, vz, k2);
        k3 = fmaf(my, vy, k3);
        k4 = fmaf(my, vz, k4);
        k5 = fmaf(mz, vz, k5);
    }
    const float d[6] = {k0, k1, k2, k3, k4, k5};
    __shared__ double t[11];
    if (close_partials<6>(d, a, &a.sc->counter[5], S)) {
        // the kinetic tensor in t[0..5], k_integrate32's displacement sums
        // in t[8..10]
        S.totals(a);
        final_sums<11>(a.partials, gridDim.x, t, a.drift_rows);
        for (int q = threadIdx.x; q < 3 * a.drift_rows; q += blockDim.x) a.partials[(q / 3) * kRedSlots + 8 + q % 3] = 0.0;
        if (threadIdx.x < 32) {
            const double fac = S.close(a, t);
            if (threadIdx.x < 3) a.sc->drift[threadIdx.x] += t[8 + threadIdx.x] * a.n_inv;
            if (threadIdx.x == 0) {
                a.sc->fac_close = fac;
                a.sc->pending_kick = 1;
                const double F = fac * S.open(a);
                a.sc->kickA = F;
                a.sc->kickB = 1.0 + F;
                a.sc->counter[5] = 0;
            }
        }
    }
}

// the same kinetic tensor per chunk of a batch (slots 7-12), for the
// per-cell closing half in k_cells_done
__global__ void __launch_bounds__(256) k_ke32b(MdArgs a) {
    dep_wait();
    const int n = a.n;
    for (int ch = blockIdx.x; ch < a.nchunk; ch += gridDim.x) {
        const int lo = a.chunk_begin[ch], hi = a.chunk_begin[ch + 1];
        float k[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
            const int e = a.elem[i];
            const float dtm = a.dtm32[e], m = a.m32[e];
            const float vx = fmaf(a.f32[i], dtm, a.v32[i]);
            const float vy = fmaf(a.f32[n + i], dtm, a.v32[n + i]);
            const float vz = fmaf(a.f32[2 * n + i], dtm, a.v32[2 * n + i]);
            const float mx = m * vx, my = m * vy, mz = m * vz;
            k[0] = fmaf(mx, vx, k[0]);
            k[1] = fmaf(mx, vy, k[1]);
            k[2] = fmaf(mx, vz, k[2]);
            k[3] = fmaf(my, vy, k[3]);
            k[4] = fmaf(my, vz, k[4]);
            k[5] = fmaf(mz, vz, k[5]);
        }
        chunk_store<6>(k, a.chunk_part + (size_t)ch * kChunkSlots + 7);
    }
}

// end of a mixed run: the pending closing kick and scale, v = (v + f dt/2m) fc,
// and the accumulated mean displacement removed from x
__global__ void k_run_end32(MdArgs a) {
    dep_wait();
    const int n = a.n;
    const bool pend = a.sc->pending_kick != 0;
    const double fc = pend ? a.sc->fac_close : a.sc->fac_x_d;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < 3 * n; q += gridDim.x * blockDim.x) {
        const int i = q % n, c = q / n;
        a.x[q] -= a.sc->drift[c];
        if (a.dof && !((a.dof[i] >> c) & 1u)) continue;  // frozen: neither kicked nor scaled
        double v = a.v[q];
        if (pend) v += (double)a.f32[q] * a.dtm[a.elem[i]];
        a.v[q] = v * fc;
    }
}

__global__ void k_clear_drift(DevScalars* sc) {
    dep_wait();
    sc->drift[0] = sc->drift[1] = sc->drift[2] = 0.0;
    sc->pending_kick = 0;
}

// ------------------------------------------------------------------ batch of cells (mixed path)
// per-cell sums of chunk slots lo..lo+K-1 by one warp per cell, fixed order
template <int K>
__device__ __forceinline__ void cell_sums(const MdArgs& a, const double* part, int stride, int c, double (&t)[K]) {
    const int lane = threadIdx.x & 31;
    const int lo = a.cell_chunk[c], hi = a.cell_chunk[c + 1];
#pragma unroll
    for (int k = 0; k < K; k++) {
        double v = 0.0;
        for (int ch = lo + lane; ch < hi; ch += 32) v += part[(size_t)ch * stride + k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        t[k] = v;
    }
}

// kinetic tensor of the incoming velocities per chunk (slots 7-12)
__global__ void __launch_bounds__(256) k_mvv_init_b(MdArgs a) {
    dep_wait();
    const int n = a.n;
    for (int ch = blockIdx.x; ch < a.nchunk; ch += gridDim.x) {
        const int lo = a.chunk_begin[ch], hi = a.chunk_begin[ch + 1];
        double d[6] = {0, 0, 0, 0, 0, 0};
        for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
            double m = a.masses[a.elem[i]];
            double v0 = a.v[i], v1 = a.v[n + i], v2 = a.v[2 * n + i];
            d[0] += __dmul_rn(__dmul_rn(v0, v0), m);
            d[1] += __dmul_rn(__dmul_rn(v0, v1), m);
            d[2] += __dmul_rn(__dmul_rn(v0, v2), m);
            d[3] += __dmul_rn(__dmul_rn(v1, v1), m);
            d[4] += __dmul_rn(__dmul_rn(v1, v2), m);
            d[5] += __dmul_rn(__dmul_rn(v2, v2), m);
        }
        chunk_store<6>(d, a.chunk_part + (size_t)ch * kChunkSlots + 7);
    }
}

// run start per cell: kinetic tensor, T, thermo row 0, no pending scale/kick
__global__ void k_cells_begin(MdArgs a) {
    dep_wait();
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (c >= a.ncell) return;
    double t[6];
    cell_sums<6>(a, a.chunk_part + 7, kChunkSlots, c, t);
    if ((threadIdx.x & 31) != 0) return;
    CellMd* m = a.cmd + c;
    for (int k = 0; k < 6; k++) m->mvv[k] = t[k];
    m->T_part = (t[0] + (t[3] + t[5])) / m->ndof_kB;
    m->step = 0;
    m->fac_x_d = 1.0;
    m->pending_kick = 0;
    if (a.thermo) {
        a.thermo[2 * c] = m->energy;
        a.thermo[2 * c + 1] = m->T_part;
    }
}

// opening half of every cell's chain and its kick factors (k_run_begin and
// CloseStep::open of one cell)
__global__ void k_cells_open(MdArgs a) {
    dep_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c == 0) a.sc->rebuild = 0;
    if (c >= a.ncell) return;
    CellMd* m = a.cmd + c;
    const NhcParams P = cell_nhc(a.nhc, m);
    const double fo = thermo_half(P, m);
    if (m->pending_kick) {
        const double F = m->fac_close * fo;
        m->kickA = F;
        m->kickB = 1.0 + F;
    } else {
        m->kickA = fo;
        m->kickB = 1.0;
    }
}

// k_integrate32 per chunk: the cell's kick factors and frame, displacement
// sums per chunk
__global__ void __launch_bounds__(256) k_integrate32b(MdArgs a) {
    dep_wait();
    const int n = a.n;
    int moved = 0;
    for (int ch = blockIdx.x; ch < a.nchunk; ch += gridDim.x) {
        int moved_ch = 0;
        const int lo = a.chunk_begin[ch], hi = a.chunk_begin[ch + 1];
        const int c = a.chunk_cell[ch];
        const CellGeo& g = a.cells[c];
        const double A = a.cmd[c].kickA;
        const float B = (float)a.cmd[c].kickB;
        // the cell's frame, read before the loop's stores
        const bool orth = g.ortho != 0;  // uniform over the chunk
        const double bs[6] = {g.bs[0], g.bs[1], g.bs[2], g.bs[3], g.bs[4], g.bs[5]};
        const float G0 = g.G[0][0], G1 = g.G[1][0], G2 = g.G[2][0], G3 = g.G[1][1], G4 = g.G[2][1], G5 = g.G[2][2];
        float dsum0 = 0.f, dsum1 = 0.f, dsum2 = 0.f;
        for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
            // all loads before the first store, which they could not pass
            const int e = a.elem[i], bc = a.binc[i];
            const float4 p0 = a.p0[i];
            double xv[3], vv[3];
            float vf[3], ff[3];
#pragma unroll
            for (int q = 0; q < 3; q++) {
                vv[q] = a.v[q * n + i];
                xv[q] = a.x[q * n + i];
                ff[q] = a.f32[q * n + i];
            }
            const float kf = a.dtm32[e] * B;
#pragma unroll
            for (int q = 0; q < 3; q++) {
                vv[q] = fma(vv[q], A, (double)(ff[q] * kf));
                xv[q] = fma(vv[q], a.dt, xv[q]);
                a.v[q * n + i] = vv[q];
                a.x[q * n + i] = xv[q];
                vf[q] = (float)vv[q];
                a.v32[q * n + i] = vf[q];
            }
            dsum0 = fmaf(vf[0], a.dt32, dsum0);
            dsum1 = fmaf(vf[1], a.dt32, dsum1);
            dsum2 = fmaf(vf[2], a.dt32, dsum2);
            const double u0 = orth ? bs[0] * xv[0] : bs[0] * xv[0] + (bs[1] * xv[1] + bs[2] * xv[2]);
            const double u1 = orth ? bs[3] * xv[1] : bs[3] * xv[1] + bs[4] * xv[2];
            const double u2 = bs[5] * xv[2];
            float4 p;
            p.x = (float)(u0 - (double)(8 * (bc & 1023)));
            p.y = (float)(u1 - (double)(8 * ((bc >> 10) & 1023)));
            p.z = (float)(u2 - (double)(8 * ((bc >> 20) & 1023)));
            p.w = 0.f;
            a.p32[i] = p;
            const float da = p.x - p0.x, db = p.y - p0.y, dc = p.z - p0.z;
            const float cx = da * G0 + db * G1 + dc * G2;
            const float cy = db * G3 + dc * G4;
            const float cz = dc * G5;
            moved_ch |= fmaf(cx, cx, fmaf(cy, cy, cz * cz)) > a.skin_sq32;
        }
        // the chunk's cell is rebuilt at the next list check
        if (__syncthreads_or(moved_ch)) {
            moved = 1;
            if (threadIdx.x == 0) a.cell_reb[c] = 1;
        }
        const float ds[3] = {dsum0, dsum1, dsum2};
        chunk_store<3>(ds, a.chunk_disp + (size_t)ch * 4);
    }
    if (__syncthreads_or(moved) && threadIdx.x == 0) a.sc->rebuild = 1;
}

// per-cell mean displacement of the step, added to the cell's drift
__global__ void k_cells_com(MdArgs a) {
    dep_wait();
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (c >= a.ncell) return;
    double t[3];
    cell_sums<3>(a, a.chunk_disp, 4, c, t);
    if ((threadIdx.x & 31) != 0) return;
    CellMd* m = a.cmd + c;
    const double natms = (double)(a.cells[c].end - a.cells[c].begin);
    for (int k = 0; k < 3; k++) {
        m->com[k] = t[k] / natms;
        m->drift[k] += m->com[k];
    }
    m->pending_kick = 0;
}

// end of a batch run: pending closing kick and scale, drift removed, per cell
__global__ void k_run_end32b(MdArgs a) {
    dep_wait();
    const int n = a.n;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < 3 * n; q += gridDim.x * blockDim.x) {
        const int i = q % n, k = q / n;
        const CellMd* m = a.cmd + a.cell_of[i];
        const bool pend = m->pending_kick != 0;
        const double fc = pend ? m->fac_close : m->fac_x_d;
        double v = a.v[q];
        if (pend) v += (double)a.f32[q] * a.dtm[a.elem[i]];
        a.v[q] = v * fc;
        a.x[q] -= m->drift[k];
    }
}

__global__ void k_cells_clear(MdArgs a) {
    dep_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= a.ncell) return;
    CellMd* m = a.cmd + c;
    m->drift[0] = m->drift[1] = m->drift[2] = 0.0;
    m->pending_kick = 0;
}

}  // namespace mappg

using namespace mappg;

namespace mappg {
void sys_build(mappg_sys* s);

static MdArgs md_args(mappg_sys* s, double T, double dt, double kB, double t_relax, int L, int niters,
                      long long nsteps, double* thermo_dev) {
    MdArgs a;
    memset(&a, 0, sizeof(a));
    a.n = s->n;
    a.pass_part = s->partials + kRedSlots * kMaxBlocks;
    a.x = s->x;
    a.v = s->v;
    a.f = s->f;
    a.f32 = s->f32;
    a.v32 = s->v32;
    a.x0 = s->x0;
    a.elem = s->elem;
    a.binc = s->binc;
    a.p32 = s->p32;
    a.p0 = s->p0;
    a.dt = dt;
    a.dt2 = dt / 2.0;
    a.n_inv = 1.0 / (double)s->n;
    a.dt32 = (float)dt;
    for (int e = 0; e < s->ne; e++) {
        a.masses[e] = s->masses[e];
        a.dtm[e] = a.dt2 / s->masses[e];
        a.dtm32[e] = (float)a.dtm[e];
        a.m32[e] = (float)a.masses[e];
    }
    a.skin_sq = 0.25 * s->skin * s->skin;
    // the FP32 skin test triggers a little early rather than late
    a.skin_sq32 = (float)(a.skin_sq * (1.0 - 1e-4));
    const double S[3] = {8.0 * s->nb[0], 8.0 * s->nb[1], 8.0 * s->nb[2]};
    const double* b6 = s->box.b6;
    a.bs[0] = b6[0] * S[0];
    a.bs[1] = b6[1] * S[0];
    a.bs[2] = b6[2] * S[0];
    a.bs[3] = b6[3] * S[1];
    a.bs[4] = b6[4] * S[1];
    a.bs[5] = b6[5] * S[2];
    a.fr = s->frame;
    a.partials = s->partials;
    a.thermo = thermo_dev;
    a.nsteps = nsteps;
    // ThermostatNHC(dt/2, t_relax, L, niters)  md_nvt.cpp:19, thermostat.cpp:20-36
    const double tdt = dt / 2.0;
    a.nhc.T = T;
    a.nhc.T_inv = 1.0 / T;
    a.nhc.ddt = tdt / (double)niters;
    a.nhc.ddt2 = 0.5 * tdt / (double)niters;
    a.nhc.freq_sq = 1.0 / (t_relax * t_relax);
    a.nhc.kB = kB;
    // MDNVT::pre_init (md_nvt.cpp:264-291): frozen components leave the
    // degrees of freedom, and the mean displacement is kept along a
    // component in which any atom is frozen
    a.dof = s->dof;
    a.nhc.ndof = 3 * s->n - (s->dof_frozen[0] + s->dof_frozen[1] + s->dof_frozen[2]);
    for (int c = 0; c < 3; c++) a.com_on[c] = s->dof_frozen[c] == 0;
    a.nhc.ndof_kB = a.nhc.ndof * kB;
    a.nhc.ndof_kB_inv = 1.0 / a.nhc.ndof_kB;
    a.nhc.ndof_d = (double)a.nhc.ndof;
    a.nhc.L = L;
    a.nhc.niters = niters;
    a.sc = s->sc;
    a.ncell = s->ncell;
    a.nchunk = s->nchunk;
    a.cells = s->cells_dev;
    a.cell_of = s->cell_of;
    a.chunk_begin = s->chunk_begin;
    a.chunk_cell = s->chunk_cell;
    a.cell_chunk = s->cell_chunk;
    a.chunk_part = s->chunk_part;
    a.chunk_disp = s->chunk_disp;
    a.cmd = s->cmd;
    a.cell_reb = s->cell_reb;
    return a;
}

// launch shapes of the streaming MD kernels.  FP64 work per atom (wide): a
// small system is spread over all SMs, 64 threads a block and up, as the FP64
// pipe of an SM is what its atoms wait for.  FP32 work and one reduction:
// blocks of 256, few partials.  A large system takes four blocks of 256 per
// SM, which keep loads in flight and the sum over the blocks' partials short.
struct MdShape {
    int grid, block;
};
static MdShape md_shape(const mappg_sys* s, bool wide) {
    const int per = ((s->n + s->sm_count - 1) / s->sm_count + 31) / 32 * 32;
    const int block = wide ? std::max(64, std::min(256, per)) : 256;
    return {std::max(1, std::min((s->n + block - 1) / block, 4 * s->sm_count)), block};
}

struct NoHook {
    void operator()() const {}
};

// listed() is called once the step's positions are final (after the list
// check; the passes after it do not move the atoms), closing() before the
// kernel that closes the step
template <class A = NoHook, class B = NoHook>
static void launch_step64(mappg_sys* s, const MdArgs& a, A listed = A(), B closing = B()) {
    const MdShape m = md_shape(s, true);
    launch_dep(s->stream, k_kick_drift64, m.grid, m.block, 0, a);
    launch_dep(s->stream, k_com_skin64, m.grid, m.block, 0, a);
    launch_rebuild_chain(s);
    listed();
    MdArgs b = a;
    {
        struct Defer {
            mappg_sys* s;
            ~Defer() { s->defer_totals = false; }
        } defer{s};
        s->defer_totals = s->own_ent != nullptr;
        launch_force(s);
        if (s->defer_totals) b.pass = s->pass_rows;
    }
    closing();
    launch_dep(s->stream, k_kick2_64, m.grid, m.block, 0, b);
}

template <class A = NoHook, class B = NoHook>
static void launch_step32(mappg_sys* s, const MdArgs& a, A listed = A(), B closing = B()) {
    const MdShape m = md_shape(s, true), c = md_shape(s, false);
    if (a.fr.ortho)
        launch_dep(s->stream, k_integrate32<true>, m.grid, m.block, 0, a);
    else
        launch_dep(s->stream, k_integrate32<false>, m.grid, m.block, 0, a);
    launch_rebuild_chain(s);
    listed();
    EamArgs e = eam_args(s);
    e.defer = 1;
    launch_density32(s, e);
    launch_force32(s, e);
    MdArgs b = a;
    b.pass = s->pass_rows;
    closing();
    launch_dep(s->stream, k_close32, c.grid, c.block, 0, b);
}

static void launch_step32b(mappg_sys* s, const MdArgs& a) {
    const int nc = s->ncell;
    launch_dep(s->stream, k_cells_open, (nc + 255) / 256, 256, 0, a);
    launch_dep(s->stream, k_integrate32b, std::min(s->nchunk, s->sm_count * 8), 256, 0, a);
    launch_dep(s->stream, k_cells_com, (nc * 32 + 255) / 256, 256, 0, a);
    launch_rebuild_chain(s);
    EamArgs e = eam_args(s);
    e.defer = 1;
    launch_density32(s, e);
    launch_force32(s, e);
    launch_dep(s->stream, k_ke32b, std::min(s->nchunk, s->sm_count * 8), 256, 0, a);
    e.thermo = a.thermo;
    e.nsteps = a.nsteps;
    e.nhc = a.nhc;
    launch_cells_done(s, e, 2);  // kinetic tensors, each cell's closing half, thermo rows
}

struct NvtRun {
    MdArgs a;
    cudaGraphExec_t exec = nullptr;
    cudaGraph_t graph = nullptr;
    // batches: the planned steps (up to kBatchGraphSteps) as one graph, so a
    // whole run of every cell is one launch
    cudaGraphExec_t exec_many = nullptr;
    cudaGraph_t graph_many = nullptr;
    long long many = 0;
    int alloc_gen = 0;  // of the device arrays that the graphs hold (mappg_sys::alloc_gen)
    int L = 3;
    long long planned = 0;
    long long done = 0;
    bool thermo = false;
};

static void run_drop_graphs(NvtRun* r) {
    if (r->exec) cudaGraphExecDestroy(r->exec);
    if (r->graph) cudaGraphDestroy(r->graph);
    if (r->exec_many) cudaGraphExecDestroy(r->exec_many);
    if (r->graph_many) cudaGraphDestroy(r->graph_many);
    r->exec = r->exec_many = nullptr;
    r->graph = r->graph_many = nullptr;
}

static void run_clear(mappg_sys* s) {
    NvtRun* r = (NvtRun*)s->run;
    if (!r) return;
    run_drop_graphs(r);
    delete r;
    s->run = nullptr;
    s->drift_rows = 0;
}

// the run's step graphs, over the device arrays as they are now
static void run_capture(mappg_sys* s, NvtRun* r) {
    run_drop_graphs(r);
    auto capture = [&](long long k, cudaGraph_t* gr, cudaGraphExec_t* ex) {
        MAPPG_CUDA(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
        try {
            for (long long q = 0; q < k; q++) {
                if (s->ncell > 1)
                    launch_step32b(s, r->a);
                else if (s->precision == MAPPG_MIXED)
                    launch_step32(s, r->a);
                else
                    launch_step64(s, r->a);
            }
        } catch (...) {
            cudaGraph_t g2 = nullptr;
            cudaStreamEndCapture(s->stream, &g2);
            if (g2) cudaGraphDestroy(g2);
            throw;
        }
        MAPPG_CUDA(cudaStreamEndCapture(s->stream, gr));
        MAPPG_CUDA(cudaGraphInstantiate(ex, *gr, 0));
    };
    capture(1, &r->graph, &r->exec);
    if (r->many) capture(r->many, &r->graph_many, &r->exec_many);
    r->alloc_gen = s->alloc_gen;
}

void nvt_free(mappg_sys* s) { run_clear(s); }

void sys_join_side(mappg_sys* s);  // system.cu

// runs this short launch their steps' kernels directly: capturing and
// instantiating the step graph costs more than it saves over a few steps
constexpr long long kGraphMinSteps = 8;
// longest run of batch steps captured as one graph (about 14 nodes a step)
constexpr long long kBatchGraphSteps = 512;

// MDNVT::init + the opening force call of MDNVT::run, then the step graph
void nvt_begin(mappg_sys* s, double T, double dt, double kB, double t_relax, int L, int niters, long long nsteps,
               const double* eta, bool thermo, const double* Tcell) {
    const bool batch = s->ncell > 1;
    if (batch && s->precision != MAPPG_MIXED) throw Error{MAPPG_ERR_UNSUPP, "batched MD runs in mixed precision"};
    if (batch && !Tcell) throw Error{MAPPG_ERR_ARG, "a batch needs one temperature per cell"};
    if (!batch && Tcell) throw Error{MAPPG_ERR_ARG, "per-cell temperatures need a batch of cells"};
    if (batch) {
        T = 1.0;
        for (int c = 0; c < s->ncell; c++)
            if (!(Tcell[c] > 0.0)) throw Error{MAPPG_ERR_ARG, "T must be positive"};
    }
    if (!(kB == kB)) throw Error{MAPPG_ERR_ARG, "boltzmann constant should be set prior to MD"};
    if (L < 1 || L > kMaxChain) throw Error{MAPPG_ERR_ARG, "L must be in 1..16"};
    if (niters < 1) throw Error{MAPPG_ERR_ARG, "niters must be positive"};
    if (!(dt > 0.0)) throw Error{MAPPG_ERR_ARG, "dt must be positive"};
    if (!(T > 0.0)) throw Error{MAPPG_ERR_ARG, "T must be positive"};
    if (!(t_relax > 0.0)) throw Error{MAPPG_ERR_ARG, "t_relax must be positive"};
    if (nsteps < 0) throw Error{MAPPG_ERR_ARG, "nsteps must be >= 0"};
    if (!s->have_v) throw Error{MAPPG_ERR_ARG, "velocities must be set before MD"};
    run_clear(s);
    double* tdev = nullptr;
    if (thermo) {
        long long need = (batch ? 2LL * s->ncell : 14LL) * (nsteps + 1);
        if (need > s->thermo_cap) {
            if (s->thermo_dev) cudaFree(s->thermo_dev);
            s->thermo_dev = nullptr;
            s->thermo_cap = 0;
            MAPPG_CUDA(cudaMalloc(&s->thermo_dev, sizeof(double) * need));
            s->thermo_cap = need;
        }
        tdev = s->thermo_dev;
    }
    NvtRun* r = new NvtRun();
    s->run = r;
    r->a = md_args(s, T, dt, kB, t_relax, L, niters, nsteps, tdev);
    r->L = L;
    r->planned = nsteps;
    r->thermo = thermo;
    MdArgs& a = r->a;
    int g = grid_for(s, s->n, 256);
    if (batch) {
        // per-cell targets, degrees of freedom and chain state
        std::vector<CellMd> cm(s->ncell);
        MAPPG_CUDA(cudaMemcpyAsync(cm.data(), s->cmd, sizeof(CellMd) * s->ncell, cudaMemcpyDeviceToHost, s->stream));
        MAPPG_CUDA(cudaStreamSynchronize(s->stream));
        for (int c = 0; c < s->ncell; c++) {
            CellMd& m = cm[c];
            m.T = Tcell[c];
            m.ndof = 3.0 * (s->cell_begin[c + 1] - s->cell_begin[c]);
            m.ndof_kB = m.ndof * kB;
            for (int k = 0; k < kMaxChain; k++) m.eta[k] = (eta && k < L) ? eta[(size_t)c * L + k] : 0.0;
            m.drift[0] = m.drift[1] = m.drift[2] = 0.0;
            m.pending_kick = 0;
            m.step = 0;
        }
        MAPPG_CUDA(cudaMemcpyAsync(s->cmd, cm.data(), sizeof(CellMd) * s->ncell, cudaMemcpyHostToDevice, s->stream));
        MAPPG_CUDA(cudaStreamSynchronize(s->stream));
        sys_build(s);
        launch_force(s);
        launch_dep(s->stream, k_mvv_init_b, std::min(s->nchunk, s->sm_count * 8), 256, 0, a);
        launch_dep(s->stream, k_cells_begin, (s->ncell * 32 + 255) / 256, 256, 0, a);
        MAPPG_CUDA(cudaGetLastError());
        r->many = std::min(nsteps, kBatchGraphSteps);
        if (r->many < kGraphMinSteps) r->many = 0;
        run_capture(s, r);
        return;
    }
    double eta_h[kMaxChain] = {0};
    if (eta)
        for (int k = 0; k < L; k++) eta_h[k] = eta[k];
    MAPPG_CUDA(cudaMemcpyAsync(s->sc->eta, eta_h, sizeof(double) * kMaxChain, cudaMemcpyHostToDevice, s->stream));
    launch_dep(s->stream, k_clear_drift, 1, 1, 0, s->sc);
    // MDNVT::run builds the list at its start.  A list built for this box
    // whose atoms all stayed within half the skin of their positions at that
    // build still holds every pair within the cutoff, so the skin test
    // decides here (the forces are the same; only their summation order can
    // differ from a fresh build's)
    if (s->list_box) {
        lb_update(s);
        s->built = true;
    } else {
        sys_build(s);
    }
    launch_force(s);
    // the list and the opening force do not read velocities: an upload of
    // them on the side stream (nvt_run_host) overlaps them and is joined here
    sys_join_side(s);
    launch_dep(s->stream, k_mvv_init, md_shape(s, true).grid, md_shape(s, true).block, 0, a);
    if (s->precision == MAPPG_MIXED) s->drift_rows = a.drift_rows = md_shape(s, true).grid;
    launch_dep(s->stream, k_run_begin, 1, 256, 0, a);
    MAPPG_CUDA(cudaGetLastError());
    if (nsteps < kGraphMinSteps) return;  // nvt_steps launches the kernels itself
    run_capture(s, r);
}

// enqueue steps (no host synchronisation)
void nvt_steps(mappg_sys* s, long long nsteps) {
    NvtRun* r = (NvtRun*)s->run;
    if (!r) throw Error{MAPPG_ERR_ARG, "no NVT run has begun on this system"};
    if (r->done + nsteps > r->planned) throw Error{MAPPG_ERR_ARG, "more steps than the run was begun with"};
    // a list build of the caller's between the steps may have moved the rows
    if (r->exec && r->alloc_gen != s->alloc_gen) run_capture(s, r);
    long long st = 0;
    if (r->exec_many)
        for (; nsteps - st >= r->many; st += r->many) MAPPG_CUDA(cudaGraphLaunch(r->exec_many, s->stream));
    for (; st < nsteps; st++) {
        if (r->exec)
            MAPPG_CUDA(cudaGraphLaunch(r->exec, s->stream));
        else if (s->precision == MAPPG_MIXED)
            launch_step32(s, r->a);
        else
            launch_step64(s, r->a);
    }
    r->done += nsteps;
}

// update_x_d_final, chain state out, thermo rows, checks
void nvt_end(mappg_sys* s, double* eta, double* thermo) {
    NvtRun* r = (NvtRun*)s->run;
    if (!r) throw Error{MAPPG_ERR_ARG, "no NVT run has begun on this system"};
    sys_join_side(s);  // a side-stream read of the positions (nvt_run_xout) comes first
    int g = grid_for(s, 3LL * s->n, 256);
    if (s->ncell > 1) {
        launch_dep(s->stream, k_run_end32b, g, 256, 0, r->a);
        launch_dep(s->stream, k_cells_clear, (s->ncell + 255) / 256, 256, 0, r->a);
        MAPPG_CUDA(cudaGetLastError());
        DevScalars h;
        std::vector<CellMd> cm(s->ncell);
        MAPPG_CUDA(cudaMemcpyAsync(&h, s->sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, s->stream));
        MAPPG_CUDA(cudaMemcpyAsync(cm.data(), s->cmd, sizeof(CellMd) * s->ncell, cudaMemcpyDeviceToHost, s->stream));
        if (thermo && r->thermo)
            MAPPG_CUDA(cudaMemcpyAsync(thermo, r->a.thermo, sizeof(double) * 2 * s->ncell * (r->done + 1),
                                       cudaMemcpyDeviceToHost, s->stream));
        MAPPG_CUDA(cudaStreamSynchronize(s->stream));
        if (eta)
            for (int c = 0; c < s->ncell; c++)
                for (int k = 0; k < r->L; k++) eta[(size_t)c * r->L + k] = cm[c].eta[k];
        run_clear(s);
        if (h.overflow) throw Error{MAPPG_ERR_NBR, "neighbour list capacity exceeded during the run"};
        if (h.bad) throw Error{MAPPG_ERR_NAN, "non-finite position, energy or temperature during the run"};
        return;
    }
    if (s->precision == MAPPG_MIXED) {
        launch_dep(s->stream, k_run_end32, g, 256, 0, r->a);
        launch_dep(s->stream, k_clear_drift, 1, 1, 0, s->sc);
    } else {
        launch_dep(s->stream, k_run_end64, g, 256, 0, r->a);
    }
    MAPPG_CUDA(cudaGetLastError());
    DevScalars h;
    MAPPG_CUDA(cudaMemcpyAsync(&h, s->sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, s->stream));
    if (thermo && r->thermo)
        MAPPG_CUDA(cudaMemcpyAsync(thermo, r->a.thermo, sizeof(double) * 14 * (r->done + 1), cudaMemcpyDeviceToHost,
                                   s->stream));
    MAPPG_CUDA(cudaStreamSynchronize(s->stream));
    if (eta)
        for (int k = 0; k < r->L; k++) eta[k] = h.eta[k];
    run_clear(s);
    if (h.overflow) throw Error{MAPPG_ERR_NBR, "neighbour list capacity exceeded during the run"};
    if (h.bad) throw Error{MAPPG_ERR_NAN, "non-finite position, energy or temperature during the run"};
}

// Positions (what = 0) or velocities (what = 1) of a run at a step boundary,
// written in the caller's atom order.  They are the state MDNVT::run exports
// between steps (md_nvt.cpp:390,436,470): after the closing kick, before the
// deferred thermostat scale.  The mixed path keeps the mean displacement in
// sc->drift and may hold the closing kick back (pending_kick); both are
// applied to the copy here, the run's own state is left as it is.
__global__ void k_snapshot(MdArgs a, const int* __restrict__ id, double* __restrict__ out, int what, int mixed) {
    const int n = a.n;
    const bool pend = mixed && a.sc->pending_kick != 0;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < 3 * n; q += gridDim.x * blockDim.x) {
        const int i = q % n, c = q / n;
        double val;
        if (what == 0) {
            val = a.x[q];
            if (mixed) val -= a.sc->drift[c];
        } else {
            val = a.v[q];
            if (pend) val += (double)a.f32[q] * a.dtm[a.elem[i]];
        }
        out[3 * (size_t)id[i] + c] = val;
    }
}

void nvt_snapshot(mappg_sys* s, double* x, double* v) {
    NvtRun* r = (NvtRun*)s->run;
    if (!r) throw Error{MAPPG_ERR_ARG, "no NVT run has begun on this system"};
    if (s->ncell > 1) throw Error{MAPPG_ERR_UNSUPP, "snapshots are taken of single-cell runs"};
    const int g = grid_for(s, 3LL * s->n, 256);
    const int mixed = s->precision == MAPPG_MIXED ? 1 : 0;
    double* out[2] = {x, v};
    for (int what = 0; what < 2; what++) {
        if (!out[what]) continue;
        k_snapshot<<<g, 256, 0, s->stream>>>(r->a, s->id, s->stage, what, mixed);
        MAPPG_CUDA(cudaGetLastError());
        MAPPG_CUDA(cudaMemcpyAsync(out[what], s->stage, sizeof(double) * 3 * (size_t)s->n, cudaMemcpyDeviceToHost,
                                   s->stream));
        MAPPG_CUDA(cudaStreamSynchronize(s->stream));
    }
    DevScalars h;
    MAPPG_CUDA(cudaMemcpyAsync(&h, s->sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, s->stream));
    MAPPG_CUDA(cudaStreamSynchronize(s->stream));
    if (h.overflow) throw Error{MAPPG_ERR_NBR, "neighbour list capacity exceeded during the run"};
    if (h.bad) throw Error{MAPPG_ERR_NAN, "non-finite position, energy or temperature during the run"};
}

// positions in the caller's order less the mean displacement not yet
// removed (sc->drift; zero on the FP64 path): what the run's end leaves in x
__global__ void k_scatter_x_final(int n, const int* __restrict__ id, const double* __restrict__ x,
                                  const DevScalars* __restrict__ sc, const double* __restrict__ partials, int rows,
                                  double n_inv, double* __restrict__ out) {
    double d[3];
    drift_now(sc, partials, rows, n_inv, d);
    const double d0 = d[0], d1 = d[1], d2 = d[2];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const size_t u = 3 * (size_t)id[i];
        out[u] = x[i] - d0;
        out[u + 1] = x[n + i] - d1;
        out[u + 2] = x[2 * n + i] - d2;
    }
}

// nvt_run whose final positions go to the host array x_out during the last
// step: they are final once that step's list check is done, so the side
// stream gathers them then and copies them out under the density and force
// passes; the run's end (which removes sc->drift from x) waits for the
// gather only.  Needs the side stream (sys_upload_side made it).
void nvt_run_xout(mappg_sys* s, double T, double dt, double kB, double t_relax, int L, int niters, int nsteps,
                  double* eta, double* thermo, double* x_out) {
    nvt_begin(s, T, dt, kB, t_relax, L, niters, nsteps, eta, thermo != nullptr, nullptr);
    NvtRun* r = (NvtRun*)s->run;
    if (nsteps > 0) {
        nvt_steps(s, nsteps - 1);
        auto gather = [&] {
            MAPPG_CUDA(cudaEventRecord(s->ev_main, s->stream));
            MAPPG_CUDA(cudaStreamWaitEvent(s->side, s->ev_main, 0));
            k_scatter_x_final<<<grid_for(s, s->n, 256), 256, 0, s->side>>>(s->n, s->id, s->x, s->sc, s->partials,
                                                                           s->drift_rows, r->a.n_inv, s->stage2);
            MAPPG_CUDA(cudaGetLastError());
            MAPPG_CUDA(cudaEventRecord(s->ev_side, s->side));
        };
        // the closing kernel moves the step's displacement into sc->drift,
        // which the gather reads
        auto gathered = [&] { MAPPG_CUDA(cudaStreamWaitEvent(s->stream, s->ev_side, 0)); };
        if (s->precision == MAPPG_MIXED)
            launch_step32(s, r->a, gather, gathered);
        else
            launch_step64(s, r->a, gather, gathered);
        r->done += 1;
        MAPPG_CUDA(cudaMemcpyAsync(x_out, s->stage2, sizeof(double) * 3 * (size_t)s->n, cudaMemcpyDeviceToHost,
                                   s->side));
    }
    nvt_end(s, eta, thermo);
}

void nvt_run(mappg_sys* s, double T, double dt, double kB, double t_relax, int L, int niters, int nsteps, double* eta,
             double* thermo, const double* Tcell) {
    nvt_begin(s, T, dt, kB, t_relax, L, niters, nsteps, eta, thermo != nullptr, Tcell);
    nvt_steps(s, nsteps);
    nvt_end(s, eta, thermo);
}

}  // namespace mappg
