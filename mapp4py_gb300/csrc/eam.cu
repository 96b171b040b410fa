// FP64 EAM kernels over the full neighbour list, and the launch dispatch for
// both precisions (the mixed kernels are in eam32.cu).  FP64 single cells take
// the passes of pair64.cu, which compute a pair once; those here serve
// batches, mixed systems where they want FP64 (line-search energies, forces
// near convergence), caller-provided scratch, and systems whose pair records
// do not fit in memory.
//
// The reference (ForceFieldEAM::__force_calc, ff_eam.cpp:65-240) walks a half
// list twice and scatters to both atoms of a pair.  Here every atom owns a
// full row, so each atom's sums are private and no atomics are needed:
//   k_density64  rho_i = sum_j rho_{e_j->e_i}(r_ij), then F(rho_i) and
//                F'(rho_i) in the same kernel (the row is complete when the
//                sum ends), with the linear extrapolation above rho_max
//                (ff_eam.cpp:180-191)
//   k_force64    f_i = sum_j -(phi'(r) + F'_i rho'_{j->i}(r) + F'_j rho'_{i->j}(r))
//                * (x_i - x_j)/r, pair energy phi/2 and virial fpair*dx(x)dx/2
//                per entry (each pair appears in both rows)
//   k_energy64   energy only (ff_eam.cpp:244-318): density and pair energy in
//                one pass, then F(rho_i)
// A group of TPA lanes serves one atom; lanes stride over the row, reduce
// with shuffles, and one lane writes the atom's results.  Per-lane energy
// and virial accumulators are reduced per block and then over blocks in a
// fixed order by the last block to finish (deterministic).
//
// Spline evaluation (value ((c3 p + c2) p + c1) p + c0, derivative
// ((3 c3 p + 2 c2) p + c1)/dr) and the index rule m = min(int(r/dr), nr-2),
// p = min(r/dr - m, 1) follow ff_eam.cpp:122-140.  Neighbour images are read
// as x_j + n*H with n from the entry's bin step and atom i's bin.
#include <math.h>

#include <algorithm>

#include "eam_common.cuh"
#include "pos64.cuh"

namespace mappg {

__device__ __forceinline__ double spl_val(const Dbl4& c, double p) { return ((c.w * p + c.z) * p + c.y) * p + c.x; }
__device__ __forceinline__ double spl_der(const Dbl4& c, double p) { return (3.0 * c.w * p + 2.0 * c.z) * p + c.y; }

// one lane's share of atom i's density (FP64)
template <int TPA, class POS>
__device__ __forceinline__ double density64_lane(const EamArgs& a, const Smem64& S, const POS& P, int ei, int i,
                                                 int lane) {
    double acc = 0.0;
    const int nn = __ldg(a.nnbr + i);
    const int* row = a.nbr + (size_t)i * a.maxnbr;
    for (int k = lane; k < nn; k += TPA) {
        const int e = __ldg(row + k);
        const int ej = entry_elem(e);
        double dx, dy, dz;
        P.delta(a, S.sh, e, dx, dy, dz);
        double rsq = dx * dx + dy * dy + dz * dz;
        if (below(rsq, S.cut_sq[ei * a.ne + ej])) {
            double p;
            const int m = knot64_fast(root_from(rsq, recip_root(rsq)), a.dr_inv, a.nr - 2, p);
            acc += spl_val(ldg4(a.rho64 + (size_t)(ej * a.ne + ei * a.rho_ei) * a.nr + m), p);
        }
    }
    return acc;
}

// one lane's share of atom i's force, pair energy and virial (FP64)
template <int TPA, class POS>
__device__ __forceinline__ void force64_lane(const EamArgs& a, const Smem64& S, const POS& P, int ei, double dFi,
                                             int i, int lane, double& fx, double& fy, double& fz, double& ep,
                                             double (&w)[6]) {
    const double dri = a.dr_inv;
    const int nn = __ldg(a.nnbr + i);
    const int* row = a.nbr + (size_t)i * a.maxnbr;
    for (int k = lane; k < nn; k += TPA) {
        const int e = __ldg(row + k);
        const int ej = entry_elem(e);
        double dx, dy, dz;
        P.delta(a, S.sh, e, dx, dy, dz);
        double rsq = dx * dx + dy * dy + dz * dz;
        if (below(rsq, S.cut_sq[ei * a.ne + ej])) {
            const int j = entry_j(e);
            // 1/r from the reciprocal square root and r = rsq/r: one root
            // instead of a root and a division, within an ulp or two of sqrt
            // and 1/sqrt (GB300's FP64 pipe bounds this kernel)
            const double rinv = recip_root(rsq);
            const double r = rsq * rinv;
            double p;
            const int m = knot64_fast(r, dri, a.nr - 2, p);
            const double der_i = spl_der(ldg4(a.rho64 + (size_t)(ej * a.ne + ei * a.rho_ei) * a.nr + m), p) * dri;
            double der_j = der_i;
            if (ej != ei) der_j = spl_der(ldg4(a.rho64 + (size_t)(ei * a.ne + ej * a.rho_ei) * a.nr + m), p) * dri;
            double z, dz_;
            spl_both(ldg4(a.rphi64 + (size_t)(ei * a.ne + ej) * a.nr + m), p, z, dz_);
            const double zp = dz_ * dri;
            const double phi = z * rinv;
            const double dphi = (zp - phi) * rinv;
            const double fp = -(dphi + dFi * der_i + __ldg(a.dF + j) * der_j) * rinv;
            const double fdx = fp * dx, fdy = fp * dy, fdz = fp * dz;
            fx += fdx;
            fy += fdy;
            fz += fdz;
            ep += phi;
            w[0] += fdx * dx;
            w[1] += fdx * dy;
            w[2] += fdx * dz;
            w[3] += fdy * dy;
            w[4] += fdy * dz;
            w[5] += fdz * dz;
        }
    }
}

// one lane's share of atom i's density (returned) and pair energy
template <int TPA, class POS>
__device__ __forceinline__ double energy64_lane(const EamArgs& a, const Smem64& S, const POS& P, int ei, int i,
                                                int lane, double& ep) {
    double acc = 0.0;
    const int nn = __ldg(a.nnbr + i);
    const int* row = a.nbr + (size_t)i * a.maxnbr;
    for (int k = lane; k < nn; k += TPA) {
        const int e = __ldg(row + k);
        const int ej = entry_elem(e);
        double dx, dy, dz;
        P.delta(a, S.sh, e, dx, dy, dz);
        const double rsq = dx * dx + dy * dy + dz * dz;
        if (below(rsq, S.cut_sq[ei * a.ne + ej])) {
            const double rinv = recip_root(rsq);  // as in force64_lane
            double p;
            const int m = knot64_fast(rsq * rinv, a.dr_inv, a.nr - 2, p);
            acc += spl_val(ldg4(a.rho64 + (size_t)(ej * a.ne + ei * a.rho_ei) * a.nr + m), p);
            ep += spl_val(ldg4(a.rphi64 + (size_t)(ei * a.ne + ej) * a.nr + m), p) * rinv;
        }
    }
    return acc;
}

template <int TPA>
__global__ void __launch_bounds__(256) k_density64(EamArgs a) {
    __shared__ Smem64 S;
    S.fill(a);
    const int lane = threadIdx.x % TPA;
    const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / TPA;
    const int stride = (gridDim.x * blockDim.x) / TPA;
    double eacc = 0.0;
    for (int base = 0;; base += stride) {
        const int i = gid + base;
        const bool active = i < a.n;
        if (!__any_sync(0xffffffffu, active)) break;
        double acc = 0.0;
        int ei = 0;
        if (active) {
            Pos64 P;
            P.load(a, i);
            ei = a.elem[i];
            acc = density64_lane<TPA>(a, S, P, ei, i, lane);
        }
#pragma unroll
        for (int o = TPA / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, TPA);
        if (active && lane == 0) {
            double Fv, dFv;
            embed64(a, ei, acc, Fv, dFv);
            a.rho[i] = acc;
            a.dF[i] = dFv;
            eacc += Fv;
        }
    }
    const double v[1] = {eacc};
    __shared__ double tot[1];
    if (block_partials<1>(v, a.partials, 0, &a.sc->counter[1])) {
        final_sums<1>(a.partials, gridDim.x, tot);
        if (threadIdx.x == 0) {
            a.sc->e_embed = tot[0];
            a.sc->counter[1] = 0;
        }
    }
}

// batch: FP64 density per chunk, embedding energy into chunk slot 13
template <int TPA>
__global__ void __launch_bounds__(256) k_density64b(EamArgs a) {
    __shared__ Smem64 S;
    S.fill(a);
    const int lane = threadIdx.x % TPA;
    const int apb = blockDim.x / TPA;
    for (int ch = blockIdx.x; ch < a.nchunk; ch += gridDim.x) {
        if (a.cell_active && !a.cell_active[a.chunk_cell[ch]]) continue;
        const CellGeo& g = a.cells[a.chunk_cell[ch]];
        S.fill_cell(g);
        const int lo = a.chunk_begin[ch], hi = a.chunk_begin[ch + 1];
        double eacc = 0.0;
        for (int i0 = lo; i0 < hi; i0 += apb) {
            const int i = i0 + (int)threadIdx.x / TPA;
            const bool active = i < hi;
            double acc = 0.0;
            int ei = 0;
            if (active) {
                Pos64 P;
                P.load(a, i, g.nb);
                ei = a.elem[i];
                acc = density64_lane<TPA>(a, S, P, ei, i, lane);
            }
#pragma unroll
            for (int o = TPA / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, TPA);
            if (active && lane == 0) {
                double Fv, dFv;
                embed64(a, ei, acc, Fv, dFv);
                a.rho[i] = acc;
                a.dF[i] = dFv;
                eacc += Fv;
            }
        }
        const double v[1] = {eacc};
        chunk_store<1>(v, a.chunk_part + (size_t)ch * kChunkSlots + 13);
    }
}

template <int TPA>
__global__ void __launch_bounds__(256) k_force64(EamArgs a) {
    __shared__ Smem64 S;
    S.fill(a);
    const int lane = threadIdx.x % TPA;
    const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / TPA;
    const int stride = (gridDim.x * blockDim.x) / TPA;
    double ep = 0;
    double w[6] = {0, 0, 0, 0, 0, 0};
    for (int base = 0;; base += stride) {
        const int i = gid + base;
        const bool active = i < a.n;
        if (!__any_sync(0xffffffffu, active)) break;
        double fx = 0, fy = 0, fz = 0;
        if (active) {
            Pos64 P;
            P.load(a, i);
            const int ei = a.elem[i];
            force64_lane<TPA>(a, S, P, ei, __ldg(a.dF + i), i, lane, fx, fy, fz, ep, w);
        }
#pragma unroll
        for (int o = TPA / 2; o > 0; o >>= 1) {
            fx += __shfl_xor_sync(0xffffffffu, fx, o, TPA);
            fy += __shfl_xor_sync(0xffffffffu, fy, o, TPA);
            fz += __shfl_xor_sync(0xffffffffu, fz, o, TPA);
        }
        if (active && lane == 0) {
            a.f[i] = fx;
            a.f[a.n + i] = fy;
            a.f[2 * a.n + i] = fz;
        }
    }
    const double v[7] = {ep, w[0], w[1], w[2], w[3], w[4], w[5]};
    __shared__ double tot[7];
    if (block_partials<7>(v, a.partials, 0, &a.sc->counter[0])) {
        // totals over blocks in a fixed order, and the density pass's
        // embedding energy
        final_sums<7>(a.partials, gridDim.x, tot);
        if (threadIdx.x == 0) {
            a.sc->energy = 0.5 * tot[0] + a.sc->e_embed;
            for (int k = 0; k < 6; k++) a.sc->virial[k] = 0.5 * tot[k + 1];
            a.sc->counter[0] = 0;
        }
    }
}

// batch: FP64 forces per chunk, pair energy and virial into slots 0-6
template <int TPA>
__global__ void __launch_bounds__(256) k_force64b(EamArgs a) {
    __shared__ Smem64 S;
    S.fill(a);
    const int lane = threadIdx.x % TPA;
    const int apb = blockDim.x / TPA;
    for (int ch = blockIdx.x; ch < a.nchunk; ch += gridDim.x) {
        if (a.cell_active && !a.cell_active[a.chunk_cell[ch]]) continue;
        const CellGeo& g = a.cells[a.chunk_cell[ch]];
        S.fill_cell(g);
        const int lo = a.chunk_begin[ch], hi = a.chunk_begin[ch + 1];
        double ep = 0;
        double w[6] = {0, 0, 0, 0, 0, 0};
        for (int i0 = lo; i0 < hi; i0 += apb) {
            const int i = i0 + (int)threadIdx.x / TPA;
            const bool active = i < hi;
            double fx = 0, fy = 0, fz = 0;
            if (active) {
                Pos64 P;
                P.load(a, i, g.nb);
                const int ei = a.elem[i];
                force64_lane<TPA>(a, S, P, ei, __ldg(a.dF + i), i, lane, fx, fy, fz, ep, w);
            }
#pragma unroll
            for (int o = TPA / 2; o > 0; o >>= 1) {
                fx += __shfl_xor_sync(0xffffffffu, fx, o, TPA);
                fy += __shfl_xor_sync(0xffffffffu, fy, o, TPA);
                fz += __shfl_xor_sync(0xffffffffu, fz, o, TPA);
            }
            if (active && lane == 0) {
                a.f[i] = fx;
                a.f[a.n + i] = fy;
                a.f[2 * a.n + i] = fz;
            }
        }
        const double v[7] = {0.5 * ep, 0.5 * w[0], 0.5 * w[1], 0.5 * w[2], 0.5 * w[3], 0.5 * w[4], 0.5 * w[5]};
        chunk_store<7>(v, a.chunk_part + (size_t)ch * kChunkSlots);
    }
}

// input features of the learned preconditioner, per atom: 16 Gaussian radial
// functions exp(-(r - mu_k)^2 / (2 w^2)) fc(r), mu_k = 2.0 + 3.5 k/15 A,
// w = 0.3 A, fc(r) = (1 + cos(pi r / 5.5))/2 for r < 5.5 A, summed over the
// neighbours of each species (A in 0..15, B in 16..31), and the host
// density rho_i (32); FP64 positions, FP32 sums
constexpr int kDescR = 16;
constexpr float kDescRc = 5.5f, kDescW = 0.3f;

// a batch: a block per chunk, whose cell's shifts are in shared memory
template <int TPA, bool BATCH>
__global__ void __launch_bounds__(256) k_descriptors(EamArgs a, float* __restrict__ out) {
    __shared__ Smem64 S;
    S.fill(a);
    const int lane = threadIdx.x % TPA;
    int gid = (blockIdx.x * blockDim.x + threadIdx.x) / TPA, stride = (gridDim.x * blockDim.x) / TPA, end = a.n;
    const int* nb = a.nb;
    if (BATCH) {
        const CellGeo& cell = a.cells[a.chunk_cell[blockIdx.x]];
        S.fill_cell(cell);
        nb = cell.nb;
        gid = a.chunk_begin[blockIdx.x] + (int)threadIdx.x / TPA;
        stride = blockDim.x / TPA;
        end = a.chunk_begin[blockIdx.x + 1];
    }
    const float inv2w2 = 1.f / (2.f * kDescW * kDescW);
    for (int base = 0;; base += stride) {
        const int i = gid + base;
        const bool active = i < end;
        if (!__any_sync(0xffffffffu, active)) break;
        float g[2 * kDescR];
#pragma unroll
        for (int q = 0; q < 2 * kDescR; q++) g[q] = 0.f;
        double rho = 0.0;
        if (active) {
            Pos64 P;
            P.load(a, i, nb);
            const int ei = a.elem[i];
            const int nn = __ldg(a.nnbr + i);
            const int* row = a.nbr + (size_t)i * a.maxnbr;
            for (int k = lane; k < nn; k += TPA) {
                const int e = __ldg(row + k);
                const int ej = entry_elem(e);
                double dx, dy, dz;
                P.delta(a, S.sh, e, dx, dy, dz);
                const double rsq = dx * dx + dy * dy + dz * dz;
                const double rd = root_from(rsq, recip_root(rsq));
                if (below(rsq, S.cut_sq[ei * a.ne + ej])) {
                    double p;
                    const int m = knot64_fast(rd, a.dr_inv, a.nr - 2, p);
                    rho += spl_val(ldg4(a.rho64 + (size_t)(ej * a.ne + ei * a.rho_ei) * a.nr + m), p);
                }
                const float r = (float)rd;
                if (r < kDescRc && ej < 2) {
                    const float fc = 0.5f * (1.f + cosf(3.14159265f * r / kDescRc));
#pragma unroll
                    for (int q = 0; q < kDescR; q++) {
                        const float d = r - (2.0f + 3.5f * (float)q / 15.f);
                        const float v = expf(-d * d * inv2w2) * fc;
                        if (ej == 0)
                            g[q] += v;
                        else
                            g[kDescR + q] += v;
                    }
                }
            }
        }
#pragma unroll
        for (int o = TPA / 2; o > 0; o >>= 1) {
#pragma unroll
            for (int q = 0; q < 2 * kDescR; q++) g[q] += __shfl_xor_sync(0xffffffffu, g[q], o, TPA);
            rho += __shfl_xor_sync(0xffffffffu, rho, o, TPA);
        }
        if (active && lane == 0) {
            float* o = out + (size_t)i * (2 * kDescR + 1);
#pragma unroll
            for (int q = 0; q < 2 * kDescR; q++) o[q] = g[q];
            o[2 * kDescR] = (float)rho;
        }
    }
}

template <int TPA>
__global__ void __launch_bounds__(256) k_energy64(EamArgs a) {
    __shared__ Smem64 S;
    S.fill(a);
    const int lane = threadIdx.x % TPA;
    const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / TPA;
    const int stride = (gridDim.x * blockDim.x) / TPA;
    double ep = 0.0, eacc = 0.0;
    for (int base = 0;; base += stride) {
        const int i = gid + base;
        const bool active = i < a.n;
        if (!__any_sync(0xffffffffu, active)) break;
        double acc = 0.0;
        int ei = 0;
        if (active) {
            Pos64 P;
            P.load(a, i);
            ei = a.elem[i];
            acc = energy64_lane<TPA>(a, S, P, ei, i, lane, ep);
        }
#pragma unroll
        for (int o = TPA / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, TPA);
        if (active && lane == 0) {
            double Fv, dFv;
            embed64(a, ei, acc, Fv, dFv);
            eacc += Fv;
        }
    }
    const double v[1] = {eacc + 0.5 * ep};
    __shared__ double tot[1];
    if (block_partials<1>(v, a.partials, 0, &a.sc->counter[2])) {
        final_sums<1>(a.partials, gridDim.x, tot);
        if (threadIdx.x == 0) {
            a.sc->energy = tot[0];
            a.sc->counter[2] = 0;
        }
    }
}

// batch: FP64 energy of every cell (the line-search energies of mixed
// batches), chunk sums into slot 0 of the chunk partials
template <int TPA>
__global__ void __launch_bounds__(256) k_energy64b(EamArgs a) {
    __shared__ Smem64 S;
    S.fill(a);
    const int lane = threadIdx.x % TPA;
    const int apb = blockDim.x / TPA;
    for (int ch = blockIdx.x; ch < a.nchunk; ch += gridDim.x) {
        if (a.cell_active && !a.cell_active[a.chunk_cell[ch]]) continue;
        const CellGeo& g = a.cells[a.chunk_cell[ch]];
        S.fill_cell(g);
        const int lo = a.chunk_begin[ch], hi = a.chunk_begin[ch + 1];
        double ep = 0.0, eacc = 0.0;
        for (int i0 = lo; i0 < hi; i0 += apb) {
            const int i = i0 + (int)threadIdx.x / TPA;
            const bool active = i < hi;
            double acc = 0.0;
            int ei = 0;
            if (active) {
                Pos64 P;
                P.load(a, i, g.nb);
                ei = a.elem[i];
                acc = energy64_lane<TPA>(a, S, P, ei, i, lane, ep);
            }
#pragma unroll
            for (int o = TPA / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, TPA);
            if (active && lane == 0) {
                double Fv, dFv;
                embed64(a, ei, acc, Fv, dFv);
                eacc += Fv;
            }
        }
        const double v[1] = {eacc + 0.5 * ep};
        chunk_store<1>(v, a.chunk_part + (size_t)ch * kChunkSlots);
    }
}

template <int TPA>
static int grid64(mappg_sys* s) {
    return grid_for(s, (long long)s->n * TPA, 256);
}

#define MAPPG_TPA64(KERNEL)                                                                    \
    switch (s->tpa) {                                                                          \
        case 4: KERNEL<4><<<grid64<4>(s), 256, 0, s->stream>>>(a); break;                     \
        case 16: KERNEL<16><<<grid64<16>(s), 256, 0, s->stream>>>(a); break;                  \
        case 32: KERNEL<32><<<grid64<32>(s), 256, 0, s->stream>>>(a); break;                  \
        default: KERNEL<8><<<grid64<8>(s), 256, 0, s->stream>>>(a); break;                    \
    }

void launch_cells_done(mappg_sys* s, const EamArgs& a, int what);  // eam32.cu

// FP64 batch passes take a block per chunk: a chunk is 50-100 us of FP64
// work, so the hardware's own assignment of blocks to free SMs beats a fixed
// share of the chunks per block (10 relaxation steps of 64 cells with 128-atom
// chunks: 48.5 -> 47.9 ms).  They are bound by the FP64 pipe: the image shifts
// of a cell are a table in shared memory (most warps of a batch hold a pair
// that reaches an image, and forming its shift took 12 operations and
// conversions), 1/r starts from an FP32 root, the knot is cut out of the
// mantissa.  330,000 atoms: energy 1.74 -> 1.28 ms, density 1.61 -> 1.17,
// forces 2.68 -> 2.23; energy of a single cell of 253,000 1.04 -> 0.85.

void launch_density_only(mappg_sys* s) {
    EamArgs a = eam_args(s);
    if (s->precision == MAPPG_MIXED && !s->force64) {
        launch_density32(s, a);
        return;
    }
    if (s->ncell > 1) {
        k_density64b<8><<<s->nchunk, 256, 0, s->stream>>>(a);
    } else if (s->own_ent) {
        launch_pair_density64(s, a);
    } else {
        MAPPG_TPA64(k_density64)
    }
    MAPPG_CUDA(cudaGetLastError());
}

// ForceFieldMD::force_calc (ff_md.cpp:138-144): components without a
// degree of freedom carry no force
template <class T>
__global__ void k_dof_mask(int n, const uint8_t* __restrict__ dof, T* __restrict__ f) {
    dep_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned d = dof[i];
        if (d == 7u) continue;
        for (int c = 0; c < 3; c++)
            if (!((d >> c) & 1u)) f[(size_t)c * n + i] = T(0);
    }
}

void launch_dof_mask(mappg_sys* s, bool f32) {
    if (!s->dof) return;
    if (f32)
        launch_dep(s->stream, k_dof_mask<float>, grid_for(s, s->n, 256), 256, 0, s->n, s->dof, s->f32);
    else
        launch_dep(s->stream, k_dof_mask<double>, grid_for(s, s->n, 256), 256, 0, s->n, s->dof, s->f);
    MAPPG_CUDA(cudaGetLastError());
}

void launch_force_only(mappg_sys* s) {
    EamArgs a = eam_args(s);
    if (s->precision == MAPPG_MIXED && !s->force64) {
        launch_force32(s, a);
        launch_dof_mask(s, true);
        s->f_is_f32 = true;
        return;
    }
    if (s->ncell > 1) {
        k_force64b<8><<<s->nchunk, 256, 0, s->stream>>>(a);
        MAPPG_CUDA(cudaGetLastError());
        launch_cells_done(s, a, 0);
    } else if (s->own_ent) {
        launch_pair_force64(s, a);
    } else {
        MAPPG_TPA64(k_force64)
        MAPPG_CUDA(cudaGetLastError());
    }
    launch_dof_mask(s, false);
    s->f_is_f32 = false;
}

void launch_force(mappg_sys* s) {
    launch_density_only(s);
    launch_force_only(s);
}

// preconditioner features of every atom (bin order), n x 33 floats
void launch_descriptors(mappg_sys* s, float* out) {
    EamArgs a = eam_args(s);
    if (s->ncell > 1)
        k_descriptors<8, true><<<s->nchunk, 256, 0, s->stream>>>(a, out);
    else
        k_descriptors<8, false><<<grid64<8>(s), 256, 0, s->stream>>>(a, out);
    MAPPG_CUDA(cudaGetLastError());
}

// FP64 density and force passes whose outputs, partial sums and device
// scalars are the ones in `a` (mappg_sys_force_noalloc points them at its
// scratch); launches only, no allocation
void launch_force64_args(mappg_sys* s, const EamArgs& a) {
    MAPPG_TPA64(k_density64)
    MAPPG_TPA64(k_force64)
    MAPPG_CUDA(cudaGetLastError());
}

// loads every instantiation launch_force64_args can pick onto the current
// device, so that later launches do no module loading of their own
void preload_force64() {
    cudaFuncAttributes fa;
    MAPPG_CUDA(cudaFuncGetAttributes(&fa, k_density64<4>));
    MAPPG_CUDA(cudaFuncGetAttributes(&fa, k_density64<8>));
    MAPPG_CUDA(cudaFuncGetAttributes(&fa, k_density64<16>));
    MAPPG_CUDA(cudaFuncGetAttributes(&fa, k_density64<32>));
    MAPPG_CUDA(cudaFuncGetAttributes(&fa, k_force64<4>));
    MAPPG_CUDA(cudaFuncGetAttributes(&fa, k_force64<8>));
    MAPPG_CUDA(cudaFuncGetAttributes(&fa, k_force64<16>));
    MAPPG_CUDA(cudaFuncGetAttributes(&fa, k_force64<32>));
}

// FP64 energy in either precision (line searches of mixed systems compare
// FP64 energies): sc->energy for one cell, CellMd::energy per cell of a batch
void launch_energy64(mappg_sys* s) {
    EamArgs a = eam_args(s);
    if (s->ncell > 1) {
        k_energy64b<8><<<s->nchunk, 256, 0, s->stream>>>(a);
        MAPPG_CUDA(cudaGetLastError());
        launch_cells_done(s, a, 1);
        return;
    }
    MAPPG_TPA64(k_energy64)
    MAPPG_CUDA(cudaGetLastError());
}

void launch_energy(mappg_sys* s) {
    EamArgs a = eam_args(s);
    if (s->precision == MAPPG_MIXED) {
        launch_energy32(s, a);
        return;
    }
    if (s->own_ent) {
        launch_pair_energy64(s, a);
        return;
    }
    MAPPG_TPA64(k_energy64)
    MAPPG_CUDA(cudaGetLastError());
}

}  // namespace mappg
