// FP64 density and forces of one cell with every pair computed once.
//
// GB300 runs 64 FP32 operations for one FP64 operation, so the FP64 passes
// are bound by the FP64 pipe while memory idles (k_density64 + k_force64: 86 %
// of the pipe, 1 % of DRAM).  Over full rows each pair is computed four times:
// by both atoms, in both passes.  Here the builder splits a row into the pairs
// the atom owns and the others (pair_owned), and the passes are
//   k_pair64    per owned pair: geometry, 1/r, both densities and their
//               derivatives, r phi; the two densities and a record
//               (A, B, C, dx) go to memory, where
//               f = (A + F'_owner B + F'_other C) dx is the force on the owner
//   k_rho64     rho_i over own and other pairs (one addition each), F, F'
//   k_gather64  f_i over own and other pairs; the virial over own ones
// ~37 FP64 operations an entry instead of ~80, and ~1.9 KB written and ~3.7 KB
// read per atom, which the memory has room for.  An other pair's record lies
// with its owner; the builder's k_link64 finds the slot once per list.
// Sums have a fixed order (lane-strided over one list, then the other), no
// atomics.
// Density + force against the full rows: 4,000 atoms 63.2 -> 41.1 us, 16,384
// 186 -> 100, 256,000 2,255 -> 1,137.  The FP64 pipe bounds them still: of it
// k_pair64 takes 89 %, k_gather64 89 and k_rho64 80, of DRAM 11, 24 and 36
// (442,368 atoms).
#include <math.h>

#include <algorithm>

#include "eam_common.cuh"
#include "pos64.cuh"

namespace mappg {

// densities of a pair outside the cutoff: a NaN pattern that no table gives
constexpr unsigned long long kOutside = 0xfff8dead00000000ull;
__device__ __forceinline__ bool is_outside(double v) {
    return (unsigned long long)__double_as_longlong(v) == kOutside;
}

__device__ __forceinline__ double spl_val(const Dbl4& c, double p) { return fma(fma(fma(c.w, p, c.z), p, c.y), p, c.x); }

// ENERGY: the densities and the pair energy only (line-search trials)
template <int TPA, bool ENERGY>
__global__ void __launch_bounds__(256) k_pair64(const __grid_constant__ EamArgs a) {
    dep_wait();
    __shared__ Smem64 S;
    S.fill(a);
    const int lane = threadIdx.x % TPA;
    const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / TPA;
    const int stride = (gridDim.x * blockDim.x) / TPA;
    const double dri = a.dr_inv;
    double ep = 0.0;
    for (int i = gid; i < a.n; i += stride) {
        const size_t base = (size_t)i * a.maxnbr;
        const int no = __ldg(a.nown + i);
        Pos64 P;
        P.load(a, i);
        const int ei = a.elem[i];
        for (int q = lane; q < no; q += TPA) {
            const int e = __ldg(a.own_ent + base + q);
            const int ej = entry_elem(e);
            double dx, dy, dz;
            P.delta(a, S.sh, e, dx, dy, dz);
            const double rsq = dx * dx + dy * dy + dz * dz;
            double2 rho = {__longlong_as_double((long long)kOutside), 0.0};
            if (below(rsq, S.cut_sq[ei * a.ne + ej])) {
                const double rinv = recip_root(rsq);
                double p;
                // (a trial's energy takes r = rsq/r, as those over full rows)
                const int m = knot64_fast(ENERGY ? rsq * rinv : root_from(rsq, rinv), dri, a.nr - 2, p);
                if (ENERGY) {
                    rho.x = spl_val(ldg4(a.rho64 + (size_t)(ej * a.ne + ei * a.rho_ei) * a.nr + m), p);
                    rho.y = ej == ei ? rho.x : spl_val(ldg4(a.rho64 + (size_t)(ei * a.ne + ej * a.rho_ei) * a.nr + m), p);
                    ep += spl_val(ldg4(a.rphi64 + (size_t)(ei * a.ne + ej) * a.nr + m), p) * rinv;
                    a.pair_rho[base + q] = rho;
                    continue;
                }
                double di, dj, z, dz_;
                spl_both(ldg4(a.rho64 + (size_t)(ej * a.ne + ei * a.rho_ei) * a.nr + m), p, rho.x, di);
                rho.y = rho.x;
                dj = di;
                if (ej != ei) spl_both(ldg4(a.rho64 + (size_t)(ei * a.ne + ej * a.rho_ei) * a.nr + m), p, rho.y, dj);
                spl_both(ldg4(a.rphi64 + (size_t)(ei * a.ne + ej) * a.nr + m), p, z, dz_);
                const double phi = z * rinv, g = -rinv * dri;
                ep += phi;
                double2* rec = a.pair_rec + 3 * (base + q);
                rec[0] = make_double2(-(fma(dz_, dri, -phi) * rinv) * rinv, di * g);
                rec[1] = make_double2(dj * g, dx);
                rec[2] = make_double2(dy, dz);
            }
            a.pair_rho[base + q] = rho;
        }
    }
    const double v[1] = {ep};
    const double t = block_sums<1>(v);
    if (threadIdx.x == 0) a.partials[blockIdx.x * kRedSlots] = t;
}

// bit t of a.pair_mask[(i * TPA + lane) * 2 + (0: own, 1: other)]: this
// lane's t-th pair of the list is inside the cutoff (lists of at most
// 32 TPA pairs; longer ones are tested again)
// ENERGY: the densities stay here, and the last block adds up the energy
template <int TPA, bool ENERGY>
__global__ void __launch_bounds__(256) k_rho64(const __grid_constant__ EamArgs a, int rows_pair) {
    dep_wait();
    const int lane = threadIdx.x % TPA;
    const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / TPA;
    const int stride = (gridDim.x * blockDim.x) / TPA;
    double eacc = 0.0;
    for (int base = 0;; base += stride) {
        const int i = gid + base;
        const bool active = i < a.n;
        if (!__any_sync(0xffffffffu, active)) break;
        double acc = 0.0;
        if (active) {
            const size_t row = (size_t)i * a.maxnbr;
            const int no = __ldg(a.nown + i), nr = __ldg(a.nother + i);
            unsigned own = 0u, oth = 0u;
            int t = 0;
            for (int q = lane; q < no; q += TPA, t++) {
                const double v = a.pair_rho[row + q].x;
                if (!is_outside(v)) {
                    acc += v;
                    if (t < 32) own |= 1u << t;
                }
            }
            t = 0;
            for (int q = lane; q < nr; q += TPA, t++) {
                const unsigned slot = __ldg(a.other_slot + row + q);
                const double2 v = slot == kNoSlot ? make_double2(__longlong_as_double((long long)kOutside), 0.0)
                                                  : a.pair_rho[slot];
                if (!is_outside(v.x)) {
                    acc += v.y;
                    if (t < 32) oth |= 1u << t;
                }
            }
            if (!ENERGY)
                *reinterpret_cast<uint2*>(a.pair_mask + ((size_t)i * TPA + lane) * 2) = make_uint2(own, oth);
        }
#pragma unroll
        for (int o = TPA / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, TPA);
        if (active && lane == 0) {
            double Fv, dFv;
            embed64(a, a.elem[i], acc, Fv, dFv);
            if (!ENERGY) {
                a.rho[i] = acc;
                a.dF[i] = dFv;
            }
            eacc += Fv;
        }
    }
    const double v[1] = {eacc};
    const double t = block_sums<1>(v);
    if (threadIdx.x == 0) a.partials[blockIdx.x * kRedSlots + 7] = t;
    if (ENERGY) {
        __shared__ double tot[8];
        if (last_block(&a.sc->counter[2])) {
            final_sums<8>(a.partials, threadIdx.x % 8 == 0 ? rows_pair : threadIdx.x % 8 == 7 ? (int)gridDim.x : 0, tot);
            if (threadIdx.x == 0) {
                a.sc->energy = tot[0] + tot[7];
                a.sc->counter[2] = 0;
            }
        }
    }
}

template <int TPA>
__global__ void __launch_bounds__(256) k_gather64(const __grid_constant__ EamArgs a, int rows_pair, int rows_rho) {
    dep_wait();
    const int lane = threadIdx.x % TPA;
    const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / TPA;
    const int stride = (gridDim.x * blockDim.x) / TPA;
    double w[6] = {0, 0, 0, 0, 0, 0};
    for (int base = 0;; base += stride) {
        const int i = gid + base;
        const bool active = i < a.n;
        if (!__any_sync(0xffffffffu, active)) break;
        double fx = 0, fy = 0, fz = 0;
        if (active) {
            const size_t row = (size_t)i * a.maxnbr;
            const int no = __ldg(a.nown + i), nr = __ldg(a.nother + i);
            const double dFi = a.dF[i];
            const uint2 mask = *reinterpret_cast<const uint2*>(a.pair_mask + ((size_t)i * TPA + lane) * 2);
            auto own = [&](int q) {
                const double dFj = a.dF[entry_j(__ldg(a.own_ent + row + q))];
                const double2* rec = a.pair_rec + 3 * (row + q);
                const double2 r0 = rec[0], r1 = rec[1], r2 = rec[2];
                const double f = fma(dFj, r1.x, fma(dFi, r0.y, r0.x));
                const double gx = f * r1.y, gy = f * r2.x, gz = f * r2.y;
                fx += gx;
                fy += gy;
                fz += gz;
                w[0] = fma(gx, r1.y, w[0]);
                w[1] = fma(gx, r2.x, w[1]);
                w[2] = fma(gx, r2.y, w[2]);
                w[3] = fma(gy, r2.x, w[3]);
                w[4] = fma(gy, r2.y, w[4]);
                w[5] = fma(gz, r2.y, w[5]);
            };
            auto other = [&](int q) {
                const double dFj = a.dF[entry_j(__ldg(a.other_ent + row + q))];
                const double2* rec = a.pair_rec + 3 * (size_t)__ldg(a.other_slot + row + q);
                const double2 r0 = rec[0], r1 = rec[1], r2 = rec[2];
                const double f = -fma(dFi, r1.x, fma(dFj, r0.y, r0.x));
                fx = fma(f, r1.y, fx);
                fy = fma(f, r2.x, fy);
                fz = fma(f, r2.y, fz);
            };
            if (nr <= 32 * TPA) {
                for (unsigned b = mask.y; b; b &= b - 1u) other(lane + (__ffs(b) - 1) * TPA);
            } else {
                for (int q = lane; q < nr; q += TPA) {
                    const unsigned slot = __ldg(a.other_slot + row + q);
                    if (slot != kNoSlot && !is_outside(a.pair_rho[slot].x)) other(q);
                }
            }
            if (no <= 32 * TPA)
                for (unsigned b = mask.x; b; b &= b - 1u) own(lane + (__ffs(b) - 1) * TPA);
            else
                for (int q = lane; q < no; q += TPA)
                    if (!is_outside(a.pair_rho[row + q].x)) own(q);
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
    // virial in slots 1-6; the last block, or the kernel that closes an MD
    // step, adds those up with the pair energy (slot 0, k_pair64's blocks) and
    // the embedding energy (slot 7, k_rho64's)
    const double v[8] = {0.0, w[0], w[1], w[2], w[3], w[4], w[5], 0.0};
    const double t = block_sums<8>(v);
    if (threadIdx.x >= 1 && threadIdx.x < 7) a.partials[blockIdx.x * kRedSlots + threadIdx.x] = t;
    if (a.defer) return;
    if (last_block(&a.sc->counter[0]))
        store_totals(a.partials, PassRows{rows_pair, (int)gridDim.x, rows_rho, 1.0}, a.sc, &a.sc->counter[0]);
}

// the record slot of each pair that another atom owns, by the mirrored entry
// in the owner's list.  Eight lanes search one list, 64 entries in two
// 16-byte loads each (a list is rarely longer), so a warp has four lists in
// flight; `parts` warps share an atom's pairs in a small system.  One list
// per warp in 4-byte loads took 698 us at 256,000 atoms and 25 at 4,000,
// 290 and ~20 so
__global__ void __launch_bounds__(256) k_link64(int n, int cap, int parts, const int* __restrict__ own_ent,
                                                const int* __restrict__ nown, const int* __restrict__ other_ent,
                                                const int* __restrict__ nother, const uint8_t* __restrict__ elem,
                                                unsigned* __restrict__ other_slot, const DevScalars* sc) {
    dep_wait();
    if (!sc->rebuild) return;
    const int lane = threadIdx.x & 31, g = lane >> 3, l = lane & 7;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n * parts; w += nw) {
        const int i = w / parts;
        const unsigned row = (unsigned)i * cap;  // slots fit 32 bits
        const int nr = __ldg(nother + i), ei = elem[i];
        for (int q0 = 4 * (w - i * parts); q0 < nr; q0 += 4 * parts) {
            const int q = min(q0 + g, nr - 1);
            const int e = __ldg(other_ent + row + q);
            const int want = mirrored_entry(e, i, ei);
            const unsigned rj = (unsigned)entry_j(e) * cap;
            const int no = __ldg(nown + entry_j(e));
            int at = cap;
            // rows start on 128 bytes and hold whole 32s; what lies beyond
            // a list's end matches beyond it
            for (int k0 = 0;; k0 += 64) {
                const int k = k0 + 4 * l;
                const int4 v = __ldg(reinterpret_cast<const int4*>(own_ent + rj + k));
                const int4 u = k0 + 32 < cap ? __ldg(reinterpret_cast<const int4*>(own_ent + rj + k + 32)) : v;
                int c = cap;
                if (u.w == want) c = k + 35;
                if (u.z == want) c = k + 34;
                if (u.y == want) c = k + 33;
                if (u.x == want) c = k + 32;
                if (v.w == want) c = k + 3;
                if (v.z == want) c = k + 2;
                if (v.y == want) c = k + 1;
                if (v.x == want) c = k;
                c = min(c, at);
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) c = min(c, __shfl_xor_sync(0xffffffffu, c, o));
                at = c;
                if (k0 + 64 >= cap || !__any_sync(0xffffffffu, at >= no && k0 + 64 < no)) break;
            }
            if (l == 0) other_slot[row + q] = at < no ? rj + at : kNoSlot;
        }
    }
}

void launch_link64(mappg_sys* s) {
    const int parts = s->n < 64 * s->sm_count ? 4 : 1;  // fill the warps that the SMs hold
    launch_dep(s->stream, k_link64, grid_for(s, 32LL * s->n * parts, 256), 256, 0, s->n, s->maxnbr, parts, s->own_ent,
               s->nown, s->other_ent, s->nother, s->elem, s->other_slot, s->sc);
    MAPPG_CUDA(cudaGetLastError());
}

template <int TPA>
static void pair_density(mappg_sys* s, const EamArgs& a, int grid) {
    launch_dep(s->stream, k_pair64<TPA, false>, grid, 256, 0, a);
    launch_dep(s->stream, k_rho64<TPA, false>, grid, 256, 0, a, grid);
}

template <int TPA>
static void pair_energy(mappg_sys* s, const EamArgs& a, int grid) {
    launch_dep(s->stream, k_pair64<TPA, true>, grid, 256, 0, a);
    launch_dep(s->stream, k_rho64<TPA, true>, grid, 256, 0, a, grid);
}

template <int TPA>
static void pair_force(mappg_sys* s, const EamArgs& a, int grid) {
    s->pass_rows = PassRows{grid, grid, grid, 1.0};
    launch_dep(s->stream, k_gather64<TPA>, grid, 256, 0, a, grid, grid);
}

#define MAPPG_PAIR64(FN)                                                  \
    {                                                                     \
        const int grid = grid_for(s, (long long)s->n * s->tpa, 256);      \
        switch (s->tpa) {                                                 \
            case 4: FN<4>(s, a, grid); break;                             \
            case 16: FN<16>(s, a, grid); break;                           \
            case 32: FN<32>(s, a, grid); break;                           \
            default: FN<8>(s, a, grid); break;                            \
        }                                                                 \
        MAPPG_CUDA(cudaGetLastError());                                   \
    }

void launch_pair_density64(mappg_sys* s, const EamArgs& a) MAPPG_PAIR64(pair_density)
void launch_pair_force64(mappg_sys* s, const EamArgs& a) MAPPG_PAIR64(pair_force)
void launch_pair_energy64(mappg_sys* s, const EamArgs& a) MAPPG_PAIR64(pair_energy)

}  // namespace mappg
