// Device state of one periodic cell, coordinate transforms, binning and the
// full neighbour-list build.
//
// The list holds, for every atom i, every periodic image j' = x_j + n*H
// (j' != i) with |x_i - x_j'|^2 < (cut_ij + skin)^2, the same set that
// NeighborMD::create_list (neighbor_md.cpp:82-152) finds in full mode
// (pair_wise = false) over the ghost images of Update::list
// (exchange.h:833-875).  Candidates come from the 27 bins around atom i; an
// FP32 distance on bin-relative positions settles every pair outside a thin
// band around the cutoff, and pairs inside the band are decided with the
// reference's FP64 arithmetic: x = S2X(s) (xmath.h:2636-2658) of the wrapped
// fractional coordinate, images at S2X(s_j + n), RSQ = d0^2 + (d1^2 + d2^2)
// (xmath.h:2464-2510), no fused multiply-adds.
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <numeric>
#include <type_traits>
#include <vector>

#include "eam_common.cuh"

namespace mappg {

// ------------------------------------------------------------------ box
// Atoms::update_H  atoms.cpp:187-194 with the lower-triangular inverse,
// depth and determinant of xmath.h:1403-1480,2399-2415
static void box_from_H(Box& b, const double* H9) {
    memcpy(b.H, H9, sizeof(double) * 9);
    double(*H)[3] = b.H;
    double(*B)[3] = b.B;
    memset(B, 0, sizeof(double) * 9);
    B[0][0] = 1.0 / H[0][0];
    B[1][1] = 1.0 / H[1][1];
    B[1][0] = -B[1][1] * (B[0][0] * H[1][0]);
    B[2][2] = 1.0 / H[2][2];
    B[2][1] = -B[2][2] * (B[1][1] * H[2][1]);
    B[2][0] = -B[2][2] * (B[0][0] * H[2][0] + B[1][0] * H[2][1]);
    b.vol = H[0][0] * (H[1][1] * H[2][2]);
    b.depth_inv[0] = sqrt(B[0][0] * B[0][0] + (B[1][0] * B[1][0] + B[2][0] * B[2][0]));
    b.depth_inv[1] = sqrt(B[1][1] * B[1][1] + B[2][1] * B[2][1]);
    b.depth_inv[2] = fabs(B[2][2]);
    b.h6[0] = H[0][0]; b.h6[1] = H[1][0]; b.h6[2] = H[2][0];
    b.h6[3] = H[1][1]; b.h6[4] = H[2][1]; b.h6[5] = H[2][2];
    b.b6[0] = B[0][0]; b.b6[1] = B[1][0]; b.b6[2] = B[2][0];
    b.b6[3] = B[1][1]; b.b6[4] = B[2][1]; b.b6[5] = B[2][2];
}

void sys_set_box(mappg_sys* s, const double* H) {
    if (!(H[0] > 0 && H[4] > 0 && H[8] > 0) || H[1] != 0.0 || H[2] != 0.0 || H[5] != 0.0)
        throw Error{MAPPG_ERR_ARG, "H must be lower triangular with a positive diagonal"};
    box_from_H(s->box, H);
    double nbv[3];
    for (int d = 0; d < 3; d++) {
        double cs = s->max_cut * s->box.depth_inv[d];
        if (!(cs < 1.0))
            throw Error{MAPPG_ERR_GEOM, "box thinner than cutoff+skin along dimension " + std::to_string(d) +
                                            ": multi-layer periodic images are not supported"};
        int nb = (int)(1.0 / (cs * (1.0 + 1e-12)));
        nb = std::max(1, std::min(nb, 1023));
        s->nb[d] = nb;
        nbv[d] = 1.0 / nb;
    }
    s->nbins = s->nb[0] * s->nb[1] * s->nb[2];
    // scaled bin frame: s'_d = s_d * 8 nb_d; Cartesian dx = dx' G with
    // G_dk = H_dk / (8 nb_d), kept as head + tail
    Frame& fr = s->frame;
    fr.ortho = (H[3] == 0.0 && H[6] == 0.0 && H[7] == 0.0) ? 1 : 0;
    for (int d = 0; d < 3; d++)
        for (int k = 0; k < 3; k++) {
            double g = s->box.H[d][k] / (8.0 * s->nb[d]);
            fr.G[d][k] = (float)g;
            fr.Glo[d][k] = (float)(g - (double)fr.G[d][k]);
        }
    // image shifts n H, indexed by image code (n0+1) + 3(n1+1) + 9(n2+1)
    for (int c = 0; c < 27; c++) {
        int d[3] = {c % 3 - 1, (c / 3) % 3 - 1, c / 9 - 1};
        for (int k = 0; k < 3; k++) {
            double sh = 0.0;
            for (int q = 0; q < 3; q++) sh += d[q] * s->box.H[q][k];
            s->shift[c][k] = sh;
        }
    }
    double pmax = s->skin;
    for (int q = 0; q < 3; q++) {
        double l = 0;
        for (int k = 0; k < 3; k++) l += s->box.H[q][k] * s->box.H[q][k];
        pmax += sqrt(l) * nbv[q];
    }
    double csk = 0;
    for (int i = 0; i < s->ne * s->ne; i++) csk = std::max(csk, s->cut_sk_sq[i]);
    s->band = 2e-5 * (csk + pmax * pmax);
    s->built = false;
    s->list_box = false;
}

// a batch: every cell gets its own box, bins (a block of global bin ids) and
// frame; the system-level box fields keep cell 0's for code that reads them
static void chunk_cells(mappg_sys* s);

void sys_set_cells(mappg_sys* s, int ncell, const int* natoms, const double* H) {
    s->ncell = ncell;
    s->cells.assign(ncell, CellGeo());
    s->cell_begin.assign(ncell + 1, 0);
    double band = 0.0;
    int bins = 0;
    bool all_ortho = true;
    for (int c = 0; c < ncell; c++) {
        sys_set_box(s, H + 9 * (size_t)c);
        CellGeo& g = s->cells[c];
        memcpy(g.h6, s->box.h6, sizeof(g.h6));
        memcpy(g.b6, s->box.b6, sizeof(g.b6));
        const double S[3] = {8.0 * s->nb[0], 8.0 * s->nb[1], 8.0 * s->nb[2]};
        g.bs[0] = g.b6[0] * S[0];
        g.bs[1] = g.b6[1] * S[0];
        g.bs[2] = g.b6[2] * S[0];
        g.bs[3] = g.b6[3] * S[1];
        g.bs[4] = g.b6[4] * S[1];
        g.bs[5] = g.b6[5] * S[2];
        memcpy(g.G, s->frame.G, sizeof(g.G));
        memcpy(g.Glo, s->frame.Glo, sizeof(g.Glo));
        for (int d = 0; d < 3; d++) g.nb[d] = s->nb[d];
        g.bin_base = bins;
        g.ortho = s->frame.ortho;
        all_ortho = all_ortho && g.ortho != 0;
        bins += s->nbins;
        band = std::max(band, s->band);
        s->cell_begin[c + 1] = s->cell_begin[c] + natoms[c];
        g.begin = s->cell_begin[c];
        g.end = s->cell_begin[c + 1];
    }
    sys_set_box(s, H);  // cell 0
    s->nbins = bins;
    s->band = band;
    s->cells_ortho = all_ortho;
    chunk_cells(s);
}

// chunks of at most s->chunk_atoms atoms, never across cells (host arrays)
static void chunk_cells(mappg_sys* s) {
    const int ncell = s->ncell;
    s->chunk_begin_h.clear();
    s->cell_chunk_h.assign(ncell + 1, 0);
    std::vector<int> chunk_cell;
    for (int c = 0; c < ncell; c++) {
        for (int a = s->cell_begin[c]; a < s->cell_begin[c + 1]; a += s->chunk_atoms) {
            s->chunk_begin_h.push_back(a);
            chunk_cell.push_back(c);
        }
        s->cell_chunk_h[c + 1] = (int)s->chunk_begin_h.size();
    }
    s->nchunk = (int)s->chunk_begin_h.size();
    s->chunk_begin_h.push_back(s->cell_begin[ncell]);
    s->cells_chunk_cell_h = chunk_cell;
}

// device copies of the chunk arrays and the per-chunk sums
static void upload_chunks(mappg_sys* s) {
    const int nc = s->ncell, nk = s->nchunk;
    void* old[] = {s->chunk_begin, s->chunk_cell, s->cell_chunk, s->chunk_part, s->chunk_disp};
    for (void* p : old)
        if (p) cudaFree(p);
    MAPPG_CUDA(cudaMalloc((void**)&s->chunk_begin, sizeof(int) * (nk + 1)));
    MAPPG_CUDA(cudaMalloc((void**)&s->chunk_cell, sizeof(int) * nk));
    MAPPG_CUDA(cudaMalloc((void**)&s->cell_chunk, sizeof(int) * (nc + 1)));
    MAPPG_CUDA(cudaMalloc((void**)&s->chunk_part, sizeof(double) * kChunkSlots * (size_t)nk));
    MAPPG_CUDA(cudaMalloc((void**)&s->chunk_disp, sizeof(double) * 4 * (size_t)nk));
    MAPPG_CUDA(cudaMemsetAsync(s->chunk_part, 0, sizeof(double) * kChunkSlots * (size_t)nk, s->stream));
    MAPPG_CUDA(cudaMemsetAsync(s->chunk_disp, 0, sizeof(double) * 4 * (size_t)nk, s->stream));
    MAPPG_CUDA(cudaMemcpyAsync(s->chunk_begin, s->chunk_begin_h.data(), sizeof(int) * (nk + 1), cudaMemcpyHostToDevice,
                               s->stream));
    MAPPG_CUDA(cudaMemcpyAsync(s->chunk_cell, s->cells_chunk_cell_h.data(), sizeof(int) * nk, cudaMemcpyHostToDevice,
                               s->stream));
    MAPPG_CUDA(cudaMemcpyAsync(s->cell_chunk, s->cell_chunk_h.data(), sizeof(int) * (nc + 1), cudaMemcpyHostToDevice,
                               s->stream));
    MAPPG_CUDA(cudaStreamSynchronize(s->stream));
}

void sys_rechunk(mappg_sys* s, int chunk_atoms) {
    if (s->ncell <= 1) return;
    if (chunk_atoms < 32) throw Error{MAPPG_ERR_ARG, "chunks hold at least 32 atoms"};
    if (chunk_atoms == s->chunk_atoms) return;
    s->chunk_atoms = chunk_atoms;
    chunk_cells(s);
    upload_chunks(s);
}

int grid_for(mappg_sys* s, long long threads, int block) {
    long long g = (threads + block - 1) / block;
    long long cap = (long long)s->sm_count * 8;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    if (g > kMaxBlocks) g = kMaxBlocks;
    return (int)g;
}

// ------------------------------------------------------------------ kernels
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }

struct Geo {
    double h6[6], b6[6];
    double bs[6];  // b6 with each column scaled by 8 nb_d: x -> s' directly
    int nb[3];
};

static Geo make_geo(mappg_sys* s) {
    Geo g;
    memcpy(g.h6, s->box.h6, sizeof(g.h6));
    memcpy(g.b6, s->box.b6, sizeof(g.b6));
    for (int d = 0; d < 3; d++) g.nb[d] = s->nb[d];
    const double S0 = 8.0 * s->nb[0], S1 = 8.0 * s->nb[1], S2 = 8.0 * s->nb[2];
    g.bs[0] = g.b6[0] * S0;
    g.bs[1] = g.b6[1] * S0;
    g.bs[2] = g.b6[2] * S0;
    g.bs[3] = g.b6[3] * S1;
    g.bs[4] = g.b6[4] * S1;
    g.bs[5] = g.b6[5] * S2;
    return g;
}

// one wrap of X2S (xmath.h:2660-2700): ++/-- until in [0,1); bounded
__device__ __forceinline__ double wrap01(double v, int* bad) {
    int it = 0;
    while (v < 0.0 && it < 64) {
        v = dadd(v, 1.0);
        it++;
    }
    while (v >= 1.0 && it < 64) {
        v = dsub(v, 1.0);
        it++;
    }
    if (it >= 64 || v != v) {
        *bad = 1;
        v = 0.0;
    }
    return v;
}

__device__ __forceinline__ void s2x(const double* h, double s0, double s1, double s2, double& x0, double& x1,
                                    double& x2) {
    x0 = dadd(dmul(h[0], s0), dadd(dmul(h[1], s1), dmul(h[2], s2)));
    x1 = dadd(dmul(h[3], s1), dmul(h[4], s2));
    x2 = dmul(s2, h[5]);
}

// FP32 positions in the scaled bin frame, relative to the atom's bin corner:
// p'_d = (x B)_d * 8 nb_d - 8 b_d (x not wrapped between builds, so p' may
// leave [0,8) by the drift since the build)
__device__ __forceinline__ float4 frame_pos(const double* bs, double x0, double x1, double x2, int bc) {
    double u0 = bs[0] * x0 + (bs[1] * x1 + bs[2] * x2);
    double u1 = bs[3] * x1 + bs[4] * x2;
    double u2 = bs[5] * x2;
    float4 p;
    p.x = (float)(u0 - (double)(8 * (bc & 1023)));
    p.y = (float)(u1 - (double)(8 * ((bc >> 10) & 1023)));
    p.z = (float)(u2 - (double)(8 * ((bc >> 20) & 1023)));
    p.w = 0.f;
    return p;
}

// what the rebuild's first steps read and write (a single cell)
struct BinArgs {
    int n, nbins;
    double *x, *s, *xb;
    Geo g;
    int *binc, *binid, *bin_count, *bin_start, *bin_tmp;
    float4 *p32, *p0, *bin_pos;
    const uint8_t* elem;
    double* partials;
    int drift_rows;
};

// atom i wrapped into the cell (x2s_lcl then s2x_all); returns its bin.  The
// build positions (x0, and p0 in the frame) are the wrapped ones; the mixed
// MD path defers its mean-displacement removal (drift) to here.
__device__ __forceinline__ int wrap_atom(const BinArgs& a, int i, const double (&drift)[3], int& bad) {
    const int n = a.n;
    const Geo& g = a.g;
    double x0 = dsub(a.x[i], drift[0]), x1 = dsub(a.x[n + i], drift[1]), x2 = dsub(a.x[2 * n + i], drift[2]);
    double s0 = dadd(dmul(g.b6[0], x0), dadd(dmul(g.b6[1], x1), dmul(g.b6[2], x2)));
    s0 = wrap01(s0, &bad);
    double s1 = dadd(dmul(g.b6[3], x1), dmul(g.b6[4], x2));
    s1 = wrap01(s1, &bad);
    double s2 = dmul(x2, g.b6[5]);
    s2 = wrap01(s2, &bad);
    s2x(g.h6, s0, s1, s2, x0, x1, x2);
    a.x[i] = a.xb[i] = x0;
    a.x[n + i] = a.xb[n + i] = x1;
    a.x[2 * n + i] = a.xb[2 * n + i] = x2;
    a.s[i] = s0;
    a.s[n + i] = s1;
    a.s[2 * n + i] = s2;
    int b0 = min((int)(s0 * g.nb[0]), g.nb[0] - 1);
    int b1 = min((int)(s1 * g.nb[1]), g.nb[1] - 1);
    int b2 = min((int)(s2 * g.nb[2]), g.nb[2] - 1);
    const int bc = b0 | (b1 << 10) | (b2 << 20);
    a.binc[i] = bc;
    a.p32[i] = a.p0[i] = frame_pos(g.bs, x0, x1, x2, bc);
    const int b = b0 + g.nb[0] * (b1 + g.nb[1] * b2);
    a.binid[i] = b;
    return b;
}

// rebuild step 1: wrap, bin, count
__global__ void k_wrap_bin(const __grid_constant__ BinArgs a, DevScalars* sc) {
    dep_wait();
    if (!sc->rebuild) return;
    int bad = 0;
    double drift[3];
    drift_now(sc, a.partials, a.drift_rows, 1.0 / (double)a.n, drift);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x)
        atomicAdd(&a.bin_count[wrap_atom(a, i, drift, bad)], 1);
    if (bad) sc->bad = 1;
}

// batch variant of step 1: each atom uses its cell's box, bins and drift
// (cells without their rebuild flag keep their wrap, bins and rows)
__global__ void k_wrap_bin_b(int n, double* __restrict__ x, double* __restrict__ s, double* __restrict__ xb,
                             const CellGeo* __restrict__ cells, const int* __restrict__ cell_of,
                             const CellMd* __restrict__ cmd, int* __restrict__ binc, int* __restrict__ binid,
                             int* __restrict__ bin_count, const uint8_t* __restrict__ cell_reb,
                             float4* __restrict__ p32, float4* __restrict__ p0, DevScalars* sc) {
    dep_wait();
    if (!sc->rebuild) return;
    int bad = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int c = cell_of[i];
        if (!cell_reb[c]) continue;
        const CellGeo& g = cells[c];
        const double* dr = cmd[c].drift;
        double x0 = dsub(x[i], dr[0]), x1 = dsub(x[n + i], dr[1]), x2 = dsub(x[2 * n + i], dr[2]);
        double s0 = dadd(dmul(g.b6[0], x0), dadd(dmul(g.b6[1], x1), dmul(g.b6[2], x2)));
        s0 = wrap01(s0, &bad);
        double s1 = dadd(dmul(g.b6[3], x1), dmul(g.b6[4], x2));
        s1 = wrap01(s1, &bad);
        double s2 = dmul(x2, g.b6[5]);
        s2 = wrap01(s2, &bad);
        s2x(g.h6, s0, s1, s2, x0, x1, x2);
        x[i] = xb[i] = x0;
        x[n + i] = xb[n + i] = x1;
        x[2 * n + i] = xb[2 * n + i] = x2;
        s[i] = s0;
        s[n + i] = s1;
        s[2 * n + i] = s2;
        int b0 = min((int)(s0 * g.nb[0]), g.nb[0] - 1);
        int b1 = min((int)(s1 * g.nb[1]), g.nb[1] - 1);
        int b2 = min((int)(s2 * g.nb[2]), g.nb[2] - 1);
        const int bc = b0 | (b1 << 10) | (b2 << 20);
        binc[i] = bc;
        p32[i] = p0[i] = frame_pos(g.bs, x0, x1, x2, bc);
        int b = g.bin_base + b0 + g.nb[0] * (b1 + g.nb[1] * b2);
        binid[i] = b;
        atomicAdd(&bin_count[b], 1);
    }
    if (bad) sc->bad = 1;
}

// what a rebuild resets once step 1 has taken the mean displacement out of x
__device__ __forceinline__ void rebuild_reset(DevScalars* sc) {
    sc->maxrow = 0;
    sc->sumrow = 0;
    sc->drift[0] = sc->drift[1] = sc->drift[2] = 0.0;
    sc->nrebuild++;
}

// rebuild step 2: exclusive scan of bin counts (one block), counts zeroed
__global__ void k_scan_bins(int nbins, int* __restrict__ bin_count, int* __restrict__ bin_start,
                            double* __restrict__ partials, int drift_rows, DevScalars* sc) {
    dep_wait();
    if (!sc->rebuild) return;
    // the running step's displacement sums went into x with the drift
    for (int q = threadIdx.x; q < 3 * drift_rows; q += blockDim.x) partials[(q / 3) * kRedSlots + 8 + q % 3] = 0.0;
    __shared__ int part[1024];
    int t = threadIdx.x, T = blockDim.x;
    int chunk = (nbins + T - 1) / T;
    int lo = min(t * chunk, nbins), hi = min(lo + chunk, nbins);
    int sum = 0;
    for (int b = lo; b < hi; b++) sum += bin_count[b];
    part[t] = sum;
    __syncthreads();
    for (int off = 1; off < T; off <<= 1) {
        int v = t >= off ? part[t - off] : 0;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    int run = part[t] - sum;
    for (int b = lo; b < hi; b++) {
        int c = bin_count[b];
        bin_start[b] = run;
        run += c;
        bin_count[b] = 0;
    }
    if (t == T - 1) bin_start[nbins] = part[T - 1];
    if (t == 0) rebuild_reset(sc);
}

// batch variant of step 2: one warp per flagged cell scans its own bins,
// from the cell's first atom (a cell's bins hold exactly its atoms, so the
// other cells' bin starts stay valid)
__global__ void k_scan_bins_b(int ncell, int n, int nbins, const CellGeo* __restrict__ cells,
                              const uint8_t* __restrict__ cell_reb, int* __restrict__ bin_count,
                              int* __restrict__ bin_start, CellMd* __restrict__ cmd, DevScalars* sc) {
    dep_wait();
    if (!sc->rebuild) return;
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        bin_start[nbins] = n;
        rebuild_reset(sc);
    }
    for (int c = warp; c < ncell; c += nw) {
        if (!cell_reb[c]) continue;
        const CellGeo& g = cells[c];
        const int nb = g.nb[0] * g.nb[1] * g.nb[2], base = g.bin_base;
        int run = g.begin;
        if (lane < 3) cmd[c].drift[lane] = 0.0;
        for (int k0 = 0; k0 < nb; k0 += 32) {
            const int k = k0 + lane;
            const int v = k < nb ? bin_count[base + k] : 0;
            int incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += u;
            }
            if (k < nb) {
                bin_start[base + k] = run + incl - v;
                bin_count[base + k] = 0;
            }
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
}

// rebuild step 3: scatter atom indices into their bins (order fixed next);
// a batch scatters the atoms of flagged cells only
__global__ void k_scatter_bins(int n, const int* __restrict__ binid, const int* __restrict__ bin_start,
                               int* __restrict__ bin_count, int* __restrict__ bin_tmp, const int* __restrict__ cell_of,
                               const uint8_t* __restrict__ cell_reb, DevScalars* sc) {
    dep_wait();
    if (!sc->rebuild) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (cell_reb && !cell_reb[cell_of[i]]) continue;
        int b = binid[i];
        int slot = atomicAdd(&bin_count[b], 1);
        bin_tmp[bin_start[b] + slot] = i;
    }
}

// rebuild step 4: one warp per bin ranks its atoms by index (deterministic
// order) and writes their frame positions with the entry bits of atom and
// element in w, bin by bin: what the builder stages of a candidate in one
// coalesced load; counts zeroed for the next rebuild
__global__ void k_sort_bins(int nbins, const int* __restrict__ bin_start, const int* __restrict__ bin_tmp,
                            const float4* __restrict__ p32, const uint8_t* __restrict__ elem,
                            float4* __restrict__ bin_pos, int* __restrict__ bin_count, const int* __restrict__ cell_of,
                            const uint8_t* __restrict__ cell_reb, DevScalars* sc) {
    dep_wait();
    if (!sc->rebuild) return;
    int lane = threadIdx.x & 31;
    int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int nw = (gridDim.x * blockDim.x) >> 5;
    for (int b = warp; b < nbins; b += nw) {
        int lo = bin_start[b], hi = bin_start[b + 1];
        // a batch bin's slots lie in its cell's atom range, so the cell of a
        // non-empty bin is the cell of atom index lo
        if (cell_reb && lo < hi && !cell_reb[cell_of[lo]]) continue;
        for (int k = lo + lane; k < hi; k += 32) {
            int a = bin_tmp[k];
            int r = 0;
            for (int q = lo; q < hi; q++) r += bin_tmp[q] < a;
            float4 p = p32[a];
            p.w = __int_as_float(make_entry(a, elem[a], 0));
            bin_pos[lo + r] = p;
        }
        if (lane == 0) bin_count[b] = 0;
    }
}

// rebuild steps 1 to 4 of a small system as one cluster of blocks: wrap, bin
// and count (an atom's place among its bin's comes back from the count), each
// block scans all counts for itself, scatter, and a warp per bin ranks its
// atoms.  A step whose gate is closed runs one kernel instead of four (100 MD
// steps of 4,000 atoms mixed 4.72 -> 4.48 ms, FP64 7.55 -> 7.28), a rebuild
// waits at two cluster barriers instead of three launches (500 atoms 25.4 ->
// 21.5 us, 2,916 31.8 -> 26.0, 6,912 31.7 -> 30.6).  Sixteen blocks: the FP64
// wrap of 6,912 atoms on eight SMs made that 38.9 us.  Larger systems need
// more SMs than a cluster has.  (One cooperative launch for systems of any
// size costs 7 us with its gate closed.)
constexpr int kSmallCluster = 16;     // blocks
constexpr int kSmallBlock = 512;      // threads of one
constexpr int kSmallAtoms = 8192;     // one atom a thread
constexpr int kSmallBins = 2048;
static_assert(kSmallAtoms <= kSmallCluster * kSmallBlock, "one atom a thread");

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __launch_bounds__(kSmallBlock) k_bin_small(const __grid_constant__ BinArgs a, DevScalars* sc) {
    dep_wait();
    if (!sc->rebuild) return;  // the same for every block: nothing writes it meanwhile
    __shared__ int s_start[kSmallBins + 1], s_warp[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // consecutive blocks take neighbouring warps' worth of atoms, so that a
    // small system spreads over the cluster's SMs
    const int i = (w * kSmallCluster + blockIdx.x) * 32 + lane;
    int bin = 0, slot = 0;
    {
        int bad = 0;
        double drift[3];
        drift_now(sc, a.partials, a.drift_rows, 1.0 / (double)a.n, drift);
        if (i < a.n) {
            bin = wrap_atom(a, i, drift, bad);
            slot = atomicAdd(&a.bin_count[bin], 1);
        }
        if (bad) sc->bad = 1;
    }
    cluster_sync();
    // exclusive scan of the counts: kPer consecutive bins a thread
    constexpr int kPer = kSmallBins / kSmallBlock;
    int c[kPer], sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        const int b = threadIdx.x * kPer + k;
        c[k] = b < a.nbins ? __ldcg(a.bin_count + b) : 0;
        sum += c[k];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_warp[w] = incl;
    __syncthreads();
    int before = lane < w ? s_warp[lane] : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    int run = before + incl - sum;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        const int b = threadIdx.x * kPer + k;
        s_start[b] = run;
        if (blockIdx.x == 0 && b <= a.nbins) a.bin_start[b] = run;
        run += c[k];
    }
    if (threadIdx.x == kSmallBlock - 1) {
        s_start[kSmallBins] = run;
        if (blockIdx.x == 0) {
            if (a.nbins == kSmallBins) a.bin_start[a.nbins] = run;
            rebuild_reset(sc);
        }
    }
    // the running step's displacement sums went into x with the drift
    if (blockIdx.x == 1)
        for (int q = threadIdx.x; q < 3 * a.drift_rows; q += kSmallBlock)
            a.partials[(q / 3) * kRedSlots + 8 + q % 3] = 0.0;
    __syncthreads();
    if (i < a.n) a.bin_tmp[s_start[bin] + slot] = i;
    cluster_sync();
    for (int b = w * kSmallCluster + blockIdx.x; b < a.nbins; b += kSmallCluster * (kSmallBlock / 32)) {
        const int lo = s_start[b], hi = s_start[b + 1];
        for (int k = lo + lane; k < hi; k += 32) {
            const int at = __ldcg(a.bin_tmp + k);
            int r = 0;
            for (int q = lo; q < hi; q++) r += __ldcg(a.bin_tmp + q) < at;
            float4 p = __ldcg(a.p32 + at);
            p.w = __int_as_float(make_entry(at, a.elem[at], 0));
            a.bin_pos[lo + r] = p;
        }
        if (lane == 0) a.bin_count[b] = 0;
    }
}

// a cluster of that many blocks is beyond the portable eight: asked for, and
// the current device asked whether it can run one (both hold for one device,
// so every system asks for its own)
static bool small_cluster_ok() {
    if (cudaFuncSetAttribute(k_bin_small, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kSmallCluster);
    cfg.blockDim = dim3(kSmallBlock);
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = kSmallCluster;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k_bin_small, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return clusters > 0;
}

// frame positions of atoms that moved without a rebuild
__global__ void k_shadow(int n, const double* __restrict__ x, const int* __restrict__ binc, float4* __restrict__ p32,
                         Geo g) {
    dep_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        p32[i] = frame_pos(g.bs, x[i], x[n + i], x[2 * n + i], binc[i]);
}

__global__ void k_shadow_b(int n, const double* __restrict__ x, const int* __restrict__ binc,
                           const CellGeo* __restrict__ cells, const int* __restrict__ cell_of,
                           float4* __restrict__ p32) {
    dep_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        p32[i] = frame_pos(cells[cell_of[i]].bs, x[i], x[n + i], x[2 * n + i], binc[i]);
}

struct BuildArgs {
    int n, maxnbr, ne;
    const double* x;
    const double* s;
    const float4* bin_pos;
    const float4* p32;
    const int* bin_start;
    int* nbr;
    int* nnbr;
    int *own_ent, *other_ent, *nown, *nother;  // FP64: the row's entries by owner (null: not kept)
    Geo g;
    Frame fr;       // frame to Cartesian
    float lo2[kMaxElem * kMaxElem], hi2[kMaxElem * kMaxElem];
    float hi2max;                    // the largest of hi2
    float in2[kMaxElem * kMaxElem];  // pair cutoff squared: entries below it lead their row
    double cut_sk_sq[kMaxElem * kMaxElem];
    const CellGeo* cells;  // batch: per-cell geometry, indexed by cell_of
    const int* cell_of;
    const uint8_t* cell_reb;  // batch: the cells to rebuild
};

// the reference's predicate for a pair inside the FP32 band: x_j' =
// S2X(s_j + n) in FP64 without fused multiply-adds, RSQ < (cut + skin)^2;
// n: the image that the bin step of entry ent reaches from bin geo[0..2]
// of geo[3..5]
__device__ __noinline__ bool exact_keep(const BuildArgs& a, const double* h6, const int* geo, int i, int ent, int pe) {
    const int n = a.n, j = entry_j(ent);
    const int u0 = geo[0] + entry_step(ent, 0), u1 = geo[1] + entry_step(ent, 1), u2 = geo[2] + entry_step(ent, 2);
    double s0 = a.s[j], s1 = a.s[n + j], s2 = a.s[2 * n + j];
    if (u0 >= geo[3]) s0 = dadd(s0, 1.0);
    if (u0 < 0) s0 = dsub(s0, 1.0);
    if (u1 >= geo[4]) s1 = dadd(s1, 1.0);
    if (u1 < 0) s1 = dsub(s1, 1.0);
    if (u2 >= geo[5]) s2 = dadd(s2, 1.0);
    if (u2 < 0) s2 = dsub(s2, 1.0);
    double xj0, xj1, xj2;
    s2x(h6, s0, s1, s2, xj0, xj1, xj2);
    double e0 = dsub(a.x[i], xj0), e1 = dsub(a.x[n + i], xj1), e2 = dsub(a.x[2 * n + i], xj2);
    double rsq = dadd(dmul(e0, e0), dadd(dmul(e1, e1), dmul(e2, e2)));
    return rsq < a.cut_sk_sq[pe];
}

// the distance of an entry as the frame positions give it, in the operations
// that say which entries lead a row: the staged Cartesian positions differ
// from it by rounding, and a pair on the other side of the cutoff would
// change the order of the row's sums
template <bool ORTHO>
__device__ __noinline__ float frame_r2(const BuildArgs& a, const CellGeo* cg, int i, int ent) {
    const float4 pi = a.p32[i], pj = a.p32[entry_j(ent)];
    const float u = pi.x - (pj.x + kBinW * (float)entry_step(ent, 0));
    const float v = pi.y - (pj.y + kBinW * (float)entry_step(ent, 1));
    const float w = pi.z - (pj.z + kBinW * (float)entry_step(ent, 2));
    const float(*G)[3] = cg ? cg->G : a.fr.G;
    const float(*L)[3] = cg ? cg->Glo : a.fr.Glo;
    float x, y, z;
    if (ORTHO) {
        x = u * G[0][0];
        y = v * G[1][1];
        z = w * G[2][2];
    } else if (cg ? cg->ortho : a.fr.ortho) {
        x = fmaf(u, G[0][0], u * L[0][0]);
        y = fmaf(v, G[1][1], v * L[1][1]);
        z = fmaf(w, G[2][2], w * L[2][2]);
    } else {
        x = fmaf(u, G[0][0], fmaf(v, G[1][0], fmaf(w, G[2][0], u * L[0][0] + v * L[1][0] + w * L[2][0])));
        y = fmaf(v, G[1][1], fmaf(w, G[2][1], v * L[1][1] + w * L[2][1]));
        z = fmaf(w, G[2][2], w * L[2][2]);
    }
    return fmaf(x, x, fmaf(y, y, z * z));
}

constexpr int kBuildWarps = 4;    // warps of a builder block
constexpr int kBuildWide = 8;     // the same for systems of few bins
constexpr int kBuildTile = 768;   // candidates staged at a time (12 KB)
constexpr int kBuildHome = 32;    // atoms of the bin worked on at a time
constexpr int kBuildAtoms = 4;    // atoms of a warp that test a candidate together
constexpr int kBuildHits = 160;   // candidates within reach noted per atom, and so the longest row put together on chip

// list thresholds of a pair: kept below lo2, decided in FP64 up to hi2, leading its row below in2
template <bool UNI>
struct BuildCut {
    float lo2, hi2, in2;  // UNI: the same for every pair
    const float* tab;     // else lo2, hi2, in2 of pair e at tab[e], tab[64 + e], tab[128 + e]
    __device__ __forceinline__ float lo(int e) const { return UNI ? lo2 : tab[e]; }
    __device__ __forceinline__ float hi(int e) const { return UNI ? hi2 : tab[kMaxElem * kMaxElem + e]; }
    __device__ __forceinline__ float in(int e) const { return UNI ? in2 : tab[2 * kMaxElem * kMaxElem + e]; }
};

// the candidates within reach2 (squared) of each of the A atoms q0, q0 + W, ... of home, by
// their place in cand and in its order, into hits[u]; nh[u] of them (those
// beyond kBuildHits are not noted)
template <int A, int W>
__device__ __forceinline__ void build_hits(const float4* cand, int nt, const float4* home, int q0, int ng, float reach2,
                                           uint16_t (*hits)[kBuildHits], int* nh) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    float hx[A], hy[A], hz[A];
    int c[A];
#pragma unroll
    for (int u = 0; u < A; u++) {
        const float4 h = home[min(q0 + u * W, ng - 1)];
        hx[u] = h.x;
        hy[u] = h.y;
        hz[u] = h.z;
        c[u] = 0;
    }
#pragma unroll 2
    for (int k0 = 0; k0 < nt; k0 += 32) {
        const float4 p = cand[k0 + lane];
#pragma unroll
        for (int u = 0; u < A; u++) {
            const float dx = hx[u] - p.x, dy = hy[u] - p.y, dz = hz[u] - p.z;
            const bool in = fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= reach2;
            const unsigned m = __ballot_sync(0xffffffffu, in);
            const int at = c[u] + __popc(m & below);
            if (in && at < kBuildHits) hits[u][at] = (uint16_t)(k0 + lane);
            c[u] += __popc(m);
        }
    }
    if (lane == 0)
#pragma unroll
        for (int u = 0; u < A; u++) nh[u] = c[u];
}

// the staged candidates (nt of them, the rest of the last 32 far away), or
// with hits the nt of them that it names, against atom h: its inner entries
// go to dst[0], dst[1], ..., its shell entries to dst[cap - 1], dst[cap - 2],
// ...; entries that would leave the row or meet are dropped (the caller sees
// it from the counts)
template <bool ORTHO, bool UNI>
__device__ __forceinline__ void build_scan(const BuildArgs& a, const BuildCut<UNI>& cut, const float4* cand, int nt,
                                           const uint16_t* hits, const float4& h, int self, const int* geo,
                                           const double* h6, const CellGeo* cg, int* dst, int cap, int& cin,
                                           int& cout) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const int pe0 = entry_elem(self) * a.ne;
    for (int k0 = 0; k0 < nt; k0 += 32) {
        const float4 p = !hits ? cand[k0 + lane] : k0 + lane < nt ? cand[hits[k0 + lane]] : make_float4(1e18f, 0.f, 0.f, 0.f);
        const int ent = __float_as_int(p.w);
        const float dx = h.x - p.x, dy = h.y - p.y, dz = h.z - p.z;
        const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        const bool other = ent != self;
        const int pe = UNI ? 0 : pe0 + entry_elem(ent);
        const unsigned mh = __ballot_sync(0xffffffffu, other && r2 <= cut.hi(pe));
        if (mh == 0u) continue;
        unsigned m = __ballot_sync(0xffffffffu, other && r2 < cut.lo(pe));
        if (m != mh) {
            // pairs within the FP32 rounding of the list cutoff
            bool keep = (m >> lane) & 1u;
            if (!keep && ((mh >> lane) & 1u))
                keep = exact_keep(a, h6, geo, entry_j(self), ent, pe0 + entry_elem(ent));
            m = __ballot_sync(0xffffffffu, keep);
        }
        const float in2 = cut.in(pe);
        unsigned mi = __ballot_sync(0xffffffffu, r2 < in2 * 0.99999f);
        const unsigned mn = __ballot_sync(0xffffffffu, r2 < in2 * 1.00001f);
        if ((mn ^ mi) & m) {
            // pairs within the rounding of the pair cutoff
            bool lead = (mi >> lane) & 1u;
            if (((mn ^ mi) & m) >> lane & 1u) lead = frame_r2<ORTHO>(a, cg, entry_j(self), ent) < in2;
            mi = __ballot_sync(0xffffffffu, lead);
        }
        mi &= m;
        const unsigned mo = m & ~mi;
        const bool inner = (mi >> lane) & 1u;
        const int at = __popc((inner ? mi : mo) & below);
        const int pos = inner ? cin + at : cap - 1 - cout - at;
        if (((m >> lane) & 1u) && (unsigned)pos < (unsigned)cap) dst[pos] = ent;
        cin += __popc(mi);
        cout += __popc(mo);
    }
}

// rebuild step 5: one block per bin.  The candidates of the bin's 27-bin
// stencil are staged in shared memory as Cartesian positions beside the bin
// (bin_pos: one coalesced load a candidate), and the block's warps take the
// bin's atoms in turn.  A warp first tests the candidates against up to four
// atoms at once, 32 at a time, and notes those within reach (one candidate in
// six); then it goes through what it noted, atom by atom, in the same order,
// with the tests that decide what is kept and where.  A row
// holds first its atom's neighbours inside the pair cutoff at build time, in
// (bin step, bin order) order, bin steps c = (d0+1) + 3(d1+1) + 9(d2+1), then
// those of the skin shell in the reverse of that order: it is put together
// in shared memory, inner entries from the front and shell entries from the
// end, and written out in one piece.  Atoms with more than kBuildHits candidates
// in reach, and those of bins whose candidates need several tiles, go through
// the candidates directly; their rows are put together in place.  With the
// inner entries in front, the lanes of an atom
// (slots lane, lane + TPA, ...) get equal shares of the pairs inside the
// cutoff, and the density pass's lanes reach the shell together.  A batch
// finds the bin's cell through its first atom (the bins of a cell hold only
// that cell's atoms).
//
// Bound by instruction issue (72 % of the slots at 500,000 atoms, 778 warp
// instructions an atom).  The atom's counters are uniform in its warp.  With
// every step of 32 candidates taking the full set of tests the pass had 1,000
// instructions an atom; the noting step has 14 for one atom, and a candidate
// read from shared memory serves four.  Four warps a block; eight where the
// bins are few (the whole rebuild 21.9 instead of 29.6 us at 4,000 atoms, 16.5
// instead of 21.5 at 500, 34 instead of 47 at 8,788; at 500,000 598 instead of
// 545).
// Whole rebuild (all its kernels) as this kernel was first built (one warp
// per bin, candidates in the outer loop), with a block a bin and direct
// tests, and now: 4,000 atoms 129, 35 and 22 us; 32,000 164, 60 and 49;
// 256,000 509, 339 and 286; 500,000 905, 650 and 545.
// ORTHO: every cell orthorhombic (one product per axis to Cartesian).
// UNI: every pair type has the same list cutoff (thresholds in registers).
template <bool BATCH, bool ORTHO, bool UNI, int W>
__global__ void __launch_bounds__(32 * W) k_build_bins(const __grid_constant__ BuildArgs a, int nbins,
                                                                 DevScalars* sc) {
    dep_wait();
    if (!sc->rebuild) return;
    __shared__ float4 cand[kBuildTile], home[kBuildHome];
    __shared__ int s_pre[33], s_lo[32], s_cin[kBuildHome], s_cout[kBuildHome], s_geo[6];
    __shared__ int s_row[W][kBuildHits], s_nh[W][kBuildAtoms];
    __shared__ uint16_t s_hits[W][kBuildAtoms][kBuildHits];
    __shared__ float s_cut[UNI ? 1 : 3 * kMaxElem * kMaxElem];
    if (!UNI)
        for (int t = threadIdx.x; t < a.ne * a.ne; t += 32 * W) {
            s_cut[t] = a.lo2[t];
            s_cut[kMaxElem * kMaxElem + t] = a.hi2[t];
            s_cut[2 * kMaxElem * kMaxElem + t] = a.in2[t];
        }
    const BuildCut<UNI> cut{a.lo2[0], a.hi2[0], a.in2[0], s_cut};
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int maxrow = 0, overflow = 0;
    long long sumrow = 0;
    for (int b = blockIdx.x; b < nbins; b += gridDim.x) {
        const int a0 = a.bin_start[b];
        const int na = a.bin_start[b + 1] - a0;
        if (na == 0) continue;
        const int cell = BATCH ? a.cell_of[a0] : 0;  // a batch bin's slots lie in its cell's atom range
        if (BATCH && !a.cell_reb[cell]) continue;
        const CellGeo* cg = BATCH ? a.cells + cell : nullptr;
        const int* nb = BATCH ? cg->nb : a.g.nb;
        const double* h6 = BATCH ? cg->h6 : a.g.h6;
        const float(*G)[3] = BATCH ? cg->G : a.fr.G;
        const int bin_base = BATCH ? cg->bin_base : 0;
        const int bl = b - bin_base;
        const int b0 = bl % nb[0], b1 = (bl / nb[0]) % nb[1], b2 = bl / (nb[0] * nb[1]);
        auto cart = [&](float4& p) {
            if (ORTHO) {
                p.x *= G[0][0];
                p.y *= G[1][1];
                p.z *= G[2][2];
            } else {
                p.x = fmaf(p.x, G[0][0], fmaf(p.y, G[1][0], p.z * G[2][0]));
                p.y = fmaf(p.y, G[1][1], p.z * G[2][1]);
                p.z *= G[2][2];
            }
        };
        __syncthreads();  // the previous bin's tables are no longer read
        if (w == 0) {
            int lo = 0, ncand = 0;
            if (lane < 27) {
                int u0 = b0 + lane % 3 - 1, u1 = b1 + (lane / 3) % 3 - 1, u2 = b2 + lane / 9 - 1;
                if (u0 < 0) u0 += nb[0];
                if (u0 >= nb[0]) u0 -= nb[0];
                if (u1 < 0) u1 += nb[1];
                if (u1 >= nb[1]) u1 -= nb[1];
                if (u2 < 0) u2 += nb[2];
                if (u2 >= nb[2]) u2 -= nb[2];
                const int v = bin_base + u0 + nb[0] * (u1 + nb[1] * u2);
                lo = a.bin_start[v];
                ncand = a.bin_start[v + 1] - lo;
            }
            int incl = ncand;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            s_pre[lane + 1] = incl;
            if (lane == 0) s_pre[0] = 0;
            s_lo[lane] = lo;
            // bin coordinates and counts, for the images of exact_keep
            if (lane < 3) {
                s_geo[lane] = lane == 0 ? b0 : lane == 1 ? b1 : b2;
                s_geo[3 + lane] = nb[lane];
            }
        }
        __syncthreads();
        const int total = s_pre[32];
        const bool one_tile = total <= kBuildTile;
        for (int g0 = 0; g0 < na; g0 += kBuildHome) {
            const int ng = min(kBuildHome, na - g0);
            if (g0) __syncthreads();  // the previous group's atoms are no longer read
            if (threadIdx.x < ng) {
                float4 p = a.bin_pos[a0 + g0 + threadIdx.x];
                cart(p);
                home[threadIdx.x] = p;
                s_cin[threadIdx.x] = s_cout[threadIdx.x] = 0;
            }
            for (int t0 = 0; t0 < total; t0 += kBuildTile) {
                const int nt = min(kBuildTile, total - t0);
                const bool last = t0 + kBuildTile >= total;
                if (t0) __syncthreads();  // the previous tile is no longer read
                if (!one_tile || g0 == 0)
                    for (int k = threadIdx.x; k < ((nt + 31) & ~31); k += 32 * W) {
                        float4 p = make_float4(1e18f, 0.f, 0.f, 0.f);
                        if (k < nt) {
                            const int t = t0 + k;
                            int c = 0;  // the stencil bin of candidate t: s_pre[c] <= t < s_pre[c + 1]
#pragma unroll
                            for (int o = 16; o > 0; o >>= 1)
                                if (s_pre[c + o] <= t) c += o;
                            p = a.bin_pos[s_lo[c] + (t - s_pre[c])];
                            p.x += kBinW * (float)(c % 3 - 1);
                            p.y += kBinW * (float)((c / 3) % 3 - 1);
                            p.z += kBinW * (float)(c / 9 - 1);
                            cart(p);
                            p.w = __int_as_float(__float_as_int(p.w) | make_entry(0, 0, c));
                        }
                        cand[k] = p;
                    }
                __syncthreads();
                for (int q = w, u = 0; q < ng; q += W, u = (u + 1) % kBuildAtoms) {
                    if (one_tile && u == 0) {
                        const int more = (ng - 1 - q) / W;  // atoms of the warp after this one
                        if (more >= 2)
                            build_hits<4, W>(cand, nt, home, q, ng, a.hi2max, s_hits[w], s_nh[w]);
                        else if (more)
                            build_hits<2, W>(cand, nt, home, q, ng, a.hi2max, s_hits[w], s_nh[w]);
                        else
                            build_hits<1, W>(cand, nt, home, q, ng, a.hi2max, s_hits[w], s_nh[w]);
                        __syncwarp();
                    }
                    const float4 h = home[q];
                    const int self = __float_as_int(h.w) | make_entry(0, 0, 13);  // the atom itself, unshifted
                    const int i = entry_j(self);
                    int* row = a.nbr + (size_t)i * a.maxnbr;
                    int cin = 0, cout = 0, tot = 0;
                    const bool chip = one_tile && s_nh[w][u] <= kBuildHits;  // the row is in s_row
                    if (chip) {
                        build_scan<ORTHO, UNI>(a, cut, cand, s_nh[w][u], s_hits[w][u], h, self, s_geo, h6, cg, s_row[w],
                                               kBuildHits, cin, cout);
                        tot = cin + cout;
                        __syncwarp();
                        // (of a row that does not fit only the inner entries)
                        for (int k = lane; k < min(tot <= a.maxnbr ? tot : cin, a.maxnbr); k += 32)
                            row[k] = s_row[w][k < cin ? k : kBuildHits - tot + k];
                    } else {
                        if (one_tile)
                            cin = cout = 0;
                        else
                            cin = s_cin[q], cout = s_cout[q];
                        build_scan<ORTHO, UNI>(a, cut, cand, nt, nullptr, h, self, s_geo, h6, cg, row, a.maxnbr, cin,
                                               cout);
                        tot = cin + cout;
                        if (!last) {
                            if (lane == 0) {
                                s_cin[q] = cin;
                                s_cout[q] = cout;
                            }
                            continue;
                        }
                        // the shell entries at the row's end move behind the
                        // inner ones, 32 at a time, each batch read before
                        // it is written (to lower slots: the gap is never
                        // negative)
                        __syncwarp();
                        for (int k0 = 0; tot <= a.maxnbr && k0 < cout; k0 += 32) {
                            const int k = k0 + lane;
                            const int v = k < cout ? row[a.maxnbr - cout + k] : 0;
                            __syncwarp();
                            if (k < cout) row[cin + k] = v;
                            __syncwarp();
                        }
                    }
                    // a row that does not fit is built again with a larger
                    // capacity; until then (the passes of an MD step may
                    // still walk it) it counts the slots that were written
                    if (lane == 0) a.nnbr[i] = tot <= a.maxnbr ? tot : min(cin, a.maxnbr);
                    if (!BATCH && a.own_ent) {
                        const int len = tot <= a.maxnbr ? tot : 0;
                        const size_t base = (size_t)i * a.maxnbr;
                        int no = 0, nx = 0;
                        for (int k0 = 0; k0 < len; k0 += 32) {
                            const int k = k0 + lane;
                            const int e = k >= len ? 0 : chip ? s_row[w][k < cin ? k : kBuildHits - tot + k] : row[k];
                            const bool own = k < len && pair_owned(i, e);
                            const unsigned mo = __ballot_sync(0xffffffffu, own);
                            const unsigned mx = __ballot_sync(0xffffffffu, k < len && !own);
                            const unsigned below = (1u << lane) - 1u;
                            if (own)
                                a.own_ent[base + no + __popc(mo & below)] = e;
                            else if (k < len)
                                a.other_ent[base + nx + __popc(mx & below)] = e;
                            no += __popc(mo);
                            nx += __popc(mx);
                        }
                        if (lane == 0) {
                            a.nown[i] = no;
                            a.nother[i] = nx;
                        }
                    }
                    __syncwarp();  // s_row is refilled for the warp's next atom
                    overflow |= tot > a.maxnbr;
                    maxrow = max(maxrow, tot);
                    sumrow += tot;
                }
            }
        }
    }
    if (lane == 0) {
        if (overflow) sc->overflow = 1;
        if (maxrow) atomicMax(&sc->maxrow, maxrow);
        if (sumrow) atomicAdd(&sc->sumrow, (unsigned long long)sumrow);
    }
}

// batch: the rebuilt cells' flags
__global__ void k_rebuild_done_b(DevScalars* sc, uint8_t* cell_reb, int ncell) {
    dep_wait();
    if (!sc->rebuild) return;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncell; c += gridDim.x * blockDim.x) cell_reb[c] = 0;
}

// skin test of DynamicMD::decide (dynamic_md.cpp:90-105): rebuild when any
// |x - x0|^2 > skin^2/4, RSQ order, FP64
__global__ void k_skin(int n, const double* __restrict__ x, const double* __restrict__ x0, double skin_sq,
                       DevScalars* sc) {
    dep_wait();
    int moved = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double d0 = dsub(x0[i], x[i]), d1 = dsub(x0[n + i], x[n + i]), d2 = dsub(x0[2 * n + i], x[2 * n + i]);
        double r = dadd(dmul(d0, d0), dadd(dmul(d1, d1), dmul(d2, d2)));
        moved |= r > skin_sq;
    }
    if (__syncthreads_or(moved) && threadIdx.x == 0) sc->rebuild = 1;
}

// batch: the same test, flagging the cells whose atoms moved
__global__ void k_skin_b(int n, const double* __restrict__ x, const double* __restrict__ x0, double skin_sq,
                         const int* __restrict__ cell_of, uint8_t* __restrict__ cell_reb, DevScalars* sc) {
    dep_wait();
    int moved = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double d0 = dsub(x0[i], x[i]), d1 = dsub(x0[n + i], x[n + i]), d2 = dsub(x0[2 * n + i], x[2 * n + i]);
        double r = dadd(dmul(d0, d0), dadd(dmul(d1, d1), dmul(d2, d2)));
        if (r > skin_sq) {
            cell_reb[cell_of[i]] = 1;
            moved = 1;
        }
    }
    if (__syncthreads_or(moved) && threadIdx.x == 0) sc->rebuild = 1;
}

__global__ void k_set_rebuild(DevScalars* sc, int v) {
    dep_wait();
    sc->rebuild = v;
}

// caller order (AoS) <-> bin-sorted order (SoA)
__global__ void k_gather_aos(int n, const int* __restrict__ id, const double* __restrict__ src,
                             double* __restrict__ dst) {
    dep_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int u = id[i];
        dst[i] = src[3 * (size_t)u];
        dst[n + i] = src[3 * (size_t)u + 1];
        dst[2 * n + i] = src[3 * (size_t)u + 2];
    }
}

__global__ void k_scatter_aos(int n, const int* __restrict__ id, const double* __restrict__ src,
                              double* __restrict__ dst) {
    dep_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int u = id[i];
        dst[3 * (size_t)u] = src[i];
        dst[3 * (size_t)u + 1] = src[n + i];
        dst[3 * (size_t)u + 2] = src[2 * n + i];
    }
}

__global__ void k_f32_to_f64(int n3, const float* __restrict__ a, double* __restrict__ b) {
    dep_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += gridDim.x * blockDim.x) b[i] = (double)a[i];
}

// ------------------------------------------------------------------ launchers
void sync_forces64(mappg_sys* s) {
    if (!s->f_is_f32) return;
    launch_dep(s->stream, k_f32_to_f64, grid_for(s, 3LL * s->n, 256), 256, 0, 3 * s->n, s->f32, s->f);
    MAPPG_CUDA(cudaGetLastError());
    s->f_is_f32 = false;
}

void request_rebuild(mappg_sys* s) {
    launch_dep(s->stream, k_set_rebuild, 1, 1, 0, s->sc, 1);
    MAPPG_CUDA(cudaGetLastError());
    if (s->cell_reb) MAPPG_CUDA(cudaMemsetAsync(s->cell_reb, 1, s->ncell, s->stream));
}

void launch_shadow(mappg_sys* s) {
    const int gb = grid_for(s, s->n, 256);
    if (s->ncell > 1)
        launch_dep(s->stream, k_shadow_b, gb, 256, 0, s->n, s->x, s->binc, s->cells_dev, s->cell_of, s->p32);
    else
        launch_dep(s->stream, k_shadow, gb, 256, 0, s->n, s->x, s->binc, s->p32, make_geo(s));
    MAPPG_CUDA(cudaGetLastError());
}

void launch_rebuild_chain(mappg_sys* s) {
    Geo g = make_geo(s);
    const int B = 256;
    int gb = grid_for(s, s->n, B);
    const bool batch = s->ncell > 1;
    // a batch rebuilds the cells whose flag is set (cell_reb), a single cell
    // all of its atoms
    const uint8_t* reb = batch ? s->cell_reb : nullptr;
    bool small = false;
    if (batch) {
        launch_dep(s->stream, k_wrap_bin_b, gb, B, 0, s->n, s->x, s->s, s->x0, s->cells_dev, s->cell_of, s->cmd,
                   s->binc, s->binid, s->bin_count, s->cell_reb, s->p32, s->p0, s->sc);
        launch_dep(s->stream, k_scan_bins_b, (s->ncell * 32 + B - 1) / B, B, 0, s->ncell, s->n, s->nbins,
                   s->cells_dev, s->cell_reb, s->bin_count, s->bin_start, s->cmd, s->sc);
    } else {
        BinArgs w;
        w.n = s->n;
        w.nbins = s->nbins;
        w.x = s->x;
        w.s = s->s;
        w.xb = s->x0;
        w.g = g;
        w.binc = s->binc;
        w.binid = s->binid;
        w.bin_count = s->bin_count;
        w.bin_start = s->bin_start;
        w.bin_tmp = s->bin_tmp;
        w.p32 = s->p32;
        w.p0 = s->p0;
        w.bin_pos = s->bin_pos;
        w.elem = s->elem;
        w.partials = s->partials;
        w.drift_rows = s->drift_rows;
        small = s->bin_cluster && s->nbins <= kSmallBins;
        if (small)
            launch_dep_cluster(s->stream, k_bin_small, kSmallCluster, kSmallCluster, kSmallBlock, 0, w, s->sc);
        else
            launch_dep(s->stream, k_wrap_bin, gb, B, 0, w, s->sc);
    }
    if (!batch && !small) {
        launch_dep(s->stream, k_scan_bins, 1, 1024, 0, s->nbins, s->bin_count, s->bin_start, s->partials,
                   s->drift_rows, s->sc);
    }
    if (!small) {
        launch_dep(s->stream, k_scatter_bins, gb, B, 0, s->n, s->binid, s->bin_start, s->bin_count, s->bin_tmp,
                   s->cell_of, reb, s->sc);
        launch_dep(s->stream, k_sort_bins, grid_for(s, (long long)s->nbins * 32, B), B, 0, s->nbins, s->bin_start,
                   s->bin_tmp, s->p32, s->elem, s->bin_pos, s->bin_count, s->cell_of, reb, s->sc);
    }
    BuildArgs a;
    a.n = s->n;
    a.maxnbr = s->maxnbr;
    a.ne = s->ne;
    a.x = s->x;
    a.s = s->s;
    a.bin_pos = s->bin_pos;
    a.p32 = s->p32;
    a.bin_start = s->bin_start;
    a.nbr = s->nbr;
    a.nnbr = s->nnbr;
    a.own_ent = s->own_ent;
    a.other_ent = s->other_ent;
    a.nown = s->nown;
    a.nother = s->nother;
    a.g = g;
    for (int p = 0; p < s->ne * s->ne; p++) {
        a.cut_sk_sq[p] = s->cut_sk_sq[p];
        a.lo2[p] = (float)(s->cut_sk_sq[p] - s->band);
        a.hi2[p] = (float)(s->cut_sk_sq[p] + s->band);
        a.in2[p] = (float)s->cut_sq[p];
        a.hi2max = std::max(p ? a.hi2max : 0.f, a.hi2[p]);
    }
    a.fr = s->frame;
    a.cells = s->cells_dev;
    a.cell_of = s->cell_of;
    a.cell_reb = reb;
    bool uni = true;
    for (int p = 1; p < s->ne * s->ne; p++) uni = uni && a.lo2[p] == a.lo2[0] && a.hi2[p] == a.hi2[0];
    auto launch_w = [&](auto BT, auto OT, auto UT, auto WT) {
        constexpr int W = decltype(WT)::value;
        constexpr auto kern = k_build_bins<decltype(BT)::value, decltype(OT)::value, decltype(UT)::value, W>;
        static int per_sm = 0;
        if (!per_sm) {
            MAPPG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * W, 0));
            per_sm = std::max(per_sm, 1);
        }
        launch_dep(s->stream, kern, std::min(s->nbins, per_sm * s->sm_count), 32 * W, 0, a, s->nbins, s->sc);
    };
    // few bins: every block is on the chip at once and a bin's atoms in turn
    // are what the pass waits for, so eight warps share them
    auto launch = [&](auto BT, auto OT, auto UT) {
        if (!decltype(BT)::value && s->nbins <= 3 * s->sm_count)
            launch_w(std::false_type(), OT, UT, std::integral_constant<int, kBuildWide>());
        else
            launch_w(BT, OT, UT, std::integral_constant<int, kBuildWarps>());
    };
    auto by_uni = [&](auto BT, auto OT) {
        if (uni)
            launch(BT, OT, std::true_type());
        else
            launch(BT, OT, std::false_type());
    };
    if (batch) {
        if (s->cells_ortho)
            by_uni(std::true_type(), std::true_type());
        else
            by_uni(std::true_type(), std::false_type());
        launch_dep(s->stream, k_rebuild_done_b, (s->ncell + 255) / 256, 256, 0, s->sc, s->cell_reb, s->ncell);
    } else {
        if (s->frame.ortho)
            by_uni(std::false_type(), std::true_type());
        else
            by_uni(std::false_type(), std::false_type());
        if (s->own_ent) launch_link64(s);
    }
    MAPPG_CUDA(cudaGetLastError());
}

void launch_skin_test(mappg_sys* s) {
    double skin_sq = 0.25 * s->skin * s->skin;
    if (s->cell_reb)
        launch_dep(s->stream, k_skin_b, grid_for(s, s->n, 256), 256, 0, s->n, s->x, s->x0, skin_sq, s->cell_of,
                   s->cell_reb, s->sc);
    else
        launch_dep(s->stream, k_skin, grid_for(s, s->n, 256), 256, 0, s->n, s->x, s->x0, skin_sq, s->sc);
    MAPPG_CUDA(cudaGetLastError());
}

EamArgs eam_args(mappg_sys* s) {
    const mappg_ff* ff = s->ff;
    EamArgs a;
    memset(&a, 0, sizeof(a));
    a.n = s->n;
    a.maxnbr = s->maxnbr;
    a.ne = s->ne;
    a.nr = ff->dev.nr;
    a.nrho = ff->dev.nrho;
    a.nbr = s->nbr;
    a.nnbr = s->nnbr;
    a.elem = s->elem;
    a.x = s->x;
    a.p32 = s->p32;
    a.binc = s->binc;
    a.own_ent = s->own_ent;
    a.nown = s->nown;
    a.other_ent = s->other_ent;
    a.nother = s->nother;
    a.other_slot = s->other_slot;
    a.pair_rec = s->pair_rec;
    a.pair_rho = s->pair_rho;
    a.pair_mask = s->pair_mask;
    a.rho64 = ff->dev.rho64;
    a.rphi64 = ff->dev.rphi64;
    a.F64 = ff->dev.F64;
    a.rho32 = ff->dev.rho32;
    a.ftab = ff->dev.ftab;
    a.fjtab = ff->dev.fjtab;
    a.F32 = ff->dev.F32;
    a.F32lo = ff->dev.F32lo;
    a.rho_ei = ff->dev.rho_ei;
    a.rho_ntab = a.rho_ei ? s->ne * s->ne : s->ne;
    a.rho_w = std::min(a.nr - 1, (int)(kDensSmemBytes / (sizeof(float) * 4 * a.rho_ntab)));
    a.rho_mlo = (a.nr - 1) - a.rho_w;  // knots up to nr - 2, the last one a pair can use
    a.dr_inv = ff->dev.dr_inv;
    a.drho_inv = ff->dev.drho_inv;
    a.rho_max = ff->dev.rho_max;
    a.cut_uniform = 1;
    for (int p = 0; p < s->ne * s->ne; p++) {
        a.cut_sq[p] = s->cut_sq[p];
        if ((float)s->cut_sq[p] != (float)s->cut_sq[0]) a.cut_uniform = 0;
    }
    memcpy(a.shift, s->shift, sizeof(a.shift));
    a.fr = s->frame;
    for (int d = 0; d < 3; d++) a.nb[d] = s->nb[d];
    a.q32 = s->q32;
    a.rho = s->rho;
    a.rho_keep = s->keep_rho64 ? s->rho : nullptr;
    a.rho0 = s->rho;
    a.h32 = s->h32;
    a.alpha = 0.0;
    a.cell_active = s->cell_active;
    a.cutmask = s->cutmask;
    a.fs_tab = s->fs_tab;
    a.fs_rec = s->fs_rec;
    a.fs_stride = s->fs_w;
    a.fs_w = s->fs_w;
    if (s->force_smem > 0 && s->fs_rec > 0) {
        const long long fit = (long long)s->force_smem * 1024 / ((long long)sizeof(float4) * s->fs_rec);
        a.fs_w = (int)std::min<long long>(s->fs_w, fit);
    }
    a.fs_off = s->fs_w - a.fs_w;
    a.fs_mlo = s->fs_mlo + a.fs_off;
    a.grp_atoms = s->grp_atoms;
    for (int g = 0; g <= s->ne; g++) a.grp_begin[g] = s->grp_begin[g];
    a.dF = s->dF;
    a.rho32out = s->rho32;
    a.f = s->f;
    a.f32 = s->f32;
    a.partials = s->partials + kRedSlots * kMaxBlocks;
    a.rows_rho = s->pass_rows.rho;
    a.defer = s->defer_totals;
    a.sc = s->sc;
    a.ncell = s->ncell;
    a.nchunk = s->nchunk;
    a.cells = s->cells_dev;
    a.chunk_begin = s->chunk_begin;
    a.chunk_cell = s->chunk_cell;
    a.chunk_part = s->chunk_part;
    return a;
}

// host check after a build: capacity, bad coordinates
void check_build(mappg_sys* s) {
    DevScalars h;
    MAPPG_CUDA(cudaMemcpyAsync(&h, s->sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, s->stream));
    MAPPG_CUDA(cudaStreamSynchronize(s->stream));
    if (h.bad) throw Error{MAPPG_ERR_NAN, "non-finite or far out-of-cell position"};
    if (h.overflow) throw Error{MAPPG_ERR_NBR, "neighbour list capacity exceeded"};
}

}  // namespace mappg

using namespace mappg;

// ------------------------------------------------------------------ system lifecycle (called from api.cpp)
namespace mappg {

static void dev_alloc(void** p, size_t bytes) { MAPPG_CUDA(cudaMalloc(p, bytes > 0 ? bytes : 16)); }

void sys_free(mappg_sys* s) {
    void* ptrs[] = {s->x, s->v, s->f, s->x0, s->s, s->elem, s->id, s->inv, s->p32, s->q32, s->p0, s->f32, s->v32,
                    s->rho32, s->binc, s->binid, s->bin_count, s->bin_start, s->bin_tmp, s->bin_pos, s->nbr, s->nnbr,
                    s->rho, s->dF, s->partials, s->sc, s->stage, s->thermo_dev, s->cells_dev, s->cell_of,
                    s->chunk_begin, s->chunk_cell, s->cell_chunk, s->chunk_part, s->chunk_disp, s->cmd,
                    s->pair_mem, s->cell_out, s->dof, s->stage2, s->cutmask, s->fs_tab, s->grp_atoms, s->cell_reb};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (s->work) cudaFree(s->work);
    if (s->landing) cudaFreeHost(s->landing);
    if (s->ev_main) cudaEventDestroy(s->ev_main);
    if (s->ev_side) cudaEventDestroy(s->ev_side);
    if (s->side) cudaStreamDestroy(s->side);
    if (s->stream) cudaStreamDestroy(s->stream);
}

static unsigned long long morton3(unsigned a, unsigned b, unsigned c) {
    auto spread = [](unsigned long long v) {
        v &= 0x1fffff;
        v = (v | v << 32) & 0x1f00000000ffffULL;
        v = (v | v << 16) & 0x1f0000ff0000ffULL;
        v = (v | v << 8) & 0x100f00f00f00f00fULL;
        v = (v | v << 4) & 0x10c30c30c30c30c3ULL;
        v = (v | v << 2) & 0x1249249249249249ULL;
        return v;
    };
    return spread(a) | (spread(b) << 1) | (spread(c) << 2);
}

void sys_alloc(mappg_sys* s, const double* x_host) {
    const int n = s->n;
    MAPPG_CUDA(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking));
    s->bin_cluster = s->ncell == 1 && n <= kSmallAtoms && small_cluster_ok();
    // fixed atom order: Morton order of the initial bins, then caller index
    // (a batch: cell by cell, Morton order within each cell)
    std::vector<unsigned long long> key(n);
    for (int c = 0; c < s->ncell; c++) {
        const bool batch = s->ncell > 1;
        const double* b6 = batch ? s->cells[c].b6 : s->box.b6;
        const int* nb = batch ? s->cells[c].nb : s->nb;
        const int u0 = batch ? s->cell_begin[c] : 0, u1 = batch ? s->cell_begin[c + 1] : n;
        for (int u = u0; u < u1; u++) {
            const double* xu = x_host + 3 * (size_t)u;
            double sv[3] = {b6[0] * xu[0] + (b6[1] * xu[1] + b6[2] * xu[2]), b6[3] * xu[1] + b6[4] * xu[2],
                            xu[2] * b6[5]};
            unsigned b[3];
            for (int d = 0; d < 3; d++) {
                double w = sv[d] - floor(sv[d]);
                if (!(w >= 0.0 && w < 1.0)) w = 0.0;
                b[d] = (unsigned)std::min((int)(w * nb[d] * 2), 2 * nb[d] - 1);
            }
            key[u] = ((unsigned long long)c << 40) | morton3(b[0], b[1], b[2]);
        }
    }
    s->host_id.resize(n);
    std::iota(s->host_id.begin(), s->host_id.end(), 0);
    std::stable_sort(s->host_id.begin(), s->host_id.end(), [&](int a, int b) { return key[a] < key[b]; });
    std::vector<int> inv(n);
    for (int i = 0; i < n; i++) inv[s->host_id[i]] = i;

    size_t nd = (size_t)3 * n * sizeof(double);
    dev_alloc((void**)&s->x, nd);
    dev_alloc((void**)&s->v, nd);
    dev_alloc((void**)&s->f, nd);
    dev_alloc((void**)&s->x0, nd);
    dev_alloc((void**)&s->s, nd);
    dev_alloc((void**)&s->stage, nd);
    dev_alloc((void**)&s->elem, n);
    dev_alloc((void**)&s->id, sizeof(int) * n);
    dev_alloc((void**)&s->inv, sizeof(int) * n);
    dev_alloc((void**)&s->p32, sizeof(float4) * n);
    dev_alloc((void**)&s->q32, sizeof(float4) * n);
    dev_alloc((void**)&s->p0, sizeof(float4) * n);
    dev_alloc((void**)&s->f32, sizeof(float) * 3 * (size_t)n);
    dev_alloc((void**)&s->v32, sizeof(float) * 3 * (size_t)n);
    dev_alloc((void**)&s->rho32, sizeof(float) * n);
    if (s->precision == MAPPG_MIXED) dev_alloc((void**)&s->cutmask, sizeof(unsigned) * 32 * (size_t)n);
    dev_alloc((void**)&s->binc, sizeof(int) * n);
    dev_alloc((void**)&s->binid, sizeof(int) * n);
    dev_alloc((void**)&s->bin_tmp, sizeof(int) * (size_t)n);
    dev_alloc((void**)&s->bin_pos, sizeof(float4) * (size_t)n);
    dev_alloc((void**)&s->nnbr, sizeof(int) * n);
    dev_alloc((void**)&s->rho, sizeof(double) * n);
    dev_alloc((void**)&s->dF, sizeof(double) * n);
    dev_alloc((void**)&s->partials, sizeof(double) * kRedSlots * kMaxBlocks * 2);
    dev_alloc((void**)&s->sc, sizeof(DevScalars));
    MAPPG_CUDA(cudaMemsetAsync(s->sc, 0, sizeof(DevScalars), s->stream));
    MAPPG_CUDA(cudaMemsetAsync(s->v, 0, nd, s->stream));
    MAPPG_CUDA(cudaMemsetAsync(s->f, 0, nd, s->stream));
    MAPPG_CUDA(cudaMemcpyAsync(s->id, s->host_id.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s->stream));
    MAPPG_CUDA(cudaMemcpyAsync(s->inv, inv.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s->stream));
    if (s->ncell > 1) {
        const int nc = s->ncell, nk = s->nchunk;
        std::vector<int> cell_of(n);
        for (int c = 0; c < nc; c++)
            for (int i = s->cell_begin[c]; i < s->cell_begin[c + 1]; i++) cell_of[i] = c;
        dev_alloc((void**)&s->cells_dev, sizeof(CellGeo) * nc);
        dev_alloc((void**)&s->cell_of, sizeof(int) * n);
        dev_alloc((void**)&s->cmd, sizeof(CellMd) * nc);
        dev_alloc((void**)&s->cell_out, sizeof(double) * 8 * nc);
        dev_alloc((void**)&s->cell_reb, nc);
        MAPPG_CUDA(cudaMemsetAsync(s->cell_reb, 1, nc, s->stream));
        MAPPG_CUDA(cudaMemsetAsync(s->cmd, 0, sizeof(CellMd) * nc, s->stream));
        MAPPG_CUDA(cudaMemcpyAsync(s->cells_dev, s->cells.data(), sizeof(CellGeo) * nc, cudaMemcpyHostToDevice,
                                   s->stream));
        MAPPG_CUDA(cudaMemcpyAsync(s->cell_of, cell_of.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s->stream));
        upload_chunks(s);
    }
    MAPPG_CUDA(cudaStreamSynchronize(s->stream));
}

void sys_alloc_bins(mappg_sys* s) {
    s->alloc_gen++;
    if (s->bin_count) cudaFree(s->bin_count);
    if (s->bin_start) cudaFree(s->bin_start);
    s->bin_count = nullptr;
    s->bin_start = nullptr;
    dev_alloc((void**)&s->bin_count, sizeof(int) * s->nbins);
    dev_alloc((void**)&s->bin_start, sizeof(int) * (s->nbins + 1));
    MAPPG_CUDA(cudaMemsetAsync(s->bin_count, 0, sizeof(int) * s->nbins, s->stream));
}

// the lists and records of pair64.cu for rows of maxnbr entries, one
// allocation of 76 bytes an entry.  Unless the caller has chosen
// (sys_choose_pairs), a system keeps the full-row passes where it would take
// more than a quarter of the card's memory, or more than half of what is free
// (other work on the card then decides which passes run, so only where it
// would be crowded out), or more slots than 32 bits count
static void alloc_pairs64(mappg_sys* s) {
    if (s->pair_mem) cudaFree(s->pair_mem);
    s->pair_mem = nullptr;
    s->own_ent = nullptr;
    if (s->precision != MAPPG_FP64 || s->ncell > 1 || s->pairs_choice == 0) return;
    const bool asked = s->pairs_choice == 1;
    const size_t n = (size_t)s->n, slots = n * s->maxnbr;
    const size_t bytes[] = {48 * slots, 16 * slots, 4 * slots, 4 * slots, 4 * slots, 256 * n, 4 * n, 4 * n};
    size_t at[9] = {0};
    for (int k = 0; k < 8; k++) at[k + 1] = at[k] + (bytes[k] + 255) / 256 * 256;
    if (slots >= kNoSlot) {
        if (asked) throw Error{MAPPG_ERR_UNSUPP, "the list has more slots than pair records can count"};
        return;
    }
    if (!asked && at[8] > (size_t)1 << 28) {
        size_t free_b = 0, total_b = 0;
        MAPPG_CUDA(cudaMemGetInfo(&free_b, &total_b));
        if (at[8] > total_b / 4 || at[8] > free_b / 2) return;
    }
    if (cudaMalloc((void**)&s->pair_mem, at[8]) != cudaSuccess) {
        cudaGetLastError();
        s->pair_mem = nullptr;
        if (asked) throw Error{MAPPG_ERR_CUDA, "no device memory for the pair records"};
        return;
    }
    char* p = s->pair_mem;
    s->pair_rec = (double2*)(p + at[0]);
    s->pair_rho = (double2*)(p + at[1]);
    s->own_ent = (int*)(p + at[2]);
    s->other_ent = (int*)(p + at[3]);
    s->other_slot = (unsigned*)(p + at[4]);
    s->pair_mask = (unsigned*)(p + at[5]);
    s->nown = (int*)(p + at[6]);
    s->nother = (int*)(p + at[7]);
}

// pair records kept (1) or not (0) from here on; the list is built again by
// the next call that needs one
void sys_choose_pairs(mappg_sys* s, int choice) {
    const int before = s->pairs_choice;
    s->built = s->list_box = false;
    s->pairs_choice = choice;
    try {
        alloc_pairs64(s);
    } catch (...) {
        s->pairs_choice = before;
        alloc_pairs64(s);
        throw;
    }
}

void sys_alloc_nbr(mappg_sys* s, int maxnbr) {
    s->alloc_gen++;
    if (s->nbr) cudaFree(s->nbr);
    s->nbr = nullptr;
    s->maxnbr = maxnbr;
    dev_alloc((void**)&s->nbr, sizeof(int) * (size_t)s->n * maxnbr);
    alloc_pairs64(s);
}

// upload caller-order AoS doubles into a SoA device array
void sys_upload(mappg_sys* s, const double* host, double* dev) {
    MAPPG_CUDA(cudaMemcpyAsync(s->stage, host, sizeof(double) * 3 * (size_t)s->n, cudaMemcpyHostToDevice, s->stream));
    launch_dep(s->stream, k_gather_aos, grid_for(s, s->n, 256), 256, 0, s->n, s->id, s->stage, dev);
    MAPPG_CUDA(cudaGetLastError());
}

// upload on the side stream, after the work queued on s->stream so far;
// s->v_pending marks the target as unfinished until s->stream waits on it
void sys_upload_side(mappg_sys* s, const double* host, double* dev) {
    if (!s->side) {
        MAPPG_CUDA(cudaStreamCreateWithFlags(&s->side, cudaStreamNonBlocking));
        MAPPG_CUDA(cudaEventCreateWithFlags(&s->ev_main, cudaEventDisableTiming));
        MAPPG_CUDA(cudaEventCreateWithFlags(&s->ev_side, cudaEventDisableTiming));
        dev_alloc((void**)&s->stage2, sizeof(double) * 3 * (size_t)s->n);
    }
    MAPPG_CUDA(cudaEventRecord(s->ev_main, s->stream));
    MAPPG_CUDA(cudaStreamWaitEvent(s->side, s->ev_main, 0));
    MAPPG_CUDA(cudaMemcpyAsync(s->stage2, host, sizeof(double) * 3 * (size_t)s->n, cudaMemcpyHostToDevice, s->side));
    launch_dep(s->side, k_gather_aos, grid_for(s, s->n, 256), 256, 0, s->n, s->id, s->stage2, dev);
    MAPPG_CUDA(cudaGetLastError());
    MAPPG_CUDA(cudaEventRecord(s->ev_side, s->side));
    s->v_pending = true;
}

// s->stream waits for the side-stream upload (if one is pending)
void sys_join_side(mappg_sys* s) {
    if (!s->v_pending) return;
    MAPPG_CUDA(cudaStreamWaitEvent(s->stream, s->ev_side, 0));
    s->v_pending = false;
}

// queue a caller-order download without waiting for it (the stage array is
// reused in stream order by the next one)
void sys_download_async(mappg_sys* s, const double* dev, double* host) {
    launch_dep(s->stream, k_scatter_aos, grid_for(s, s->n, 256), 256, 0, s->n, s->id, dev, s->stage);
    MAPPG_CUDA(cudaGetLastError());
    MAPPG_CUDA(cudaMemcpyAsync(host, s->stage, sizeof(double) * 3 * (size_t)s->n, cudaMemcpyDeviceToHost, s->stream));
}

void sys_download(mappg_sys* s, const double* dev, double* host) {
    launch_dep(s->stream, k_scatter_aos, grid_for(s, s->n, 256), 256, 0, s->n, s->id, dev, s->stage);
    MAPPG_CUDA(cudaGetLastError());
    MAPPG_CUDA(cudaMemcpyAsync(host, s->stage, sizeof(double) * 3 * (size_t)s->n, cudaMemcpyDeviceToHost, s->stream));
    MAPPG_CUDA(cudaStreamSynchronize(s->stream));
}

// Between runs the system keeps up to this much: a minimization allocated
// and freed each of its 23 to 27 vectors (140 MB for 253,000 atoms).  With
// that, and one scalar read a pass instead of two, a run of 4,000 atoms went
// from 3.09 to 2.29 ms and one of 253,000 from 13.3 to 11.0.  Larger
// workspaces are given back at the end of their run, where the allocation is
// small next to the passes.
static const size_t kWorkKeep = (size_t)256 << 20;

void Work::reserve(size_t bytes) {
    shared_ = !s_->work_busy;
    if (!shared_) {
        MAPPG_CUDA(cudaMalloc((void**)&base_, bytes));
        return;
    }
    s_->work_busy = true;
    if (bytes > s_->work_bytes) {
        drop();
        MAPPG_CUDA(cudaMalloc((void**)&s_->work, bytes));
        s_->work_bytes = bytes;
    }
    base_ = s_->work;
}

void Work::drop() {
    if (s_->work) cudaFree(s_->work);
    s_->work = nullptr;
    s_->work_bytes = 0;
}

Work::~Work() {
    if (!shared_) {
        if (base_) cudaFree(base_);
        return;
    }
    s_->work_busy = false;
    if (s_->work_bytes > kWorkKeep) drop();
}

void* sys_landing(mappg_sys* s) {
    if (!s->landing) MAPPG_CUDA(cudaMallocHost(&s->landing, 4096));
    return s->landing;
}

// full build with capacity growth: first build sizes the rows from a count
void sys_build(mappg_sys* s) {
    for (int attempt = 0; attempt < 4; attempt++) {
        request_rebuild(s);
        MAPPG_CUDA(cudaMemsetAsync(&s->sc->overflow, 0, sizeof(int), s->stream));
        launch_rebuild_chain(s);
        DevScalars h;
        MAPPG_CUDA(cudaMemcpyAsync(&h, s->sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, s->stream));
        MAPPG_CUDA(cudaStreamSynchronize(s->stream));
        if (h.bad) throw Error{MAPPG_ERR_NAN, "non-finite or far out-of-cell position"};
        if (!h.overflow) {
            launch_dep(s->stream, k_set_rebuild, 1, 1, 0, s->sc, 0);
            s->built = true;
            s->list_box = true;
            return;
        }
        int need = (int)h.maxrow;
        int cap = ((need + need / 4 + 16) + 31) / 32 * 32;
        sys_alloc_nbr(s, cap);
    }
    throw Error{MAPPG_ERR_NBR, "neighbour list capacity could not be sized"};
}

// the cell of atom i (bin-sorted order) of a batch
static int cell_of_host(const mappg_sys* s, int i) {
    return (int)(std::upper_bound(s->cell_begin.begin(), s->cell_begin.end(), i) - s->cell_begin.begin()) - 1;
}

void sys_neighbors(mappg_sys* s, int* counts, int* entries, long long* total) {
    const int n = s->n;
    std::vector<int> nn(n), bc(n);
    MAPPG_CUDA(cudaMemcpyAsync(nn.data(), s->nnbr, sizeof(int) * n, cudaMemcpyDeviceToHost, s->stream));
    MAPPG_CUDA(cudaMemcpyAsync(bc.data(), s->binc, sizeof(int) * n, cudaMemcpyDeviceToHost, s->stream));
    std::vector<int> rows;
    if (entries) {
        rows.resize((size_t)n * s->maxnbr);
        MAPPG_CUDA(cudaMemcpyAsync(rows.data(), s->nbr, sizeof(int) * rows.size(), cudaMemcpyDeviceToHost, s->stream));
    }
    MAPPG_CUDA(cudaStreamSynchronize(s->stream));
    long long tot = 0;
    std::vector<long long> off(n + 1, 0);
    for (int i = 0; i < n; i++) {
        int u = s->host_id[i];
        if (counts) counts[u] = nn[i];
        tot += nn[i];
    }
    if (total) *total = tot;
    if (!entries) return;
    // caller order offsets
    std::vector<long long> uoff(n + 1, 0);
    std::vector<int> ucount(n);
    for (int i = 0; i < n; i++) ucount[s->host_id[i]] = nn[i];
    for (int u = 0; u < n; u++) uoff[u + 1] = uoff[u] + ucount[u];
    for (int i = 0; i < n; i++) {
        int u = s->host_id[i];
        int b[3] = {bc[i] & 1023, (bc[i] >> 10) & 1023, (bc[i] >> 20) & 1023};
        int* out = entries + 4 * uoff[u];
        for (int k = 0; k < nn[i]; k++) {
            int e = rows[(size_t)i * s->maxnbr + k];
            int j = entry_j(e);
            int d[3] = {entry_step(e, 0), entry_step(e, 1), entry_step(e, 2)};
            out[4 * k] = s->host_id[j];
            const int* nbq = s->ncell > 1 ? s->cells[cell_of_host(s, i)].nb : s->nb;
            for (int q = 0; q < 3; q++) {
                int uq = b[q] + d[q];
                out[4 * k + 1 + q] = uq < 0 ? -1 : (uq >= nbq[q] ? 1 : 0);
            }
        }
    }
}

}  // namespace mappg
