// Reduction helpers shared by the kernels: block partials written to a
// per-block slot row, and a fixed-order final sum by the last block to
// finish (deterministic, no floating-point atomics).
//
// What these cost is FP64 issue: GB300 runs ~2 FP64 operations per clock per
// SM, so one warp-wide FP64 add holds the SM's pipe for 16 clocks, and a
// butterfly per value (five adds each) of seven values in the 32 warps of an
// SM held it for ~9 us, as long as the force pass itself on 4,000 atoms.
// So K values are summed together (warp_sums: the lanes halve the values
// among themselves, 9 adds instead of 40 for eight values), sums of
// compensated FP32 pairs stay in FP32 across the warp (Sum32), and
// all threads of the last block, not one warp, add up the blocks' partials.
// Density + force on 256 mixed atoms, where nothing else counts: 49.8 us
// with butterflies, 19.5 so; 4,000 atoms at eight lanes: 53.3 and 21.6.
#pragma once

#include "system.h"

namespace mappg {

// Programmatic dependent launch: a kernel launched by launch_dep is brought
// onto the SMs as the blocks of the kernel before it in the stream leave
// them, and waits in dep_wait, its first statement, until that kernel has
// completed and its writes are visible.  What it hides is launch latency: a
// force call of 500 FP64 atoms 152 -> 138 us, 10 L-BFGS iterations of 4,000
// 3.55 -> 2.99 ms, 100 MD steps of 4,000 mixed atoms 4.87 -> 4.76.  Letting the
// next kernel on earlier (griddepcontrol.launch_dependents) was measured and
// not kept: its blocks crowd the SMs that happen to be free (100 FP64 steps
// 7.5 -> 8.7 ms at the start of a kernel, 8.2 before its reduction).  A kernel
// with dep_wait launched in the ordinary way runs as ever.
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// cluster: blocks of the grid's thread-block clusters
template <class... P, class... A>
static void launch_dep_cluster(cudaStream_t stream, void (*kernel)(P...), int cluster, int grid, int block, size_t smem,
                               A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cluster;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    MAPPG_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}

template <class... P, class... A>
static void launch_dep(cudaStream_t stream, void (*kernel)(P...), int grid, int block, size_t smem, A&&... args) {
    launch_dep_cluster(stream, kernel, 1, grid, block, smem, std::forward<A>(args)...);
}

// 32-byte read-only loads (one sector per lane, one instruction): the spline
// records are 32 bytes and 32-byte aligned, so a lane fetches a whole record
// with one L1 request instead of two
__device__ __forceinline__ Dbl4 ldg4(const Dbl4* p) {
    Dbl4 r;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w) : "l"(p));
    return r;
}

__device__ __forceinline__ void ldg8(const float4* p, float4& a, float4& b) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

// s + e == a + b exactly (Knuth's two-sum)
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

// a sum of FP32 terms held as three floats, value s + e + g: the rounding
// errors of the additions in s go into e, exactly, and those in e into g, so
// only g is rounded, about 2^-72 of the terms' size.  The warp's total then
// carries more than an FP64 sum of the terms would, in FP32 instructions only:
// 21 an addition, a third of the time of one FP64 addition.  (With two floats,
// good to 2^-47, runs of 4,000 to 256,000 atoms were 0.4 to 0.9 % faster;
// converting in the block's first warp alone, not in each warp, made them 1.5
// % slower.)
struct Sum32 {
    float s, e, g;
};

__device__ __forceinline__ double red_add(double a, double b) { return a + b; }
__device__ __forceinline__ float red_add(float a, float b) { return a + b; }
__device__ __forceinline__ Sum32 red_add(Sum32 a, Sum32 b) {
    Sum32 r;
    float t, u, v, w;
    two_sum(a.s, b.s, r.s, t);
    two_sum(a.e, b.e, u, v);
    two_sum(u, t, r.e, w);
    r.g = (a.g + b.g) + (v + w);
    return r;
}
template <class T>
__device__ __forceinline__ T red_xor(T v, int o) {
    return __shfl_xor_sync(0xffffffffu, v, o);
}
__device__ __forceinline__ Sum32 red_xor(Sum32 v, int o) {
    return {__shfl_xor_sync(0xffffffffu, v.s, o), __shfl_xor_sync(0xffffffffu, v.e, o),
            __shfl_xor_sync(0xffffffffu, v.g, o)};
}
__device__ __forceinline__ double red_double(double v) { return v; }
__device__ __forceinline__ double red_double(float v) { return (double)v; }
__device__ __forceinline__ double red_double(Sum32 v) { return (double)v.s + ((double)v.e + (double)v.g); }
template <class T>
__device__ __forceinline__ T red_zero() {
    return T(0);
}
template <>
__device__ __forceinline__ Sum32 red_zero<Sum32>() {
    return {0.f, 0.f, 0.f};
}

struct RedAdd {
    template <class T>
    __device__ __forceinline__ T operator()(T a, T b) const {
        return red_add(a, b);
    }
};
// maximum of the bit patterns of non-negative doubles (they order as the
// values do), in integer instructions; see bits_of_abs
struct RedMaxBits {
    __device__ __forceinline__ unsigned long long operator()(unsigned long long a, unsigned long long b) const {
        return a > b ? a : b;
    }
};
// the bits of |v|, zero for a NaN (fmax leaves a NaN out)
__device__ __forceinline__ unsigned long long bits_of_abs(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    return b > 0x7ff0000000000000ull ? 0ull : b;
}

constexpr int red_pow2(int k) { return k <= 1 ? 1 : 2 * red_pow2((k + 1) / 2); }

// the warp's totals of P values (P a power of two): with log2 P exchanges
// each lane ends up with one of them, value lane / (32 / P), which the other
// lanes of that value hold too
template <class Op, class T, int P>
__device__ __forceinline__ T warp_reduce(T (&v)[P], Op op) {
    const int lane = threadIdx.x & 31;
    int o = 16;
#pragma unroll
    for (int h = P / 2; h > 0; h >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < h; k++) {
            const T give = up ? v[k] : v[k + h], keep = up ? v[k + h] : v[k];
            v[k] = op(keep, red_xor(give, o));
        }
    }
    T t = v[0];
#pragma unroll
    for (; o > 0; o >>= 1) t = op(t, red_xor(t, o));
    return t;
}

// one row of P doubles (room for 8 or 16) per warp, shared by the sums of a
// kernel
constexpr int red_width(int p) { return p <= 8 ? 8 : 16; }
template <int W>
__device__ __forceinline__ double (*red_rows())[W] {
    __shared__ double red[32][W];
    return red;
}

// the sum of the block's rows of P values in red_rows, by the first warp:
// lane k < P returns value k.  A dependent FP64 add takes 65 clocks here, so
// the lanes share the rows and add up pairwise; ORDERED adds the warps' rows
// one by one (the minimizers' dot products: their order is part of a
// relaxation's path, which magnifies a last bit)
template <int P, bool ORDERED>
__device__ __forceinline__ double rows_sum() {
    double(*red)[red_width(P)] = red_rows<red_width(P)>();
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    double t = 0.0;
    if (ORDERED) {
        if (lane < P)
            for (int q = 0; q < nw; q++) t += red[q][lane];
        return t;
    }
    for (int q = lane / P; q < nw; q += 32 / P) t += red[q][lane % P];
#pragma unroll
    for (int o = P; o < 32; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

// block totals of K values of type T, as doubles: value k in lane k of the
// first warp
template <int K, bool ORDERED = false, class T>
__device__ __forceinline__ double block_sums(const T (&v)[K]) {
    constexpr int P = red_pow2(K);
    static_assert(P <= 16, "a row holds 16 values");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T u[P];
#pragma unroll
    for (int k = 0; k < P; k++) u[k] = k < K ? v[k < K ? k : 0] : red_zero<T>();
    const T t = warp_reduce(u, RedAdd());
    if (lane % (32 / P) == 0) red_rows<red_width(P)>()[w][lane / (32 / P)] = red_double(t);
    __syncthreads();
    return w == 0 ? rows_sum<P, ORDERED>() : 0.0;
}

// the first warp, whose lanes stored the block's partials, counts the block
// in; true in every thread of the block that came last, which then sees all
// blocks' partials
__device__ __forceinline__ bool last_block(unsigned* counter) {
    __shared__ bool last;
    if (threadIdx.x < 32) {
        __threadfence();
        __syncwarp();
        if (threadIdx.x == 0) {
            last = atomicAdd(counter, 1u) == gridDim.x - 1;
            if (last) __threadfence();
        }
    }
    __syncthreads();
    return last;
}

// block-wide sums of K values (double, float, or Sum32: three floats within a
// warp, FP64 across warps and blocks; float values are for quantities whose
// warp sums need no more than FP32) into
// partials[blockIdx.x*kRedSlots + slot0 + k]; returns true in the block that
// finished last (its threads then see all partials)
template <int K, bool ORDERED = false, class T>
__device__ bool block_partials(const T (&v)[K], double* partials, int slot0, unsigned* counter) {
    const double t = block_sums<K, ORDERED>(v);
    if (threadIdx.x < K) partials[blockIdx.x * kRedSlots + slot0 + threadIdx.x] = t;
    return last_block(counter);
}

// sums of the first K partial slots over nblk blocks by the whole block, in
// a fixed order, into tot[0..K-1] (shared memory, ready for every thread on
// return); four rows per thread are loaded at a time.  nblk8: the rows of
// slots 8 and up, where another kernel's blocks left them (-1: nblk)
template <int K>
__device__ void final_sums(const double* partials, int nblk, double* tot, int nblk8 = -1) {
    constexpr int P = red_pow2(K);
    if (K > 8 && nblk8 >= 0 && threadIdx.x % P >= 8) nblk = nblk8;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int k = threadIdx.x % P, rows = blockDim.x / P;
    double t = 0.0;
    for (int b0 = threadIdx.x / P; b0 < nblk; b0 += 4 * rows) {
        double u[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int b = b0 + q * rows;
            u[q] = k < K && b < nblk ? __ldcg(partials + b * kRedSlots + k) : 0.0;
        }
        t += (u[0] + u[1]) + (u[2] + u[3]);
    }
#pragma unroll
    for (int o = P; o < 32; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane < P) red_rows<red_width(P)>()[w][lane] = t;
    __syncthreads();
    if (w == 0) {
        const double r = rows_sum<P, false>();
        if (lane < K) tot[lane] = r;
    }
    __syncthreads();
}

// the same in an order that does not depend on the block's size (see
// rows_sum): 32 strided sums of the blocks' rows per slot, then a butterfly
// over them, a warp per slot
template <int K>
__device__ void final_sums_ordered(const double* partials, int nblk, double* tot) {
    constexpr int P = red_pow2(K);
    double(*red)[red_width(P)] = red_rows<red_width(P)>();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int k = threadIdx.x % P;
    for (int r = threadIdx.x / P; r < 32; r += blockDim.x / P) {
        double t = 0.0;
        for (int b0 = r; b0 < nblk; b0 += 8 * 32) {
            double u[8];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int b = b0 + 32 * q;
                u[q] = k < K && b < nblk ? __ldcg(partials + b * kRedSlots + k) : 0.0;
            }
#pragma unroll
            for (int q = 0; q < 8; q++) t += u[q];
        }
        red[r][k] = t;
    }
    __syncthreads();
    for (int c = w; c < K; c += nw) {
        double t = red[lane][c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) tot[c] = t;
    }
    __syncthreads();
}

// mixed MD: the mean displacement not yet removed from x, in every thread of
// the block: what earlier steps left in sc->drift, and the running step's
// per-block sums in slots 8-10 of the first `rows` partial rows (0: none)
__device__ inline void drift_now(const DevScalars* sc, const double* partials, int rows, double n_inv,
                                 double (&d)[3]) {
    __shared__ double tot[3];
    if (rows) final_sums<3>(partials + 8, rows, tot);
    for (int c = 0; c < 3; c++) d[c] = sc->drift[c] + (rows ? tot[c] * n_inv : 0.0);
}

// energy and virial of a force call from its passes' rows, by the whole block:
// out[0] the energy, out[1..6] the virial (shared memory, set by the first
// warp, which may read them after __syncwarp)
__device__ inline void pass_totals(const double* partials, const PassRows& r, double* out) {
    __shared__ double tot[8];
    const int k = threadIdx.x % 8;
    final_sums<8>(partials, k == 0 ? r.pair : k == 7 ? r.rho : r.force, tot);
    if (threadIdx.x < 7) out[threadIdx.x] = r.scale * tot[threadIdx.x] + (threadIdx.x == 0 ? tot[7] : 0.0);
    if (threadIdx.x < 32) __syncwarp();
}

// the last block of a force pass (all threads): energy and virial of the call
__device__ inline void store_totals(const double* partials, const PassRows& r, DevScalars* sc, unsigned* counter) {
    __shared__ double out[7];
    pass_totals(partials, r, out);
    if (threadIdx.x < 7) (threadIdx.x ? sc->virial[threadIdx.x - 1] : sc->energy) = out[threadIdx.x];
    if (threadIdx.x == 0) *counter = 0;
}

// block sums of K values (as block_partials) into out[0..K-1], one batch chunk
template <int K, class T>
__device__ __forceinline__ void chunk_store(const T (&v)[K], double* out) {
    const double t = block_sums<K>(v);
    if (threadIdx.x < K) out[threadIdx.x] = t;
    __syncthreads();
}

}  // namespace mappg
