// Applying the AMG hierarchy: V-cycle and the outer flexible CG.
//
// Replaces the solve half of SEMO's solveAMGCL (src/solvers/solveAMGCL.cpp:
// 974-980, AMGCL's V-cycle lib/amgcl/mpi/amg.hpp:343-380 and its Krylov
// loop).  The hierarchy is built by amg_setup.cu.
//
// Layout and kernels, GB300-first:
//  * the finest level and the FP64 outer operator are stored SELL-32 (slices
//    of 32 rows, column-major inside a slice, padded to the slice's longest
//    row): one thread per row, every load coalesced.  Rows there have ~7
//    entries, so a warp-per-row or sub-warp CSR kernel is latency-bound;
//    coarse levels (27-60 entries a row) stay CSR with 4-32 lanes a row;
//  * degree-2 Chebyshev smoothing is fused: pre-smoothing from a zero guess
//    is one kernel (the first iterate D^-1 b / theta is formed on the fly
//    for the neighbours), post-smoothing is two, with no separate x += d;
//  * the CG update uses q = A z + beta q (so p and q update in place) and
//    the dot products are folded into the kernels that produce their
//    operands; one CG iteration is 22 launches at 48^3 to 128^3 cells (16 at
//    32^3), captured as a CUDA graph; small systems are solved in one kernel
//    (cycle_cluster.cuh).
// FP32 V-cycle arithmetic stays on the FP32 pipes (FP64 is 1/58 of FP32
// on GB300); dot products and the outer residual are FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <vector>

#include "convert.cuh"
#include "index.h"
#include "semo_internal.h"

namespace semo {
namespace {

// Grid of the kernels that end in a reduction (dot products fused into the
// SpMVs and vector updates), grid-stride: a fixed 608-way partition of the
// rows at most (a block per 256 rows below that), one partial sum per block, summed in a fixed order.  608 is 4 blocks
// of 256 per multiprocessor on GB300's 152 (measured faster here than 16 a
// multiprocessor); it is not taken from the device so that the partition,
// and with it every sum's bits, is the same on any GPU.
constexpr int kRedBlocks = 608;
constexpr int kRedThreads = 256;
inline int blocks(int64_t n, int t) { return (int)((n + t - 1) / t); }

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
// sum over a block of kRedThreads (sh: kRedThreads doubles), in thread 0.  The
// values go through shared memory to one warp: a shuffle tree in every warp is
// 40 FP64 warp instructions of 16 clocks a multiprocessor each where this is 12.
__device__ __forceinline__ double block_sum(double v, double* sh) {
    __syncthreads();   // sh may still be read
    sh[threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = sh[threadIdx.x];
#pragma unroll
        for (int k = 1; k < kRedThreads / 32; ++k) v += sh[threadIdx.x + 32 * k];
        v = warp_sum(v);
    }
    return v;
}
// sum of a kernel's nb partial sums, by one warp (every lane gets it); four
// chains of additions and eight loads in flight: the kernels that begin with it
// wait for it
__device__ __forceinline__ double parts_sum(const double* part, int nb) {
    double s[4] = {};
    for (int i = threadIdx.x & 31; i < nb; i += 256) {
        double v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = i + 32 * k < nb ? part[i + 32 * k] : 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) s[k & 3] += v[k];
    }
    return __shfl_sync(0xffffffffu, warp_sum((s[0] + s[1]) + (s[2] + s[3])), 0);
}
// blocks of a reducing kernel over n rows
inline int red_blocks(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>(kRedBlocks, (n + kRedThreads - 1) / kRedThreads)); }

// ------------------------------------------------------------ matrix views
// CSR with VS lanes per row.
template <class V, int VS>
struct CsrView {
    static constexpr int kVS = VS, kEven = 0;
    const int* __restrict__ ptr;
    const int* __restrict__ col;
    const V* __restrict__ val;
    int n;
    template <class F>
    __device__ __forceinline__ V dot(int row, int lane, const F& x) const {
        V s = V(0);
        if (row < n) {
            const int e = ptr[row + 1];
            for (int k = ptr[row] + lane; k < e; k += VS) s += val[k] * x(col[k]);
        }
#pragma unroll
        for (int o = VS / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, VS);
        return s;
    }
};

// SELL-32: slice s holds rows 32s..32s+31; entry j of row 32s+l at
// sptr[s] + 32j + l; padding entries point at column 0 with value 0.
template <class V>
struct SellView {
    static constexpr int kVS = 1, kEven = 0;
    const int* __restrict__ sptr;
    const int* __restrict__ col;
    const V* __restrict__ val;
    int n;
    template <class F>
    __device__ __forceinline__ V dot(int row, int, const F& x) const {
        V s = V(0);
        if (row < n) {
            const int sl = row >> 5, l = row & 31;
            const int b = sptr[sl], w = (sptr[sl + 1] - b) >> 5;
            int k = b + l;
            int j = 0;
            if constexpr (sizeof(V) == 4) {   // transfer operators: eight entries in flight
                for (; j < w; j += 8, k += 256) {
                    int cj[8];
                    V vj[8], xj[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (j + q < w) { cj[q] = col[k + 32 * q]; vj[q] = val[k + 32 * q]; }
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (j + q < w) xj[q] = x(cj[q]);
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (j + q < w) s += vj[q] * xj[q];
                }
            } else {
                for (; j + 1 < w; j += 2, k += 64) {   // two independent loads in flight
                    const int c0 = col[k], c1 = col[k + 32];
                    const V v0 = val[k], v1 = val[k + 32];
                    s += v0 * x(c0);
                    s += v1 * x(c1);
                }
                if (j < w) s += val[k] * x(col[k]);
            }
        }
        return s;
    }
};

// SELL-32 with 16-bit columns.  Each slice of 32 rows picks one of three
// encodings (smode[s]), a choice that is uniform across the warp that walks it:
//  0  a signed offset from the row (every |col - row| <= 32767: an RCM-ordered
//     mesh matrix up to ~200^3 cells has all its slices so);
//  1  an unsigned offset from a base column of its (slice, j) group,
//     gbase[(sptr[s] >> 5) + j]: consecutive rows of an RCM order have their
//     j-th entries next to one another (median spread 31 columns), so this
//     holds at any bandwidth unless a group spans more than 65,535 columns;
//  2  32-bit columns in wcol[wptr[s] ..] (values stay in val).
// An FP32 entry moves 6 bytes instead of 8 in modes 0 and 1.  Padding entries
// point at the row (mode 0) or at the group's base (1, 2) with value 0.
template <class V>
struct Sell16View {
    static constexpr int kVS = 1, kEven = 0;
    const int* __restrict__ sptr;
    const int* __restrict__ smode;
    const int* __restrict__ gbase;
    const int* __restrict__ wptr;
    const unsigned short* __restrict__ dcol;
    const int* __restrict__ wcol;
    const V* __restrict__ val;
    int n;
    template <class F>
    __device__ __forceinline__ V dot(int row, int, const F& x) const {
        V s = V(0);
        if (row < n) {
            const int sl = row >> 5, l = row & 31;
            const int b = sptr[sl], w = (sptr[sl + 1] - b) >> 5;
            const int mode = smode[sl];
            int k = b + l;
            int j = 0;
            if (sizeof(V) == 4 && mode == 0 && w <= 8) {
                // short FP32 rows (the finest mesh level): every entry load,
                // then every gather, then the products in entry order -- two
                // memory round trips a slice instead of one per pair of
                // entries (measured 11 % faster at 2.1M rows; the FP64 copy
                // of this path loses more to its register count than it gains)
                int cj[8];
                V vj[8], xj[8];
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (q < w) { cj[q] = row + (short)dcol[k + 32 * q]; vj[q] = val[k + 32 * q]; }
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (q < w) xj[q] = x(cj[q]);
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (q < w) s += vj[q] * xj[q];
            } else if (mode == 0) {
                if (sizeof(V) == 4)   // longer FP32 rows (coarse levels): eight entries in flight
                    for (; j + 7 < w; j += 8, k += 256) {
                        int cj[8];
                        V vj[8], xj[8];
#pragma unroll
                        for (int q = 0; q < 8; ++q) { cj[q] = row + (short)dcol[k + 32 * q]; vj[q] = val[k + 32 * q]; }
#pragma unroll
                        for (int q = 0; q < 8; ++q) xj[q] = x(cj[q]);
#pragma unroll
                        for (int q = 0; q < 8; ++q) s += vj[q] * xj[q];
                    }
                for (; j + 1 < w; j += 2, k += 64) {   // two independent loads in flight
                    const int c0 = row + (short)dcol[k], c1 = row + (short)dcol[k + 32];
                    const V v0 = val[k], v1 = val[k + 32];
                    s += v0 * x(c0);
                    s += v1 * x(c1);
                }
                if (j < w) s += val[k] * x(row + (short)dcol[k]);
            } else if (mode == 1) {
                const int* __restrict__ gb = gbase + (b >> 5);
                for (; j + 1 < w; j += 2, k += 64) {
                    const int c0 = __ldg(gb + j) + dcol[k], c1 = __ldg(gb + j + 1) + dcol[k + 32];
                    const V v0 = val[k], v1 = val[k + 32];
                    s += v0 * x(c0);
                    s += v1 * x(c1);
                }
                if (j < w) s += val[k] * x(__ldg(gb + j) + dcol[k]);
            } else {
                const int* __restrict__ wc = wcol + wptr[sl] + l;
                for (; j + 1 < w; j += 2, k += 64) {
                    const int c0 = wc[32 * j], c1 = wc[32 * j + 32];
                    const V v0 = val[k], v1 = val[k + 32];
                    s += v0 * x(c0);
                    s += v1 * x(c1);
                }
                if (j < w) s += val[k] * x(wc[32 * j]);
            }
        }
        return s;
    }
};

// SELL-32 with 16-bit columns whose slices are all W entries wide and all of mode
// 0 (the finest level of a mesh of one cell type: 7 for hexahedra, 5 for
// tetrahedra).  A slice's place follows from its number, so the entries are
// fetched at once, without the trip for the slice pointer and encoding, and the
// width is known to the compiler: y = b - A x in FP32 at 128^3 cells 30.8 -> 22.6
// us (111 MB: 4.9 TB/s), at 96^3 10.3 -> 6.4 (the width as a run-time value: 26.7
// and 10.3).
template <class V, int W>
struct Sell16UView {
    static constexpr int kVS = 1, kEven = W;
    const unsigned short* __restrict__ dcol;
    const V* __restrict__ val;
    int n;
    // a row in registers: its entries, then the gathered values
    template <class F>
    struct Row {
        int cj[W];
        V vj[W];
        typename F::Raw xj[W];
    };
    template <class F>
    __device__ __forceinline__ void entries(int row, Row<F>& t) const {
        const int k = (row >> 5) * (32 * W) + (row & 31);
#pragma unroll
        for (int q = 0; q < W; ++q) { t.cj[q] = row + (short)dcol[k + 32 * q]; t.vj[q] = val[k + 32 * q]; }
    }
    template <class F>
    __device__ __forceinline__ void gather(Row<F>& t, const F& x) const {
#pragma unroll
        for (int q = 0; q < W; ++q) t.xj[q] = x.load(t.cj[q]);
    }
    template <class F>
    __device__ __forceinline__ V sum(const Row<F>& t, const F& x) const {
        V s = V(0);
#pragma unroll
        for (int q = 0; q < W; ++q) s += t.vj[q] * x.value(t.xj[q]);
        return s;
    }
    template <class F>
    __device__ __forceinline__ V dot(int row, int, const F& x) const {
        if (row >= n) return V(0);
        Row<F> t;
        entries(row, t);
        gather(t, x);
        return sum(t, x);
    }
};

template <class V, class X>
struct Vec {
    using Raw = X;
    const X* __restrict__ p;
    __device__ __forceinline__ X load(int j) const { return __ldg(p + j); }
    __device__ __forceinline__ V value(X x) const { return widen<V>(x); }
    __device__ __forceinline__ V operator()(int j) const { return value(load(j)); }
};
// The first Chebyshev iterate from zero, d0 = D^-1 b / theta, of a vector b that
// the V-cycle starts a level with.  Below the finest level the kernel that
// writes b writes d0 beside it (into the level's t, free until k_post0): formed
// in k_pre2 it is two gathers and two products an entry instead of one gather
// (second level at 128^3, 188k rows of 33 entries: 19.4 us formed there, 15.9
// now).  On the finest level k_xr would have to write it, 25 MB more at 128^3
// for +6 us there against -1 us in k_pre2, so k_pre2 forms it.
template <class V>
struct FirstIterate {
    const V* dinv;   // null: not wanted
    V inv_theta;
    V* d0;
    __device__ __forceinline__ void put(int i, V bi) const {
        if (dinv) d0[i] = dinv[i] * bi * inv_theta;
    }
};
template <class V>
struct FirstGather {   // d0 formed on the fly
    using Raw = V;
    const V* __restrict__ dinv;
    const V* __restrict__ b;
    V inv_theta;
    __device__ __forceinline__ V load(int j) const { return __ldg(dinv + j) * __ldg(b + j) * inv_theta; }
    __device__ __forceinline__ V value(V x) const { return x; }
    __device__ __forceinline__ V operator()(int j) const { return load(j); }
};

// ------------------------------------------- programmatic dependent launch
// The 16 to 22 kernels of a CG iteration each depend on the one before and are
// short, so the gap between one kernel's last block and the next one's first
// is a real share of an iteration.  They are launched with programmatic
// stream serialisation: a kernel's launch is processed while its predecessor
// drains (the predecessor's blocks signal it implicitly as they exit), and
// the kernel waits at pdl_enter() -- its first statement: nothing is read
// before it -- until the predecessor has finished and its writes are
// visible.  Measured at 128^3: 0.42 -> 0.40 ms a CG iteration.  Signalling
// early instead (griddepcontrol.launch_dependents after the wait) put the
// waiting successor's blocks on the multiprocessors beside the running
// kernel and made the iteration 8 % slower than plain launches.  Without a
// programmatic predecessor the wait returns at once, so the kernels stay
// correct under plain launches.
__device__ __forceinline__ void pdl_enter() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <class... P, class... A>
void launch_pdl(void (*k)(P...), int grid, int block, cudaStream_t s, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    SEMO_CUDA(cudaLaunchKernelEx(&cfg, k, std::forward<A>(args)...));
    SEMO_CHECK_LAUNCH();
}

// ------------------------------------------------------- V-cycle kernels
// pre-smoothing, degree 2 from x = 0:  x = d0 + c1 d0 + c2 D^-1 (b - A d0),  d0 = D^-1 b / theta
template <class M, class V, class X>
__global__ void __launch_bounds__(256) k_pre2(M A, const V* __restrict__ dinv, const V* __restrict__ b,
                                              X d0, V c1, V c2, V* __restrict__ x) {
    pdl_enter();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = g / M::kVS, lane = g % M::kVS;
    const bool mine = row < A.n && lane == 0;   // the row's own values are loaded before the product's wait
    const V d = mine ? d0(row) : V(0), di = mine ? dinv[row] : V(0), bi = mine ? b[row] : V(0);
    const V s = A.dot(row, lane, d0);
    if (mine) x[row] = d + c1 * d + c2 * (di * (bi - s));
}
// r = b - A x
template <class M, class V>
__global__ void __launch_bounds__(256) k_res(M A, const V* __restrict__ x, const V* __restrict__ b,
                                             V* __restrict__ r) {
    pdl_enter();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = g / M::kVS, lane = g % M::kVS;
    const bool mine = row < A.n && lane == 0;
    const V bi = mine ? b[row] : V(0);
    const V s = A.dot(row, lane, Vec<V, V>{x});
    if (mine) r[row] = bi - s;
}
// y = A x (restriction with R, and then the coarse level's d0; or any plain product)
template <class M, class V>
__global__ void __launch_bounds__(256) k_mv(M A, const V* __restrict__ x, V* __restrict__ y, FirstIterate<V> f) {
    pdl_enter();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = g / M::kVS, lane = g % M::kVS;
    const V s = A.dot(row, lane, Vec<V, V>{x});
    if (row < A.n && lane == 0) {
        y[row] = s;
        f.put(row, s);
    }
}
// x += P xc
template <class M, class V>
__global__ void __launch_bounds__(256) k_prolong_add(M P, const V* __restrict__ xc, V* __restrict__ x) {
    pdl_enter();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = g / M::kVS, lane = g % M::kVS;
    const bool mine = row < P.n && lane == 0;
    const V xi = mine ? x[row] : V(0);
    const V s = P.dot(row, lane, Vec<V, V>{xc});
    if (mine) x[row] = xi + s;
}
// post-smoothing step 0 from x:  d = D^-1 (b - A x) / theta ;  y = x + d
template <class M, class V>
__global__ void __launch_bounds__(256) k_post0(M A, const V* __restrict__ dinv, const V* __restrict__ b,
                                               V inv_theta, const V* __restrict__ x, V* __restrict__ d,
                                               V* __restrict__ y) {
    pdl_enter();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = g / M::kVS, lane = g % M::kVS;
    const bool mine = row < A.n && lane == 0;
    const V di = mine ? dinv[row] : V(0), bi = mine ? b[row] : V(0), xi = mine ? x[row] : V(0);
    const V s = A.dot(row, lane, Vec<V, V>{x});
    if (mine) {
        const V dv = di * (bi - s) * inv_theta;
        d[row] = dv;
        y[row] = xi + dv;
    }
}
// post-smoothing step 1:  x = y + c1 d + c2 D^-1 (b - A y)
template <class M, class V>
__global__ void __launch_bounds__(256) k_post1(M A, const V* __restrict__ dinv, const V* __restrict__ b, V c1, V c2,
                                               const V* __restrict__ y, const V* __restrict__ d,
                                               V* __restrict__ x) {
    pdl_enter();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = g / M::kVS, lane = g % M::kVS;
    const bool mine = row < A.n && lane == 0;
    const V yi = mine ? y[row] : V(0), dv = mine ? d[row] : V(0), di = mine ? dinv[row] : V(0);
    const V bi = mine ? b[row] : V(0);
    const V s = A.dot(row, lane, Vec<V, V>{y});
    if (mine) x[row] = yi + c1 * dv + c2 * (di * (bi - s));
}
// finest-level post-smoothing step 1 (SELL), also folding in the CG dots
// z.r and z.q (q = A p of the previous iteration); grid-stride, fixed grid
template <class M, class V>
__global__ void __launch_bounds__(kRedThreads, 4) k_post1_dots(M A, const V* __restrict__ dinv,
                                                            const V* __restrict__ b, V c1, V c2,
                                                            const V* __restrict__ y, const V* __restrict__ d,
                                                            V* __restrict__ z, const double* __restrict__ r,
                                                            const double* __restrict__ q,
                                                            double* __restrict__ part) {
    pdl_enter();
    __shared__ double sh[kRedThreads];
    double zr = 0.0, zq = 0.0;
    if constexpr (M::kEven != 0 && sizeof(V) == 4) {
        // two rows a thread in flight: with one the fixed grid's half-filled
        // multiprocessors wait for memory (35.9 -> 32.9 us at 128^3; FP64 rows
        // would not fit the registers)
        const int stride = gridDim.x * blockDim.x;
        const Vec<V, V> yv{y};
        for (int row0 = blockIdx.x * blockDim.x + threadIdx.x; row0 < A.n; row0 += 2 * stride) {
            const int rows[2] = {row0, row0 + stride < A.n ? row0 + stride : row0};
            typename M::template Row<Vec<V, V>> t[2];
            V yi[2], dv[2], di[2], bi[2];
            double ri[2], qi[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) A.entries(rows[k], t[k]);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                A.gather(t[k], yv);
                yi[k] = y[rows[k]]; dv[k] = d[rows[k]]; di[k] = dinv[rows[k]]; bi[k] = b[rows[k]];
                ri[k] = r[rows[k]]; qi[k] = q[rows[k]];
            }
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                if (k == 1 && rows[1] == row0) break;
                const V zi = yi[k] + c1 * dv[k] + c2 * (di[k] * (bi[k] - A.sum(t[k], yv)));
                z[rows[k]] = zi;
                const double zd = widen<double>(zi);
                zr += zd * ri[k];
                zq += zd * qi[k];
            }
        }
    } else {
        const int per_block = blockDim.x / M::kVS, lane = threadIdx.x % M::kVS;
        for (int row0 = blockIdx.x * per_block; row0 < A.n; row0 += gridDim.x * per_block) {
            const int row = row0 + threadIdx.x / M::kVS;   // every lane runs the dot's shuffles
            const bool mine = row < A.n && lane == 0;
            const V yi = mine ? y[row] : V(0), dv = mine ? d[row] : V(0), di = mine ? dinv[row] : V(0);
            const V bi = mine ? b[row] : V(0);
            const double ri = mine ? r[row] : 0.0, qi = mine ? q[row] : 0.0;
            const V s = A.dot(row, lane, Vec<V, V>{y});
            if (mine) {
                const V zi = yi + c1 * dv + c2 * (di * (bi - s));
                z[row] = zi;
                const double zd = widen<double>(zi);
                zr += zd * ri;
                zq += zd * qi;
            }
        }
    }
    zr = block_sum(zr, sh);
    zq = block_sum(zq, sh);
    if (threadIdx.x == 0) { part[blockIdx.x] = zr; part[kRedBlocks + blockIdx.x] = zq; }
}

// generic Chebyshev pieces for degrees other than 2 (CSR)
template <class M, class V>
__global__ void __launch_bounds__(256) k_cheb_d(M A, const V* __restrict__ dinv, const V* __restrict__ b,
                                                const V* __restrict__ x, V c1, V c2, V* __restrict__ d) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = g / M::kVS, lane = g % M::kVS;
    const V s = A.dot(row, lane, Vec<V, V>{x});
    if (row < A.n && lane == 0) d[row] = c1 * d[row] + c2 * (dinv[row] * (b[row] - s));
}
template <class V>
__global__ void k_axpy1(int n, const V* __restrict__ d, V* __restrict__ x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] += d[i];
}
template <class V>
__global__ void k_zero(int n, V* __restrict__ x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = V(0);
}
template <class V>
__global__ void k_copy_t(int n, const V* __restrict__ a, V* __restrict__ b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = a[i];
}

// coarsest level: x = A^-1 b with the explicit FP64 inverse, one block, 4 lanes a
// row with eight entries each in flight (a thread a row: 15 us for 61 rows)
template <class V>
__global__ void __launch_bounds__(256) k_coarse_solve(int n, const double* __restrict__ inv, const V* __restrict__ b,
                                                      V* __restrict__ x) {
    pdl_enter();
    const int sub = threadIdx.x & 3, rows = blockDim.x >> 2;
    for (int i0 = 0; i0 < n; i0 += rows) {
        const int i = i0 + (threadIdx.x >> 2);
        double s = 0.0;
        if (i < n) {
            const double* const m = inv + (size_t)i * n;
            for (int k0 = sub; k0 < n; k0 += 32) {
                double v[8];
                V w[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int k = min(k0 + 4 * u, n - 1);
                    v[u] = m[k];
                    w[u] = b[k];
                }
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (k0 + 4 * u < n) s += v[u] * widen<double>(w[u]);
            }
        }
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if (i < n && sub == 0) x[i] = (V)s;
    }
}

// ---------------------------------------------------------- CG kernels
// device scalars: 0 rz, 2 pq, 4 alpha of the last iteration, 7 its rz, 10
// iterations begun, 11 b.b, 12 r0.r0, 13 iterations done, 14 status, 16 the
// true residual's r.r
// sum of nb partial sums by a block of kRedThreads, in thread 0
__device__ __forceinline__ double sum_parts(const double* part, int nb, double* sh) {
    double s = 0.0;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) s += part[i];
    return block_sum(s, sh);
}
template <class M, class F, int kEven = M::kEven>
struct OuterRow { using type = typename M::template Row<F>; };
template <class M, class F>
struct OuterRow<M, F, 0> { struct type {}; };
// The scalars of an iteration are formed by the kernels that use them, each
// block adding the producer's partial sums itself (one warp): a kernel of their
// own for beta, alpha and r.r cost ~2.75 us each.  Block 0 keeps what later
// kernels need; no block reads a scalar that this kernel writes.
// beta from z.r and z.q (part);  w = A z;  q = w + beta q;  p = z + beta p;
// ppq = p.q   (FP64 SELL operator)
template <class M, class Z>
__global__ void __launch_bounds__(kRedThreads, 4) k_outer_mv(M A, const Z* __restrict__ z,
                                                          double* __restrict__ p, double* __restrict__ q,
                                                          double* __restrict__ scal,
                                                          const double* __restrict__ part, int nb,
                                                          double* __restrict__ ppq) {
    pdl_enter();
    __shared__ double sh[kRedThreads], sbeta;
    const int stride = gridDim.x * blockDim.x;
    int row = blockIdx.x * blockDim.x + threadIdx.x;
    const Vec<double, Z> zv{z};
    // a row's values, on equal slices with its entries; the first row's are under
    // way while beta is formed
    double q0 = 0.0, p0 = 0.0;
    Z zi = Z(0);
    auto fetch = [&](auto& t) {
        if (row >= A.n) return;
        q0 = q[row];
        p0 = p[row];
        zi = z[row];
        if constexpr (M::kEven != 0) {
            A.entries(row, t);
            A.gather(t, zv);
        }
    };
    typename OuterRow<M, Vec<double, Z>>::type t;
    fetch(t);
    if (threadIdx.x < 32) {
        const double rz = parts_sum(part, nb);
        // Polak-Ribiere: beta = z.(r_k - r_{k-1}) / (z_{k-1}.r_{k-1}) = -alpha_{k-1} z.q_{k-1} / rz_prev
        const double bt = scal[10] == 0.0 ? 0.0 : -scal[4] * parts_sum(part + kRedBlocks, nb) / scal[7];
        if (threadIdx.x == 0) {
            sbeta = bt;
            if (blockIdx.x == 0) scal[0] = rz;
        }
    }
    __syncthreads();
    const double beta = sbeta;
    double pq = 0.0;
    while (row < A.n) {
        double w;
        if constexpr (M::kEven != 0) w = A.sum(t, zv);
        else w = A.dot(row, 0, zv);
        const double qi = w + beta * q0;
        const double pi = widen<double>(zi) + beta * p0;
        q[row] = qi;
        p[row] = pi;
        pq += pi * qi;
        row += stride;
        fetch(t);
    }
    pq = block_sum(pq, sh);
    if (threadIdx.x == 0) ppq[blockIdx.x] = pq;
}
// alpha from p.q (ppq);  x += alpha p;  r -= alpha q;  rv = r in the V-cycle's
// type;  part = r.r
template <class V>
__global__ void __launch_bounds__(kRedThreads) k_xr(int n, double* __restrict__ x, double* __restrict__ r,
                                                    V* __restrict__ rv, const double* __restrict__ p,
                                                    const double* __restrict__ q, double* __restrict__ scal,
                                                    const double* __restrict__ ppq, int nb,
                                                    double* __restrict__ part) {
    pdl_enter();
    __shared__ double sh[kRedThreads], salpha;
    // two rows a thread in flight, the first two while alpha is formed (24.7 ->
    // 18.8 us at 128^3, 109 MB: 5.8 TB/s)
    const int stride = gridDim.x * blockDim.x;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double xv[2], pv[2], rr[2], qv[2];
    auto fetch = [&] {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int j = i + k * stride;
            if (j < n) { xv[k] = x[j]; pv[k] = p[j]; rr[k] = r[j]; qv[k] = q[j]; }
        }
    };
    fetch();
    if (threadIdx.x < 32) {
        const double pq = parts_sum(ppq, nb), rz = scal[0];
        if (threadIdx.x == 0) {
            salpha = rz / pq;
            if (blockIdx.x == 0) {
                scal[2] = pq;
                scal[4] = rz / pq;
                scal[7] = rz;
                scal[10] += 1.0;
            }
        }
    }
    __syncthreads();
    const double alpha = salpha;
    double s = 0.0;
    while (i < n) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int j = i + k * stride;
            if (j >= n) break;
            x[j] = xv[k] + alpha * pv[k];
            const double ri = rr[k] - alpha * qv[k];
            r[j] = ri;
            rv[j] = narrow<V>(ri);
            s += ri * ri;
        }
        i += 2 * stride;
        fetch();
    }
    s = block_sum(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}
// out[0] = sum of nb partial sums
__global__ void k_fin_sum(const double* __restrict__ part, int nb, double* __restrict__ out) {
    __shared__ double sh[kRedThreads];
    const double s = sum_parts(part, nb, sh);
    if (threadIdx.x == 0) out[0] = s;
}
// generic dots for the non-fused path: part = a.b, part+R = a.c
template <class A>
__global__ void __launch_bounds__(kRedThreads) k_dot2(int n, const A* __restrict__ a, const double* __restrict__ b,
                                                      const double* __restrict__ c, double* __restrict__ part) {
    __shared__ double sh[kRedThreads];
    double s = 0.0, t = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double ai = (double)(a[i]);
        s += ai * b[i];
        t += ai * c[i];
    }
    s = block_sum(s, sh);
    t = block_sum(t, sh);
    if (threadIdx.x == 0) { part[blockIdx.x] = s; part[kRedBlocks + blockIdx.x] = t; }
}
__global__ void __launch_bounds__(kRedThreads) k_dot(int n, const double* __restrict__ a, const double* __restrict__ b,
                                                     double* __restrict__ part) {
    __shared__ double sh[kRedThreads];
    double s = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) s += a[i] * b[i];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}
template <class A, class B>
__global__ void k_conv(int n, const A* __restrict__ a, B* __restrict__ b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = (B)a[i];
}
// r = b - A x in FP64 (CSR, 8 lanes a row)
__global__ void __launch_bounds__(256) k_res64(CsrView<double, 8> A, const double* __restrict__ x,
                                               const double* __restrict__ b, double* __restrict__ r) {
    const int row = (int)min(row_of(blockIdx.x, blockDim.x, threadIdx.x, 8), (int64_t)A.n), lane = threadIdx.x % 8;
    const double s = A.dot(row, lane, Vec<double, double>{x});
    if (row < A.n && lane == 0) r[row] = b[row] - s;
}

// the same on equally wide slices, a thread a row: the products and the order
// of their sum are those of the 8 lanes above, whose sums take 8 x 4 FP64
// instructions a row where this takes 2 W: 164 -> 60 us at 128^3 (W = 7, bound
// by the FP64 unit)
template <int W>
__global__ void __launch_bounds__(256) k_res64_even(Sell16UView<double, W> A, const double* __restrict__ x,
                                                    const double* __restrict__ b, double* __restrict__ r) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= A.n) return;
    const int k = (row >> 5) * (32 * W) + (row & 31);
    double t[8] = {};
    const double bi = b[row];
#pragma unroll
    for (int q = 0; q < W; ++q) t[q] = __dmul_rn(A.val[k + 32 * q], __ldg(x + row + (short)A.dcol[k + 32 * q]));
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < o; ++q)
            if (q + o < W) t[q] = __dadd_rn(t[q], t[q + o]);
    r[row] = bi - t[0];
}

// --------------------------------------------------------------- SELL build
__global__ void k_sell_width(int n, const int* __restrict__ ptr, int* __restrict__ slice_len) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    const int len = (row < n) ? ptr[row + 1] - ptr[row] : 0;
    const int w = __reduce_max_sync(0xffffffffu, len);
    if ((threadIdx.x & 31) == 0 && row < ((n + 31) & ~31)) slice_len[row >> 5] = 32 * w;
}
template <class V, class W>
__global__ void k_sell_fill(int n, const int* __restrict__ ptr, const int* __restrict__ col,
                            const V* __restrict__ val, const int* __restrict__ sptr, int* __restrict__ scol,
                            W* __restrict__ sval) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= ((n + 31) & ~31)) return;
    const int sl = row >> 5, l = row & 31;
    const int b = sptr[sl], w = (sptr[sl + 1] - b) >> 5;
    const int rb = (row < n) ? ptr[row] : 0, len = (row < n) ? ptr[row + 1] - rb : 0;
    for (int j = 0; j < w; ++j) {
        const int k = b + 32 * j + l;
        // padding reads column 0, which exists for every operator (P and R are not square)
        if (j < len) { scol[k] = col[rb + j]; sval[k] = (W)val[rb + j]; }
        else { scol[k] = 0; sval[k] = W(0); }
    }
}

// ------------------------------------------------------------ host side
template <class V>
struct Sell {
    int n = 0, nslices = 0;
    DBuf<int> sptr, col;
    DBuf<V> val;
    SellView<V> view() const { return SellView<V>{sptr.p, col.p, val.p, n}; }
};

template <class V>
CsrView<V, 4> csr4(const DCsr<V>& A) { return CsrView<V, 4>{A.ptr.p, A.col.p, A.val.p, A.n}; }

template <class V>
int pick_vs(const DCsr<V>& A) {
    const double avg = A.n ? (double)A.nnz / A.n : 1.0;
    return avg <= 6 ? 4 : (avg <= 12 ? 8 : (avg <= 24 ? 16 : 32));
}

// launch a row kernel on a CSR matrix with the lanes-per-row that suits it
template <class V, class F>
void with_csr(const DCsr<V>& A, F&& f) {
    switch (pick_vs(A)) {
        case 4: f(CsrView<V, 4>{A.ptr.p, A.col.p, A.val.p, A.n}); break;
        case 8: f(CsrView<V, 8>{A.ptr.p, A.col.p, A.val.p, A.n}); break;
        case 16: f(CsrView<V, 16>{A.ptr.p, A.col.p, A.val.p, A.n}); break;
        default: f(CsrView<V, 32>{A.ptr.p, A.col.p, A.val.p, A.n}); break;
    }
}
template <class M>
int grid_for(const M& A) { return blocks((int64_t)A.n * M::kVS, 256); }

// SELL-32 copy of a CSR matrix's structure and values (value type W); hpin:
// a pinned int of the calling thread for the slice scan's total
template <class V, class W>
void build_sell(cudaStream_t s, const int* ptr, const int* col, const V* val, int n, Sell<W>& S, int* hpin) {
    S.n = n;
    S.nslices = (n + 31) / 32;
    S.sptr.alloc(S.nslices + 1, s);
    SEMO_CUDA(cudaMemsetAsync(S.sptr.p + S.nslices, 0, sizeof(int), s));
    const int rows_pad = S.nslices * 32;
    k_sell_width<<<blocks(rows_pad, 256), 256, 0, s>>>(n, ptr, S.sptr.p);
    SEMO_CHECK_LAUNCH();
    const int total = device_scan(s, S.sptr.p, S.nslices + 1, hpin);
    S.col.alloc(std::max(total, 1), s);
    S.val.alloc(std::max(total, 1), s);
    k_sell_fill<V, W><<<blocks(rows_pad, 256), 256, 0, s>>>(n, ptr, col, val, S.sptr.p, S.col.p, S.val.p);
    SEMO_CHECK_LAUNCH();
}

// One warp per slice (blocks of whole warps): the slice's encoding, the base
// column (smallest column) of every (slice, j) group and the slice's 32-bit
// column count in wsz (0 unless its encoding is 2).  most (or null): the widest
// slice, and whether any has another encoding than 0.
__global__ void k_sell16_groups(int n, const int* __restrict__ ptr, const int* __restrict__ col,
                                const int* __restrict__ sptr, int* __restrict__ smode, int* __restrict__ gbase,
                                int* __restrict__ wsz, int* most) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    const int sl = row >> 5;
    if (sl >= ((n + 31) >> 5)) return;   // whole warps: the test is uniform in a warp
    const int b = sptr[sl], w = (sptr[sl + 1] - b) >> 5;
    const int rb = (row < n) ? ptr[row] : 0, len = (row < n) ? ptr[row + 1] - rb : 0;
    bool wide = false, near = true;
    for (int j = 0; j < w; ++j) {
        const int c = (j < len) ? col[rb + j] : -1;
        const int mn = __reduce_min_sync(0xffffffffu, (c >= 0) ? c : INT_MAX);
        const int mx = __reduce_max_sync(0xffffffffu, c);
        wide |= (long long)mx - (long long)mn > 65535;
        near &= (c < 0) || (c - row >= -32768 && c - row <= 32767);
        if ((threadIdx.x & 31) == 0) gbase[(b >> 5) + j] = mn;
    }
    near = __all_sync(0xffffffffu, near);
    const int mode = near ? 0 : (wide ? 2 : 1);
    if ((threadIdx.x & 31) == 0) {
        smode[sl] = mode;
        wsz[sl] = (mode == 2) ? 32 * w : 0;
        if (most) {
            if (most[0] < w) atomicMax(most, w);
            if (mode != 0) most[1] = 1;
        }
    }
}
__global__ void k_sell16_even(int nslices, int width, int* __restrict__ sptr) {
    const int sl = blockIdx.x * blockDim.x + threadIdx.x;
    if (sl <= nslices) sptr[sl] = 32 * width * sl;
}

__global__ void k_sell16_cols(int n, const int* __restrict__ ptr, const int* __restrict__ col,
                              const int* __restrict__ sptr, const int* __restrict__ smode,
                              const int* __restrict__ gbase, const int* __restrict__ wptr,
                              unsigned short* __restrict__ dcol, int* __restrict__ wcol) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= ((n + 31) & ~31)) return;
    const int sl = row >> 5, l = row & 31;
    const int b = sptr[sl], w = (sptr[sl + 1] - b) >> 5;
    const int mode = smode[sl];
    const int rb = (row < n) ? ptr[row] : 0, len = (row < n) ? ptr[row + 1] - rb : 0;
    for (int j = 0; j < w; ++j) {
        const int k = b + 32 * j + l;
        const int base = (mode == 0) ? row : gbase[(b >> 5) + j];
        const int c = (j < len) ? col[rb + j] : base;
        dcol[k] = (mode == 2) ? (unsigned short)0 : (unsigned short)(c - base);
        if (mode == 2) wcol[wptr[sl] + 32 * j + l] = c;
    }
}
// the values into a layout's slots (padding slots 0)
template <class V, class W>
__global__ void k_sell16_vals(int n, const int* __restrict__ ptr, const V* __restrict__ val,
                              const int* __restrict__ sptr, W* __restrict__ sval) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= ((n + 31) & ~31)) return;
    const int sl = row >> 5, l = row & 31;
    const int b = sptr[sl], w = (sptr[sl + 1] - b) >> 5;
    const int rb = (row < n) ? ptr[row] : 0, len = (row < n) ? ptr[row + 1] - rb : 0;
    for (int j = 0; j < w; ++j) sval[b + 32 * j + l] = (j < len) ? (W)val[rb + j] : W(0);
}

// The structure of a SELL-32 layout with 16-bit columns (slice pointers,
// per-slice encodings, group bases, 16- and 32-bit columns).  It depends on
// the pattern only, so the FP64 outer operator and the finest level of the
// pressure hierarchy, both on the mesh's pattern, share one, built once per
// mesh; a setup then only writes the two value arrays.
struct Sell16Struct {
    int n = 0, nslices = 0;
    int slots = 0;   // padded entries (sptr[nslices])
    int width = 0;   // every slice's, when they are made equal (all of mode 0)
    DBuf<int> sptr, smode, gbase, wptr, wcol;
    DBuf<unsigned short> dcol;
};
template <class V>
struct Sell16 {
    std::shared_ptr<Sell16Struct> st;
    DBuf<V> val;
    Sell16View<V> view() const {
        return Sell16View<V>{st->sptr.p, st->smode.p, st->gbase.p, st->wptr.p, st->dcol.p, st->wcol.p, val.p,
                             st->n};
    }
    // run f on the view that suits the structure
    template <class F>
    void with(F&& f) const {
        switch (st->width) {
            case 5: f(Sell16UView<V, 5>{st->dcol.p, val.p, st->n}); break;
            case 6: f(Sell16UView<V, 6>{st->dcol.p, val.p, st->n}); break;
            case 7: f(Sell16UView<V, 7>{st->dcol.p, val.p, st->n}); break;
            default: f(view());
        }
    }
};

// SELL-32 structure with 16-bit columns of a square CSR pattern (slices that
// fit no 16-bit encoding keep 32-bit columns).  hmost (two pinned ints, or
// null): make the slices equally wide where Sell16UView has that width and
// every slice has encoding 0 (even_slots).
std::shared_ptr<Sell16Struct> build_sell16_struct(cudaStream_t s, const int* ptr, const int* col, int n,
                                                  int* hpin, int* hmost) {
    auto S = std::make_shared<Sell16Struct>();
    S->n = n;
    S->nslices = (n + 31) / 32;
    S->sptr.alloc(S->nslices + 1, s);
    S->wptr.alloc(S->nslices + 1, s);
    S->smode.alloc(S->nslices + 2, s);   // and the widest slice, any encoding but 0
    int* const most = hmost ? S->smode.p + S->nslices : nullptr;
    if (most) SEMO_CUDA(cudaMemsetAsync(most, 0, 2 * sizeof(int), s));
    SEMO_CUDA(cudaMemsetAsync(S->sptr.p + S->nslices, 0, sizeof(int), s));
    SEMO_CUDA(cudaMemsetAsync(S->wptr.p + S->nslices, 0, sizeof(int), s));
    const int rows_pad = S->nslices * 32;
    k_sell_width<<<blocks(rows_pad, 256), 256, 0, s>>>(n, ptr, S->sptr.p);
    SEMO_CHECK_LAUNCH();
    S->slots = device_scan(s, S->sptr.p, S->nslices + 1, hpin);
    S->gbase.alloc(std::max(S->slots / 32, 1), s);
    k_sell16_groups<<<blocks(rows_pad, 256), 256, 0, s>>>(n, ptr, col, S->sptr.p, S->smode.p, S->gbase.p,
                                                          S->wptr.p, most);
    SEMO_CHECK_LAUNCH();
    if (most) SEMO_CUDA(cudaMemcpyAsync(hmost, most, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
    const int wide = device_scan(s, S->wptr.p, S->nslices + 1, hpin);   // its sync lands hmost too
    const int64_t even = most && hmost[1] == 0 ? even_slots(hmost[0], 5, 7, S->nslices, S->slots) : 0;
    if (even) {
        S->width = hmost[0];
        S->slots = (int)even;
        k_sell16_even<<<blocks(S->nslices + 1, 256), 256, 0, s>>>(S->nslices, S->width, S->sptr.p);
        SEMO_CHECK_LAUNCH();
    }
    S->dcol.alloc(std::max(S->slots, 1), s);
    S->wcol.alloc(std::max(wide, 1), s);
    k_sell16_cols<<<blocks(rows_pad, 256), 256, 0, s>>>(n, ptr, col, S->sptr.p, S->smode.p, S->gbase.p, S->wptr.p,
                                                         S->dcol.p, S->wcol.p);
    SEMO_CHECK_LAUNCH();
    return S;
}
// the values of a CSR operator on the structure's pattern into S (type W)
template <class V, class W>
void fill_sell16(cudaStream_t s, const int* ptr, const V* val, const std::shared_ptr<Sell16Struct>& st,
                 Sell16<W>& S) {
    S.st = st;
    S.val.alloc(std::max(st->slots, 1), s);
    k_sell16_vals<V, W><<<blocks((int64_t)st->nslices * 32, 256), 256, 0, s>>>(st->n, ptr, val, st->sptr.p,
                                                                              S.val.p);
    SEMO_CHECK_LAUNCH();
}
template <class V, class W>
bool build_sell16(cudaStream_t s, const int* ptr, const int* col, const V* val, int n, Sell16<W>& S, int* hpin,
                  int* hmost) {
    fill_sell16<V, W>(s, ptr, val, build_sell16_struct(s, ptr, col, n, hpin, hmost), S);
    return true;
}

// The FP64 outer operator
struct OuterOp {
    Sell16<double> s16;
    template <class F>
    void with(F&& f) const { s16.with(f); }
};

struct ChebCoef {
    double inv_theta, c1, c2;
};
ChebCoef cheb2(double lam) {
    const double hi = lam, lo = lam / 30.0;
    const double theta = 0.5 * (hi + lo), delta = 0.5 * (hi - lo);
    const double sigma = theta / delta, rho0 = 1.0 / sigma;
    const double rho1 = 1.0 / (2.0 * sigma - rho0);
    return ChebCoef{1.0 / theta, rho1 * rho0, 2.0 * rho1 / delta};
}

// Everything the V-cycle needs beyond the hierarchy: SELL copies of the
// operators it pays for.  SELL runs one thread per row, so it needs enough
// rows to fill the GPU (65536 rows = 2048 warps, ~13 per SM) unless rows are
// short; a few thousand long rows (a coarse level, ~60 entries each) would
// leave ~2 warps per SM walking 60 dependent loads, and run faster as CSR
// with 32 lanes a row.  Small operators are launch-latency bound either way
// and stay CSR.
constexpr int kSellMinRows = 4096;
constexpr int kSellFullRows = 65536;
constexpr double kSellMaxAvgRow = 12.0;
template <class V>
bool sell_pays(const DCsr<V>& M) {
    if (M.n < kSellMinRows) return false;
    return M.n >= kSellFullRows || (double)M.nnz <= kSellMaxAvgRow * (double)M.n;
}
template <class V>
struct LevelMats {
    Sell<V> A, P, R;
    Sell16<V> A16;
    bool a = false, p = false, r = false, a16 = false;
    // multicolour Gauss-Seidel (semo_params.smoother == 1): the level's rows
    // grouped by colour, colour k at crow[cptr[k] .. cptr[k + 1])
    bool gs = false;
    DBuf<int> crow;
    std::vector<int> cptr;
};
template <class V>
struct Cycle {
    std::vector<LevelMats<V>> lev;
    int local_from = -1;   // first level of k_local_cycle
};

#include "cycle_cluster.cuh"

// run f on the SELL view of a level operator if it has one, else on CSR
template <class V, class F>
void with_op(const Sell<V>& S, bool use_sell, const DCsr<V>& M, F&& f) {
    if (use_sell) f(S.view());
    else with_csr(M, f);
}
// the level's A: 16-bit-offset SELL, SELL, or CSR
template <class V, class F>
void with_A(const LevelMats<V>& M, const DCsr<V>& A, F&& f) {
    if (M.a16) M.A16.with(f);
    else with_op(M.A, M.a, A, f);
}

// ---------------------------------------------- multicolour Gauss-Seidel
__device__ __forceinline__ uint32_t color_hash(uint32_t x) {
    // integer avalanche mixer (public-domain "lowbias32" constants), as the MIS uses
    x ^= x >> 16; x *= 0x7feb352dU; x ^= x >> 15; x *= 0x846ca68bU; x ^= x >> 16;
    return x;
}
// One synchronous Jones-Plassmann round on the pattern of A: an uncoloured row
// whose (hash, index) key is larger than every uncoloured neighbour's takes
// the smallest colour no neighbour coloured in an earlier round holds (the
// rows coloured in one round are independent, so they never clash).  Reads
// cold, writes cnew (a copy of cold); counts the rows still uncoloured and
// flags a row that would need a colour beyond 127.
__global__ void k_color_round(int n, const int* __restrict__ ptr, const int* __restrict__ col,
                              const int* __restrict__ cold, int* __restrict__ cnew, int* __restrict__ left,
                              int* __restrict__ overflow) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || cold[i] >= 0) return;
    const unsigned long long ki = ((unsigned long long)color_hash((uint32_t)i) << 32) | (unsigned)i;
    unsigned long long used0 = 0, used1 = 0;
    bool top = true;
    for (int k = ptr[i]; k < ptr[i + 1]; ++k) {
        const int j = col[k];
        if (j == i) continue;
        const int cj = cold[j];
        if (cj < 0) {
            const unsigned long long kj = ((unsigned long long)color_hash((uint32_t)j) << 32) | (unsigned)j;
            if (kj > ki) { top = false; break; }
        } else if (cj < 64) {
            used0 |= 1ull << cj;
        } else if (cj < 128) {
            used1 |= 1ull << (cj - 64);
        }
    }
    if (!top) { atomicAdd(left, 1); return; }
    int c = -1;
    if (~used0) c = __ffsll((long long)~used0) - 1;
    else if (~used1) c = 64 + __ffsll((long long)~used1) - 1;
    if (c < 0) { atomicExch(overflow, 1); c = 127; }
    cnew[i] = c;
}

// One colour of a Gauss-Seidel sweep: x_i += (b_i - (A x)_i) / a_ii for the
// rows of that colour (no two of them are coupled, so the order is free)
template <class M, class V>
__global__ void __launch_bounds__(256) k_gs_color(M A, const int* __restrict__ rows, int nrows,
                                                  const V* __restrict__ dinv, const V* __restrict__ b,
                                                  V* __restrict__ x) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = g / M::kVS, lane = g % M::kVS;
    const int row = (t < nrows) ? rows[t] : A.n;   // rows past the list: an empty dot
    const V s = A.dot(row, lane, Vec<V, V>{x});
    if (t < nrows && lane == 0) x[row] += dinv[row] * (b[row] - s);
}
// Under the Gauss-Seidel option only the finest level, when it has more than
// this many rows, is swept by colours; the coarser levels keep Chebyshev.
// A sweep is one launch per colour: the finest mesh graph needs a handful of
// colours, a coarse level (denser rows) 20-40, each colour a launch of a few
// thousand rows, and there the sweeps cost launch latency, not bandwidth
// (measured at 128^3: 50 extra launches per V-cycle, twice the solve time).
constexpr int kGsMinRows = 16384;

template <class V>
void color_level(semo_ctx* c, cudaStream_t s, const DCsr<V>& A, LevelMats<V>& M) {
    const int n = A.n;
    DBuf<int> c0, c1, cnt;
    c0.alloc(n, s);
    c1.alloc(n, s);
    cnt.alloc(2, s);
    SEMO_CUDA(cudaMemsetAsync(c0.p, 0xff, sizeof(int) * n, s));   // -1: uncoloured
    int h[2] = {1, 0};
    int* cold = c0.p;
    int* cnew = c1.p;
    // rounds in batches of 4 between host checks (a round over a fully
    // coloured graph changes nothing)
    for (int batch = 0; h[0] > 0; ++batch) {
        if (batch > 1024) throw Error(SEMO_ERR_CUDA, "graph colouring did not finish");
        for (int r = 0; r < 4; ++r) {
            SEMO_CUDA(cudaMemcpyAsync(cnew, cold, sizeof(int) * n, cudaMemcpyDeviceToDevice, s));
            SEMO_CUDA(cudaMemsetAsync(cnt.p, 0, 2 * sizeof(int), s));
            k_color_round<<<blocks(n, 256), 256, 0, s>>>(n, A.ptr, A.col, cold, cnew, cnt.p, cnt.p + 1);
            SEMO_CHECK_LAUNCH();
            std::swap(cold, cnew);
        }
        SEMO_CUDA(cudaMemcpyAsync(h, cnt.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
        SEMO_CUDA(cudaStreamSynchronize(s));
        if (h[1]) throw Error(SEMO_ERR_CUDA, "graph colouring needs more than 128 colours");
    }
    // rows grouped by colour (counting sort on the host; the order inside a colour is free)
    std::vector<int> hc(n);
    SEMO_CUDA(cudaMemcpyAsync(hc.data(), cold, sizeof(int) * n, cudaMemcpyDeviceToHost, s));
    SEMO_CUDA(cudaStreamSynchronize(s));
    int ncol = 0;
    for (int v : hc) ncol = std::max(ncol, v + 1);
    M.cptr.assign(ncol + 1, 0);
    for (int v : hc) M.cptr[v + 1]++;
    for (int k = 0; k < ncol; ++k) M.cptr[k + 1] += M.cptr[k];
    std::vector<int> fill(M.cptr.begin(), M.cptr.end() - 1), rows(n);
    for (int i = 0; i < n; ++i) rows[fill[hc[i]]++] = i;
    M.crow.upload(rows.data(), n, s);
    SEMO_CUDA(cudaStreamSynchronize(s));   // the host vector above is freed on return
    M.gs = true;
}

// one Gauss-Seidel sweep of level L (forward: colours ascending)
template <class V>
void gs_sweep(cudaStream_t s, AmgLevel<V>& L, const LevelMats<V>& M, bool backward, bool zero_start) {
    const int n = L.A.n;
    const int ncol = (int)M.cptr.size() - 1;
    if (zero_start) {
        k_zero<V><<<blocks(n, 256), 256, 0, s>>>(n, L.x.p);
        SEMO_CHECK_LAUNCH();
    }
    for (int q = 0; q < ncol; ++q) {
        const int k = backward ? ncol - 1 - q : q;
        const int nr = M.cptr[k + 1] - M.cptr[k];
        if (nr == 0) continue;
        with_csr(L.A, [&](auto A) {
            using MV = decltype(A);
            k_gs_color<<<blocks((int64_t)nr * MV::kVS, 256), 256, 0, s>>>(A, M.crow.p + M.cptr[k], nr, L.dinv.p,
                                                                          L.b.p, L.x.p);
        });
        SEMO_CHECK_LAUNCH();
    }
}

template <class V>
void chebyshev_generic(cudaStream_t s, AmgLevel<V>& L, int degree, bool zero_start) {
    const int n = L.A.n;
    const double hi = L.lam_max, lo = hi / 30.0;
    const double theta = 0.5 * (hi + lo), delta = 0.5 * (hi - lo);
    const double sigma = theta / delta;
    double rho = 1.0 / sigma;
    V* x = L.x.p;
    V* d = L.t.p;
    if (zero_start) {
        k_zero<V><<<blocks(n, 256), 256, 0, s>>>(n, x);
        SEMO_CHECK_LAUNCH();
    }
    k_zero<V><<<blocks(n, 256), 256, 0, s>>>(n, d);
    SEMO_CHECK_LAUNCH();
    // d = D^-1 (b - A x) / theta ; x += d
    with_csr(L.A, [&](auto M) {
        k_cheb_d<<<grid_for(M), 256, 0, s>>>(M, L.dinv.p, L.b.p, x, V(0), (V)(1.0 / theta), d);
    });
    SEMO_CHECK_LAUNCH();
    k_axpy1<V><<<blocks(n, 256), 256, 0, s>>>(n, d, x);
    SEMO_CHECK_LAUNCH();
    for (int k = 1; k < degree; ++k) {
        const double rho_new = 1.0 / (2.0 * sigma - rho);
        const V c1 = (V)(rho_new * rho), c2 = (V)(2.0 * rho_new / delta);
        with_csr(L.A, [&](auto M) { k_cheb_d<<<grid_for(M), 256, 0, s>>>(M, L.dinv.p, L.b.p, x, c1, c2, d); });
        SEMO_CHECK_LAUNCH();
        k_axpy1<V><<<blocks(n, 256), 256, 0, s>>>(n, d, x);
        SEMO_CHECK_LAUNCH();
        rho = rho_new;
    }
}

// what writes level l's b writes beside it: d0, on the levels that k_pre2 starts
template <class V>
FirstIterate<V> first_iterate(semo_ctx* c, Amg<V>& h, const Cycle<V>& cy, int l) {
    AmgLevel<V>& L = h.lev[l];
    if (l == (int)h.lev.size() - 1 || l == cy.local_from || cy.lev[l].gs || c->prm.cheb_degree != 2)
        return FirstIterate<V>{nullptr, V(0), nullptr};
    return FirstIterate<V>{L.dinv.p, (V)cheb2(L.lam_max).inv_theta, L.t.p};
}

// V-cycle from level l down, input L.b (and d0 below the finest level), output L.x
template <class V>
void vcycle_from(semo_ctx* c, Amg<V>& h, Cycle<V>& cy, int l) {
    cudaStream_t s = c->stream;
    AmgLevel<V>& L = h.lev[l];
    if (l == cy.local_from) {   // this level and those below in one kernel
        ClArgs<V> a;
        if (!cl_args<V>(h, l, false, a, nullptr)) throw Error(SEMO_ERR_STATE, "V-cycle: the small levels do not fit");
        launch_cluster(k_local_cycle<V>, s, 1, a.smem, true, a);
        return;
    }
    if (l == (int)h.lev.size() - 1) {
        launch_pdl(k_coarse_solve<V>, 1, 256, s, h.coarse_n, h.cinv.p, L.b.p, L.x.p);
        return;
    }
    const LevelMats<V>& M = cy.lev[l];
    const int degree = c->prm.cheb_degree;
    const ChebCoef cc = cheb2(L.lam_max);
    if (M.gs) {
        gs_sweep(s, L, M, false, true);   // forward sweep from x = 0
    } else if (degree == 2) {
        with_A(M, L.A, [&](auto A) {
            if (l == 0)
                launch_pdl(k_pre2<decltype(A), V, FirstGather<V>>, grid_for(A), 256, s, A, L.dinv.p, L.b.p,
                           FirstGather<V>{L.dinv.p, L.b.p, (V)cc.inv_theta}, (V)cc.c1, (V)cc.c2, L.x.p);
            else
                launch_pdl(k_pre2<decltype(A), V, Vec<V, V>>, grid_for(A), 256, s, A, L.dinv.p, L.b.p,
                           Vec<V, V>{L.t.p}, (V)cc.c1, (V)cc.c2, L.x.p);
        });
    } else {
        chebyshev_generic(s, L, degree, true);
    }
    with_A(M, L.A, [&](auto A) { launch_pdl(k_res<decltype(A), V>, grid_for(A), 256, s, A, L.x.p, L.b.p, L.r.p); });
    AmgLevel<V>& C = h.lev[l + 1];
    with_op(M.R, M.r, L.R, [&](auto R) {
        launch_pdl(k_mv<decltype(R), V>, grid_for(R), 256, s, R, L.r.p, C.b.p, first_iterate(c, h, cy, l + 1));
    });
    vcycle_from(c, h, cy, l + 1);
    with_op(M.P, M.p, L.P,
            [&](auto P) { launch_pdl(k_prolong_add<decltype(P), V>, grid_for(P), 256, s, P, C.x.p, L.x.p); });
    if (M.gs) {
        gs_sweep(s, L, M, true, false);   // backward sweep: the cycle stays symmetric
    } else if (degree == 2) {
        with_A(M, L.A, [&](auto A) {
            launch_pdl(k_post0<decltype(A), V>, grid_for(A), 256, s, A, L.dinv.p, L.b.p, (V)cc.inv_theta, L.x.p,
                       L.t.p, L.r.p);
        });
        if (l > 0) {
            with_A(M, L.A, [&](auto A) {
                launch_pdl(k_post1<decltype(A), V>, grid_for(A), 256, s, A, L.dinv.p, L.b.p, (V)cc.c1, (V)cc.c2,
                           L.r.p, L.t.p, L.x.p);
            });
        }
        // on the finest level the last step is fused with the CG dot products (cg_iteration)
    } else {
        chebyshev_generic(s, L, degree, false);
    }
}

struct Red {
    double* part;
    double* scal;
};
Red red_area(semo_ctx* c) {
    c->red.alloc(4 * kRedBlocks + 32, c->stream);
    return Red{c->red.p, c->red.p + 4 * kRedBlocks + 8};
}

// One preconditioned CG iteration.  In: r (FP64) and its copy L0.b in V; out: x, r, L0.b updated.
template <class V>
void cg_iteration(semo_ctx* c, Amg<V>& h, Cycle<V>& cy, const OuterOp& outer, double* x, const Red& R) {
    cudaStream_t s = c->stream;
    AmgLevel<V>& L = h.lev[0];
    const int n = L.A.n;
    double* r = c->kr.p;
    double* p = c->kp.p;
    double* q = c->kq.p;
    const int degree = c->prm.cheb_degree;
    const bool single = h.lev.size() == 1;
    const int nb = red_blocks(n);
    if (single) {
        k_coarse_solve<V><<<1, 256, 0, s>>>(h.coarse_n, h.cinv, L.b, L.x);
        SEMO_CHECK_LAUNCH();
        k_dot2<V><<<nb, kRedThreads, 0, s>>>(n, L.x.p, r, q, R.part);
        SEMO_CHECK_LAUNCH();
    } else if (degree == 2 && !cy.lev[0].gs) {
        const ChebCoef cc = cheb2(L.lam_max);
        vcycle_from(c, h, cy, 0);   // everything but the last smoothing step of the finest level
        // z lands in L.x; z.r and z.q folded in
        with_A(cy.lev[0], L.A, [&](auto A) {
            launch_pdl(k_post1_dots<decltype(A), V>, nb, kRedThreads, s, A, L.dinv.p, L.b.p, (V)cc.c1, (V)cc.c2,
                       L.r.p, L.t.p, L.x.p, r, q, R.part);
        });
    } else {
        vcycle_from(c, h, cy, 0);
        k_dot2<V><<<nb, kRedThreads, 0, s>>>(n, L.x.p, r, q, R.part);
        SEMO_CHECK_LAUNCH();
    }
    outer.with([&](auto A) {
        launch_pdl(k_outer_mv<decltype(A), V>, nb, kRedThreads, s, A, L.x.p, p, q, R.scal, R.part, nb,
                   R.part + 2 * kRedBlocks);
    });
    launch_pdl(k_xr<V>, nb, kRedThreads, s, n, x, r, L.b.p, p, q, R.scal, R.part + 2 * kRedBlocks, nb,
               R.part + 3 * kRedBlocks);
}

struct GraphGuard {
    cudaGraph_t g = nullptr;
    cudaGraphExec_t e = nullptr;
    ~GraphGuard() {
        if (e) cudaGraphExecDestroy(e);
        if (g) cudaGraphDestroy(g);
    }
};

// The loop's stopping threshold on r.r: (tol |b|)^2, |b| = 1 for b = 0
// (scal[11] = b.b)
__device__ __forceinline__ double cg_stop_rr(const double* scal, double tol) {
    const double bn = sqrt(scal[11]);
    const double bnorm = (bn > 0.0) ? bn : 1.0;
    return (tol * bnorm) * (tol * bnorm);
}
// Before the loop: iterate at all? (no when r0 already meets the tolerance,
// or b or r0 is not finite -- the host reports that after the graph)
__global__ void k_cg_begin(cudaGraphConditionalHandle h, const double* __restrict__ scal, double tol, int max_iter) {
    const double bn = sqrt(scal[11]), rn = sqrt(scal[12]);
    const double bnorm = (bn > 0.0) ? bn : 1.0;
    const bool go = isfinite(bn) && isfinite(rn) && rn > tol * bnorm && max_iter > 0;
    cudaGraphSetConditional(h, go ? 1u : 0u);
}
// End of one CG iteration on the device: count it and decide whether the
// loop goes on (scal[13] iterations, scal[14] status: 1 NaN/Inf, 2 p.q <= 0).
// The loop is a conditional WHILE node, so no iteration waits for the host;
// max_iter bounds it.
// One warp; prr: the iteration's partial sums of r.r.
__global__ void k_cg_check(cudaGraphConditionalHandle h, double* __restrict__ scal, const double* __restrict__ prr,
                           int nb, double tol, int max_iter) {
    pdl_enter();
    const double rr = parts_sum(prr, nb);
    if (threadIdx.x != 0) return;
    const double stop_rr = cg_stop_rr(scal, tol);
    const double it = scal[13] + 1.0;
    scal[13] = it;
    const double pq = scal[2];
    unsigned go = 1;
    if (!isfinite(rr) || !isfinite(pq)) { scal[14] = 1.0; go = 0; }
    else if (!(pq > 0.0)) { scal[14] = 2.0; go = 0; }
    else if (!(rr > stop_rr) || it >= (double)max_iter) go = 0;
    cudaGraphSetConditional(h, go);
}

// what a solve reports: h2 the scalars read back, nodes the loop's kernels
void pcg_outcome(const double* h2, size_t nodes, semo_solve_info* info) {
    const double bn = std::sqrt(h2[11]), rn0 = std::sqrt(h2[12]);
    if (!std::isfinite(bn) || !std::isfinite(rn0)) throw Error(SEMO_ERR_NAN, "non-finite right-hand side");
    const int it = (int)h2[13];
    if (nodes) __atomic_add_fetch(&g_kernel_launches, 1LL + (long long)nodes * it, __ATOMIC_RELAXED);
    if (h2[14] == 1.0) throw Error(SEMO_ERR_NAN, "NaN/Inf in the Krylov residual");
    if (h2[14] == 2.0) throw Error(SEMO_ERR_BREAKDOWN, "CG breakdown: p.Ap <= 0 (matrix not SPD?)");
    info->iterations = it;
    info->rel_residual = (bn > 0.0) ? std::sqrt(h2[16]) / bn : 0.0;
}

// systems that k_cluster_cg solves whole: its arguments
template <class V>
bool cluster_cg_fits(const semo_ctx* c, const Amg<V>& h, const Cycle<V>& cy, ClArgs<V>& a, ClCg& g) {
    if (c->prm.cheb_degree != 2 || (!cy.lev.empty() && cy.lev[0].gs)) return false;
    return h.lev[0].A.n <= kClBlocks * kClThreads && cl_args<V>(h, 0, h.lev.size() > 1, a, &g);
}

// same: the hierarchy and outer were built from this matrix (ptr, col, val).
// Without it they may belong to another one with as many rows, whose pattern
// k_cluster_cg would not fit and whose residual is not this matrix's: the
// iteration then runs on outer, and the residuals are formed with the caller's
// matrix, so that a solution of the other system is not taken for converged.
template <class V>
void pcg(semo_ctx* c, Amg<V>& h, Cycle<V>& cy, const OuterOp& outer, bool same, const int* ptr, const int* col,
         const double* val, int n, const double* b, double* x, bool zero_guess, semo_solve_info* info) {
    cudaStream_t s = c->stream;
    Red R = red_area(c);
    c->kr.alloc(n, s); c->kp.alloc(n, s); c->kq.alloc(n, s);
    double* h2 = c->hpin;
    double* r = c->kr.p;
    const int nb = red_blocks(n);
    size_t body_nodes = 0;
    ClArgs<V> ca;
    ClCg g{};
    g.A.gptr = ptr;
    g.A.gcol = col;
    g.A.gval = val;
    g.b = b;
    g.x = x;
    g.scal = R.scal;
    g.tol = c->prm.tol;
    g.max_iter = c->prm.max_iter;
    g.zero_guess = zero_guess;
    if (same && cluster_cg_fits(c, h, cy, ca, g)) {   // the whole solve in one kernel
        SEMO_CUDA(cudaMemsetAsync(R.scal, 0, sizeof(double) * 17, s));
        launch_cluster(k_cluster_cg<V>, s, kClBlocks, ca.smem, false, ca, g);
        SEMO_CUDA(cudaMemcpyAsync(h2, R.scal, sizeof(double) * 17, cudaMemcpyDeviceToHost, s));
        SEMO_CUDA(cudaStreamSynchronize(s));
        pcg_outcome(h2, 0, info);
        return;
    }
    auto residual = [&] {
        bool done = false;
        if (same)
            outer.with([&](auto A) {
                if constexpr (decltype(A)::kEven > 0) {
                    k_res64_even<decltype(A)::kEven><<<blocks(n, 256), 256, 0, s>>>(A, x, b, r);
                    done = true;
                }
            });
        if (!done) k_res64<<<blocks((int64_t)n * 8, 256), 256, 0, s>>>(CsrView<double, 8>{ptr, col, val, n}, x, b, r);
        SEMO_CHECK_LAUNCH();
    };
    if (zero_guess) {
        SEMO_CUDA(cudaMemsetAsync(x, 0, sizeof(double) * n, s));
        SEMO_CUDA(cudaMemcpyAsync(r, b, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    } else {
        residual();
    }
    k_conv<double, V><<<blocks(n, 256), 256, 0, s>>>(n, r, h.lev[0].b.p);
    SEMO_CHECK_LAUNCH();
    SEMO_CUDA(cudaMemsetAsync(c->kq.p, 0, sizeof(double) * n, s));
    SEMO_CUDA(cudaMemsetAsync(c->kp.p, 0, sizeof(double) * n, s));
    SEMO_CUDA(cudaMemsetAsync(R.scal, 0, sizeof(double) * 17, s));
    k_dot<<<nb, kRedThreads, 0, s>>>(n, b, b, R.part);
    SEMO_CHECK_LAUNCH();
    k_dot<<<nb, kRedThreads, 0, s>>>(n, r, r, R.part + kRedBlocks);
    SEMO_CHECK_LAUNCH();
    k_fin_sum<<<1, kRedThreads, 0, s>>>(R.part, nb, R.scal + 11);   // ||b||^2
    SEMO_CHECK_LAUNCH();
    k_fin_sum<<<1, kRedThreads, 0, s>>>(R.part + kRedBlocks, nb, R.scal + 12);   // ||r0||^2
    SEMO_CHECK_LAUNCH();
    // The loop is one graph: k_cg_begin, then a conditional WHILE node whose
    // body is one CG iteration plus k_cg_check, which decides on
    // the device whether to go on.  It is captured and instantiated while the
    // kernels above run, and the host waits once, after the true residual.
    GraphGuard gg;
    SEMO_CUDA(cudaGraphCreate(&gg.g, 0));
    cudaGraphConditionalHandle handle;
    SEMO_CUDA(cudaGraphConditionalHandleCreate(&handle, gg.g, 0, cudaGraphCondAssignDefault));
    cudaKernelNodeParams kb = {};
    const double tol = c->prm.tol;
    const int max_iter = c->prm.max_iter;
    const double* scal_c = R.scal;
    void* kb_args[] = {(void*)&handle, (void*)&scal_c, (void*)&tol, (void*)&max_iter};
    kb.func = (void*)k_cg_begin;
    kb.gridDim = dim3(1);
    kb.blockDim = dim3(1);
    kb.kernelParams = kb_args;
    cudaGraphNode_t begin;
    SEMO_CUDA(cudaGraphAddKernelNode(&begin, gg.g, nullptr, 0, &kb));
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = handle;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t loop;
    SEMO_CUDA(cudaGraphAddNode(&loop, gg.g, &begin, nullptr, 1, &cp));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    const long long before = __atomic_load_n(&g_kernel_launches, __ATOMIC_RELAXED);
    SEMO_CUDA(cudaStreamBeginCaptureToGraph(s, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    try {
        cg_iteration(c, h, cy, outer, x, R);
        launch_pdl(k_cg_check, 1, 32, s, handle, R.scal, R.part + 3 * kRedBlocks, nb, tol, max_iter);
    } catch (...) {
        cudaGraph_t junk = nullptr;
        cudaStreamEndCapture(s, &junk);
        throw;
    }
    cudaGraph_t captured = nullptr;
    SEMO_CUDA(cudaStreamEndCapture(s, &captured));
    SEMO_CUDA(cudaGraphGetNodes(body, nullptr, &body_nodes));
    __atomic_store_n(&g_kernel_launches, before, __ATOMIC_RELAXED);
    SEMO_CUDA(cudaGraphInstantiate(&gg.e, gg.g, 0));
    SEMO_CUDA(cudaGraphLaunch(gg.e, s));
    // true FP64 residual of the returned solution -> scal[16]
    residual();
    k_dot<<<nb, kRedThreads, 0, s>>>(n, r, r, R.part);
    SEMO_CHECK_LAUNCH();
    k_fin_sum<<<1, kRedThreads, 0, s>>>(R.part, nb, R.scal + 16);
    SEMO_CHECK_LAUNCH();
    SEMO_CUDA(cudaMemcpyAsync(h2, R.scal, sizeof(double) * 17, cudaMemcpyDeviceToHost, s));
    SEMO_CUDA(cudaStreamSynchronize(s));
    pcg_outcome(h2, body_nodes, info);
}

template <class V>
void fill_info(const Amg<V>& h, int64_t nnz, semo_solve_info* info) {
    info->levels = (int)h.lev.size();
    info->coarse_size = h.coarse_n;
    info->operator_complexity = (double)h.total_nnz / (double)std::max<int64_t>(nnz, 1);
}

// per-context apply state (kept for the adjoint solve on the same hierarchy)
struct ApplyState {
    Cycle<float> cy32;
    Cycle<double> cy64;
    OuterOp outer;
    // the SELL-32/16-bit structure of the context's mesh pattern (A_ptr, A_col)
    // and the mesh generation it was built for
    std::shared_ptr<Sell16Struct> pat16;
    int pat16_gen = 0;
    // the matrix values the current hierarchy was built from (pressure path only)
    DBuf<double> src_val;
    int src_n = 0;
    int64_t src_nnz = 0;
    int src_prec = -1;
    // the generation of the mesh's matrix (semo_ctx::matrix_gen) that the
    // hierarchy and outer were built from; -1: another matrix's
    int of_gen = -1;
};

// flag[0] = 1 if a and b differ anywhere (bit patterns)
__global__ void k_differs(int64_t n, const double* __restrict__ a, const double* __restrict__ b,
                          int* __restrict__ flag) {
    bool d = false;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        d |= __double_as_longlong(a[i]) != __double_as_longlong(b[i]);
    if (__any_sync(0xffffffffu, d) && (threadIdx.x & 31) == 0) flag[0] = 1;
}
ApplyState& apply_state(semo_ctx* c) {
    if (!c->apply) c->apply = std::shared_ptr<void>(new ApplyState(), [](void* p) { delete (ApplyState*)p; });
    return *(ApplyState*)c->apply.get();
}

template <class V>
void prepare_cycle(semo_ctx* c, Amg<V>& h, Cycle<V>& cy, const std::shared_ptr<Sell16Struct>& lev0 = nullptr) {
    cudaStream_t s = setup_stream(c);
    const int nl = (int)h.lev.size();
    cy.lev.resize(std::max(nl - 1, 0));
    cy.local_from = -1;
    if (c->prm.cheb_degree == 2)
        for (int l = 1; l + 1 < nl && cy.local_from < 0; ++l) {
            ClArgs<V> a;
            if (h.lev[l].A.nnz <= kLocalNnz && cl_args<V>(h, l, false, a, nullptr)) cy.local_from = l;
        }
    for (int l = 0; l + 1 < nl; ++l) {
        AmgLevel<V>& L = h.lev[l];
        LevelMats<V>& M = cy.lev[l];
        if (cy.local_from >= 0 && l >= cy.local_from) {   // CSR, all of them
            M.a = M.p = M.r = M.a16 = M.gs = false;
            continue;
        }
        M.a = sell_pays(L.A);
        M.p = sell_pays(L.P);
        M.r = sell_pays(L.R);
        int* const hp = c->hpin_int + 4;
        if (l == 0 && M.a && lev0 && lev0->n == L.A.n) {   // the mesh pattern's structure, shared
            fill_sell16<V, V>(s, L.A.ptr, L.A.val, lev0, M.A16);
            M.a16 = true;
        } else {
            M.a16 = M.a && build_sell16<V, V>(s, L.A.ptr, L.A.col, L.A.val, L.A.n, M.A16, hp,
                                                  l == 0 ? c->hpin_int + 14 : nullptr);
        }
        if (M.a16) M.a = false;
        if (M.a) build_sell<V, V>(s, L.A.ptr, L.A.col, L.A.val, L.A.n, M.A, hp);
        if (M.p) build_sell<V, V>(s, L.P.ptr, L.P.col, L.P.val, L.P.n, M.P, hp);
        if (M.r) build_sell<V, V>(s, L.R.ptr, L.R.col, L.R.val, L.R.n, M.R, hp);
        M.gs = false;
        if (c->prm.smoother == 1 && l == 0 && L.A.n > kGsMinRows) color_level(c, s, L.A, M);
    }
}

// ---------------------------------- momentum and VOF: batched BiCGStab
// NR right-hand sides (3 for the velocity components, 1 for the volume
// fraction) share one matrix: every kernel walks the rows once and serves all
// of them, so the operator is read once per product for the NR systems.  Right
// preconditioning by D^-1 (the momentum matrix is dominated by its BDF2 diagonal
// at the time steps of interest): the iteration solves B xh = b, B = A D^-1, and
// x = D^-1 xh at the end.  B's diagonal is 1 and is not stored: a product starts
// from the row's own value and adds the off-diagonal entries.
// What bounds the iteration is the FP64 unit (2 lanes a clock and
// multiprocessor): 69 instructions a row and iteration of three systems, and
// 600 bytes.  So D^-1 p and D^-1 s are never formed (the search directions
// themselves are gathered), and the scalars but beta are formed by the kernels
// that use them: six kernels an iteration, and one for the residual of the
// result.  Momentum solve at 75^3 cells 0.391 -> 0.277 ms, three right-hand sides
// of 67,080 caller's rows 0.60 -> 0.385.  rho is the sum (rh,r) itself: as
// (rh,s) - omega (rh,t), from the sums of the second product, it would save the
// kernel that forms p, 3 us of a solve at 75^3, but on implicit transport systems
// of 1,980 to 34,720 rows its error against extended precision was 3 to 40 times
// as large (rms 1.3e-15 against 1.3e-16 at 34,720).
// Per system j the scalars live at scal[16 j + k]:
//   0 rho, 1 alpha, 2 omega, 3 beta, 7 (r,r), 8 (b,b), 9 active, 10 breakdown,
//   11 iterations
constexpr int kMomScal = 16;
// Grid: at most 152 blocks (one a GB300 multiprocessor; not taken from the
// device, so that every sum's bits are the same on any GPU), because each block
// adds up the partial sums of all (12 sums: 1 us with 152 partials, 9 us with
// four blocks of 256 threads a multiprocessor, at 16 clocks an FP64 warp
// instruction; a kernel here needs 6).  Threads: what deals n out in equal sweeps.
constexpr int kBiBlocks = 152, kBiThreads = 512, kBiStream = 1024;
struct BiGrid { int blocks, threads; };
inline BiGrid bi_grid(int n, int most) {
    const int64_t sweeps = std::max<int64_t>(1, ((int64_t)n + kBiBlocks * most - 1) / (kBiBlocks * most));
    const int64_t per = ((int64_t)n + kBiBlocks * sweeps - 1) / (kBiBlocks * sweeps);
    const int t = (int)std::max<int64_t>(128, (per + 31) / 32 * 32);
    return BiGrid{(int)std::min<int64_t>(kBiBlocks, ((int64_t)n + t - 1) / t), t};
}

// The off-diagonal entries of B in slices of 32 rows, entry j of row 32 s + l at
// the slice's start + 32 j + l; padding entries point at the row with value 0.
// All slices W wide: every entry load, then every gather of a system.
template <int W>
struct OffEven {
    const int* __restrict__ col;
    const double* __restrict__ val;
    int n;
    template <int NR>
    __device__ __forceinline__ void mv(int row, unsigned act, const double* __restrict__ x, double* y) const {
        const int k = (row >> 5) * (32 * W) + (row & 31);
        int cj[W];
        double vj[W];
#pragma unroll
        for (int q = 0; q < W; ++q) { cj[q] = col[k + 32 * q]; vj[q] = val[k + 32 * q]; }
#pragma unroll
        for (int j = 0; j < NR; ++j) {
            if (!(act >> j & 1)) continue;
            const double* const xs = x + (size_t)j * n;
            double g[W];
#pragma unroll
            for (int q = 0; q < W; ++q) g[q] = __ldg(xs + cj[q]);
            y[j] = __ldg(xs + row);
#pragma unroll
            for (int q = 0; q < W; ++q) y[j] += vj[q] * g[q];
        }
    }
};
struct OffSell {
    const int* __restrict__ sptr;
    const int* __restrict__ col;
    const double* __restrict__ val;
    int n;
    template <int NR>
    __device__ __forceinline__ void mv(int row, unsigned act, const double* __restrict__ x, double* y) const {
        const int sl = row >> 5, b = sptr[sl] + (row & 31), w = (sptr[sl + 1] - sptr[sl]) >> 5;
#pragma unroll
        for (int j = 0; j < NR; ++j) y[j] = __ldg(x + (size_t)j * n + row);
        for (int e = 0, k = b; e < w; e += 4, k += 128) {   // four entries in flight
            int cj[4];
            double vj[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (e + q < w) { cj[q] = col[k + 32 * q]; vj[q] = val[k + 32 * q]; }
#pragma unroll
            for (int j = 0; j < NR; ++j) {
                if (!(act >> j & 1)) continue;
                double g[4];
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (e + q < w) g[q] = __ldg(x + (size_t)j * n + cj[q]);
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (e + q < w) y[j] += vj[q] * g[q];
            }
        }
    }
};
__global__ void k_off_width(int n, const int* __restrict__ ptr, int* __restrict__ slice_len, int* __restrict__ most) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    const int len = (row < n) ? ptr[row + 1] - ptr[row] - 1 : 0;
    const int w = __reduce_max_sync(0xffffffffu, len);
    if ((threadIdx.x & 31) == 0 && row < ((n + 31) & ~31)) {
        slice_len[row >> 5] = 32 * w;
        if (*most < w) atomicMax(most, w);
    }
}
// B's off-diagonal values (and, into a new layout, columns: scol not null).  width 0: slices as sptr says
__global__ void k_off_fill(int n, const int* __restrict__ ptr, const int* __restrict__ col,
                           const int* __restrict__ dig, const double* __restrict__ val,
                           const double* __restrict__ dinv, const int* __restrict__ sptr, int width,
                           int* __restrict__ scol, double* __restrict__ sval) {
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= ((n + 31) & ~31)) return;
    const int sl = row >> 5, l = row & 31;
    const int b = width ? 32 * width * sl : sptr[sl], w = width ? width : (sptr[sl + 1] - b) >> 5;
    const int rb = (row < n) ? ptr[row] : 0, len = (row < n) ? ptr[row + 1] - rb - 1 : 0;
    const int d = (row < n) ? dig[row] - rb : 0;   // the diagonal's place in the row
    for (int j = 0; j < w; ++j) {
        const int k = b + 32 * j + l;
        int c = min(row, n - 1);
        double v = 0.0;
        if (j < len) {
            const int e = rb + j + (j >= d);
            c = col[e];
            v = val[e] * dinv[c];
        }
        if (scol) scol[k] = c;
        sval[k] = v;
    }
}
struct OffDiag {
    int n = 0, nslices = 0, width = 0;
    DBuf<int> sptr, col;
    DBuf<double> val;
    // run f on the view that suits the layout
    template <class F>
    void with(F&& f) const {
        switch (width) {
            case 4: f(OffEven<4>{col.p, val.p, n}); break;
            case 5: f(OffEven<5>{col.p, val.p, n}); break;
            case 6: f(OffEven<6>{col.p, val.p, n}); break;
            default: f(OffSell{sptr.p, col.p, val.p, n});
        }
    }
};
// the layout of a pattern, without values and columns; hpin: two pinned ints.
// Slices are made equally wide where OffEven has that width (even_slots)
void build_offdiag(cudaStream_t s, const int* ptr, int n, OffDiag& S, int* hpin) {
    S.n = n;
    S.nslices = (n + 31) / 32;
    S.width = 0;
    S.sptr.alloc(S.nslices + 2, s);   // and the widest slice
    SEMO_CUDA(cudaMemsetAsync(S.sptr.p + S.nslices, 0, 2 * sizeof(int), s));
    k_off_width<<<blocks((int64_t)S.nslices * 32, 256), 256, 0, s>>>(n, ptr, S.sptr.p, S.sptr.p + S.nslices + 1);
    SEMO_CHECK_LAUNCH();
    SEMO_CUDA(cudaMemcpyAsync(hpin + 1, S.sptr.p + S.nslices + 1, sizeof(int), cudaMemcpyDeviceToHost, s));
    int total = device_scan(s, S.sptr.p, S.nslices + 1, hpin);   // its sync lands hpin[1] too
    if (const int64_t even = even_slots(hpin[1], 4, 6, S.nslices, total)) {
        S.width = hpin[1];
        total = (int)even;
    }
    S.col.alloc(std::max(total, 1), s);
    S.val.alloc(std::max(total, 1), s);
}

__device__ __forceinline__ unsigned bi_active(const double* scal, int nr) {
    // 0.0 or 1.0, told apart by the high word: a comparison is an FP64 instruction of every thread
    unsigned a = 0;
    for (int j = 0; j < nr; ++j)
        a |= (__double2hiint(scal[kMomScal * j + 9]) != 0 && __double2hiint(scal[kMomScal * j + 10]) == 0 ? 1u : 0u) << j;
    return a;
}
// part[k * kBiBlocks + block] = sum over the block of v[k], a warp a sum (sh: K * blockDim.x doubles)
template <int K>
__device__ __forceinline__ void bi_put(const double* v, double* sh, double* __restrict__ part) {
    __syncthreads();   // sh may still be read
#pragma unroll
    for (int k = 0; k < K; ++k) sh[k * blockDim.x + threadIdx.x] = v[k];
    __syncthreads();
    for (int k = threadIdx.x >> 5; k < K; k += blockDim.x >> 5) {
        const double* const a = sh + k * blockDim.x + (threadIdx.x & 31);
        double t = a[0];
        for (unsigned m = 32; m < blockDim.x; m += 32) t += a[m];
        t = warp_sum(t);
        if ((threadIdx.x & 31) == 0) part[k * kBiBlocks + blockIdx.x] = t;
    }
}
// tot[k] = sum of the nb partial sums k, k < K, in shared memory for the whole block
template <int K>
__device__ __forceinline__ void bi_get(const double* __restrict__ part, int nb, double* tot) {
    for (int k = threadIdx.x >> 5; k < K; k += blockDim.x >> 5) {
        const double t = parts_sum(part + k * kBiBlocks, nb);
        if ((threadIdx.x & 31) == 0) tot[k] = t;
    }
    __syncthreads();
}

// xh = 0, r = p = b, dinv;  part = (b,b) per system
template <int NR>
__global__ void __launch_bounds__(kBiStream) k_bi_init(int n, const int* __restrict__ dig,
                                                       const double* __restrict__ val, const double* __restrict__ b,
                                                       double* __restrict__ dinv, double* __restrict__ xh,
                                                       double* __restrict__ r, double* __restrict__ p,
                                                       double* __restrict__ part) {
    __shared__ double sh[NR * kBiStream];
    double bb[NR] = {};
    const size_t N = n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        dinv[i] = 1.0 / val[dig[i]];
#pragma unroll
        for (int j = 0; j < NR; ++j) {
            const double bi = b[j * N + i];
            xh[j * N + i] = 0.0; r[j * N + i] = bi; p[j * N + i] = bi;
            bb[j] += bi * bi;
        }
    }
    bi_put<NR>(bb, sh, part);
}
template <int NR>
__global__ void k_bi_fin0(const double* __restrict__ part, int nb, double* __restrict__ scal, double tol2) {
    __shared__ double tot[NR];
    bi_get<NR>(part, nb, tot);
    if (threadIdx.x < NR) {
        const double bb = tot[threadIdx.x];
        double* S = scal + kMomScal * threadIdx.x;
        for (int k = 0; k < kMomScal; ++k) S[k] = 0.0;
        S[0] = bb; S[1] = 1.0; S[2] = 1.0; S[7] = bb; S[8] = bb;
        S[9] = (bb > 0.0 && !(bb <= tol2 * bb)) ? 1.0 : 0.0;
    }
    if (threadIdx.x == 0) scal[3 * kMomScal] = 0.0;   // iterations of the loop
}
// v = B p;  part = (rh,v) per system
template <int NR, class M>
__global__ void __launch_bounds__(kBiThreads) k_bi_mv1(M B, const double* __restrict__ p, double* __restrict__ v,
                                                       const double* __restrict__ rh,
                                                       const double* __restrict__ scal, double* __restrict__ part) {
    pdl_enter();
    __shared__ double sh[NR * kBiThreads];
    const size_t N = B.n;
    const unsigned act = bi_active(scal, NR);
    double d[NR] = {};
    for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < B.n; row += gridDim.x * blockDim.x) {
        double y[NR];
        B.template mv<NR>(row, act, p, y);
#pragma unroll
        for (int j = 0; j < NR; ++j) {
            if (!(act >> j & 1)) continue;
            v[j * N + row] = y[j];
            d[j] += rh[j * N + row] * y[j];
        }
    }
    bi_put<NR>(d, sh, part);
}
// alpha = rho / (rh,v);  s = r - alpha v (in place in r).  One thread a system
// forms the scalars here and in k_bi_xr: the divisions in every thread took 5 us
// and more
template <int NR>
__global__ void __launch_bounds__(kBiStream) k_bi_s(int n, double* __restrict__ r, const double* __restrict__ v,
                                                    double* __restrict__ scal, const double* __restrict__ part,
                                                    int nb) {
    pdl_enter();
    __shared__ double tot[NR], sal[NR];
    __shared__ int go[NR];
    bi_get<NR>(part, nb, tot);
    if (threadIdx.x < NR) {
        double* const S = scal + kMomScal * threadIdx.x;   // no block reads what this kernel writes
        const double rv = tot[threadIdx.x], alpha = S[0] / rv;
        const bool act = S[9] != 0.0, bad = rv == 0.0 || !isfinite(rv);
        go[threadIdx.x] = act && !bad;
        sal[threadIdx.x] = alpha;
        if (blockIdx.x == 0 && act) {
            if (bad) S[10] = 1.0;
            else S[1] = alpha;
        }
    }
    __syncthreads();
    const size_t N = n;
#pragma unroll
    for (int j = 0; j < NR; ++j) {
        if (!go[j]) continue;
        const double alpha = sal[j];
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
            r[j * N + i] -= alpha * v[j * N + i];
    }
}
// t = B s;  part = (t,s), (t,t) per system
template <int NR, class M>
__global__ void __launch_bounds__(kBiThreads) k_bi_mv2(M B, const double* __restrict__ s, double* __restrict__ t,
                                                       const double* __restrict__ scal, double* __restrict__ part) {
    pdl_enter();
    __shared__ double sh[2 * NR * kBiThreads];
    const size_t N = B.n;
    const unsigned act = bi_active(scal, NR);
    double d[2 * NR] = {};
    for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < B.n; row += gridDim.x * blockDim.x) {
        double y[NR];
        B.template mv<NR>(row, act, s, y);
#pragma unroll
        for (int j = 0; j < NR; ++j) {
            if (!(act >> j & 1)) continue;
            t[j * N + row] = y[j];
            d[2 * j] += y[j] * s[j * N + row];
            d[2 * j + 1] += y[j] * y[j];
        }
    }
    bi_put<2 * NR>(d, sh, part);
}
// omega = (t,s) / (t,t);  xh += alpha p + omega s;  r = s - omega t;  part = (r,r),
// (rh,r) per system
template <int NR>
__global__ void __launch_bounds__(kBiStream) k_bi_xr(int n, double* __restrict__ xh, const double* __restrict__ p,
                                                     double* __restrict__ r, const double* __restrict__ t,
                                                     const double* __restrict__ rh, double* __restrict__ scal,
                                                     const double* __restrict__ parts, int nb,
                                                     double* __restrict__ part) {
    pdl_enter();
    __shared__ double sh[2 * kBiStream], tot[2 * NR], sal[NR], som[NR];
    bi_get<2 * NR>(parts, nb, tot);
    if (threadIdx.x < NR) {
        const int j = threadIdx.x;
        double* const S = scal + kMomScal * j;   // no block reads what this kernel writes
        const double tt = tot[2 * j + 1], omega = (tt > 0.0) ? tot[2 * j] / tt : 0.0;
        sal[j] = S[1];
        som[j] = omega;
        if (blockIdx.x == 0 && S[9] != 0.0 && S[10] == 0.0) S[2] = omega;
    }
    __syncthreads();
    const unsigned act = bi_active(scal, NR);
    const size_t N = n;
    double d[2 * NR] = {};
#pragma unroll
    for (int j = 0; j < NR; ++j) {
        if (!(act >> j & 1)) continue;
        const double alpha = sal[j], omega = som[j];
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
            const size_t k = j * N + i;
            const double si = r[k], hi = rh[k];
            xh[k] += alpha * p[k] + omega * si;
            const double ri = si - omega * t[k];
            r[k] = ri;
            d[2 * j] += ri * ri;
            d[2 * j + 1] += hi * ri;
        }
    }
#pragma unroll
    for (int j = 0; j < NR; ++j) bi_put<2>(d + 2 * j, sh, part + 2 * j * kBiBlocks);
}
// p = r + beta (p - omega v)
template <int NR>
__global__ void __launch_bounds__(kBiStream) k_bi_p(int n, double* __restrict__ p, const double* __restrict__ r,
                                                    const double* __restrict__ v, const double* __restrict__ scal) {
    pdl_enter();
    const unsigned act = bi_active(scal, NR);
    const size_t N = n;
#pragma unroll
    for (int j = 0; j < NR; ++j) {
        if (!(act >> j & 1)) continue;
        const double omega = scal[kMomScal * j + 2], beta = scal[kMomScal * j + 3];
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
            const size_t k = j * N + i;
            p[k] = r[k] + beta * (p[k] - omega * v[k]);
        }
    }
}
// The end of an iteration but for p: each system's state, the next rho and beta =
// (rho' / rho) (alpha / omega), and whether the loop goes on (a system is active
// and the cap is not reached; scal[3 * 16] counts iterations)
template <int NR>
__global__ void k_bi_check(cudaGraphConditionalHandle h, double* __restrict__ scal, const double* __restrict__ part,
                           int nb, double tol2, int max_iter) {
    pdl_enter();
    __shared__ double tot[2 * NR];
    bi_get<2 * NR>(part, nb, tot);
    bool any = false;
    if (threadIdx.x < NR) {
        double* S = scal + kMomScal * threadIdx.x;
        const double rr = tot[2 * threadIdx.x], rho = tot[2 * threadIdx.x + 1];
        if (S[9] == 0.0) {
        } else if (S[10] != 0.0) {
            S[9] = 0.0;                                         // (rh,v) was 0 or not finite
        } else {
            S[11] += 1.0;                                       // iterations of this system
            S[7] = rr;
            if (rr <= tol2 * S[8]) {
                S[9] = 0.0;                                     // converged
            } else if (rho == 0.0 || S[2] == 0.0 || !isfinite(rr)) {
                S[10] = 1.0; S[9] = 0.0;                        // breakdown
            } else {
                S[3] = (rho / S[0]) * (S[1] / S[2]);
                S[0] = rho;
                any = true;
            }
        }
    }
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) {
        double* const it = scal + 3 * kMomScal;
        const double done = it[0] + 1.0;
        it[0] = done;
        cudaGraphSetConditional(h, (any && done < (double)max_iter) ? 1u : 0u);
    }
}
// x = D^-1 xh (0 where no iteration was made)
template <int NR>
__global__ void k_bi_x(int n, const double* __restrict__ xh, const double* __restrict__ dinv,
                       const double* __restrict__ scal, double* __restrict__ x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t N = n;
    const double di = dinv[i];
#pragma unroll
    for (int j = 0; j < NR; ++j)
        x[j * N + i] = __double2hiint(scal[kMomScal * j + 11]) == 0 ? 0.0 : di * xh[j * N + i];
}
// part = (r,r) of r = b - A x per system, with the matrix itself (CSR, a thread
// a row, four entries in flight) and the x that is returned: the iteration's
// scaled values, whose residual takes part in no product with A, are not looked
// at (momentum pass at 75^3 cells 1.372 -> 1.384 ms)
template <int NR>
__global__ void __launch_bounds__(kBiStream) k_bi_res(int n, const int* __restrict__ ptr,
                                                      const int* __restrict__ col, const double* __restrict__ val,
                                                      const double* __restrict__ x, const double* __restrict__ b,
                                                      double* __restrict__ part) {
    __shared__ double sh[NR * kBiStream];
    const size_t N = n;
    double d[NR] = {};
    for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < n; row += gridDim.x * blockDim.x) {
        const int e1 = ptr[row + 1];
        double y[NR] = {};
        for (int e = ptr[row]; e < e1; e += 4) {
            int cj[4];
            double vj[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (e + q < e1) { cj[q] = col[e + q]; vj[q] = val[e + q]; }
#pragma unroll
            for (int j = 0; j < NR; ++j) {
                double g[4];
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (e + q < e1) g[q] = __ldg(x + j * N + cj[q]);
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (e + q < e1) y[j] += vj[q] * g[q];
            }
        }
#pragma unroll
        for (int j = 0; j < NR; ++j) {
            const double ri = b[j * N + row] - y[j];
            d[j] += ri * ri;
        }
    }
    bi_put<NR>(d, sh, part);
}
template <int NR>
__global__ void k_bi_fin_res(const double* __restrict__ part, int nb, double* __restrict__ out) {
    __shared__ double tot[NR];
    bi_get<NR>(part, nb, tot);
    if (threadIdx.x < NR) out[threadIdx.x] = tot[threadIdx.x];
}

// The instantiated iteration graph of a batched BiCGStab, kept while every
// pointer and scalar baked into its kernels stays the same (the buffers below
// are reused from call to call, so the momentum and volume-fraction solves of
// successive outer iterations launch it without capturing it again).
struct BiGraphKey {
    int nr = 0, n = 0, max_iter = 0, width = 0;
    double tol2 = 0.0;
    const void* ptrs[8] = {};
    bool operator==(const BiGraphKey& o) const {
        if (nr != o.nr || n != o.n || max_iter != o.max_iter || width != o.width || tol2 != o.tol2) return false;
        for (int k = 0; k < 8; ++k)
            if (ptrs[k] != o.ptrs[k]) return false;
        return true;
    }
};
struct BiGraph {
    BiGraphKey key;
    cudaGraph_t g = nullptr;
    cudaGraphExec_t e = nullptr;
    void reset() {
        if (e) cudaGraphExecDestroy(e);
        if (g) cudaGraphDestroy(g);
        e = nullptr;
        g = nullptr;
        key = BiGraphKey{};
    }
    BiGraph() = default;
    BiGraph(const BiGraph&) = delete;
    BiGraph& operator=(const BiGraph&) = delete;
    ~BiGraph() { reset(); }
};
struct MomState {
    OffDiag B;
    int gen = -1;                 // mesh generation the layout was built for
    DBuf<double> dinv, vec, part, scal;
    BiGraph graph[2];             // NR = 1, NR = 3
};

MomState& mom_state(semo_ctx* c) {
    if (!c->mom_apply) c->mom_apply = std::shared_ptr<void>(new MomState(), [](void* p) { delete (MomState*)p; });
    return *(MomState*)c->mom_apply.get();
}

}  // namespace

void pressure_setup(semo_ctx* c, const int* ptr, const int* col, const double* val, int n, int64_t nnz,
                    bool may_reuse, semo_solve_info* info) {
    cudaStream_t s = setup_stream(c);
    ApplyState& st = apply_state(c);
    c->sflag.alloc(16, s);
    SEMO_CUDA(cudaMemsetAsync(c->sflag.p, 0, 16 * sizeof(int), s));
    SEMO_CUDA(cudaEventRecord(c->setup_ev[0], s));
    const bool mesh_matrix = ptr == c->A_ptr.p && col == c->A_col.p && val == c->A_val.p;
    {
        StageScope sc(c, ST_AMG_SETUP);
        // The hierarchy is a deterministic function of the matrix: when the
        // values are bit-identical to the ones it was built from (the pressure
        // matrix depends only on geometry, dt and the densities, so it repeats
        // across the outer iterations of a time step), rebuilding would give
        // the same hierarchy bit for bit, and it is kept instead.
        bool reuse = false;
        const Amg<float>& h32 = c->amg32;
        const Amg<double>& h64 = c->amg64;
        const bool have = (c->prm.precision == SEMO_PREC_MIXED) ? h32.ready : h64.ready;
        if (may_reuse && c->prm.reuse_hierarchy && have && st.src_prec == c->prm.precision && st.src_n == n &&
            st.src_nnz == nnz) {
            k_differs<<<kRedBlocks, kRedThreads, 0, s>>>(nnz, val, st.src_val, c->sflag.p + 10);
            SEMO_CHECK_LAUNCH();
            int* const differs = c->hpin_int + 13;
            SEMO_CUDA(cudaMemcpyAsync(differs, c->sflag.p + 10, sizeof(int), cudaMemcpyDeviceToHost, s));
            SEMO_CUDA(cudaStreamSynchronize(s));
            reuse = *differs == 0;
        }
        st.of_gen = -1;
        if (!reuse) {
            if (c->prm.precision == SEMO_PREC_MIXED) {
                c->amg64.clear();
                build_hierarchy<float>(c, c->amg32, ptr, col, val, n, nnz);
            } else {
                c->amg32.clear();
                build_hierarchy<double>(c, c->amg64, ptr, col, val, n, nnz);
            }
            StageScope scy(c, ST_SETUP_CYCLE);
            // on the mesh's own pattern the layout structure is built once per mesh
            std::shared_ptr<Sell16Struct> pat;
            if (ptr == c->A_ptr.p && col == c->A_col.p) {
                if (!st.pat16 || st.pat16_gen != c->mesh_gen || st.pat16->n != n)
                    st.pat16 = build_sell16_struct(s, ptr, col, n, c->hpin_int + 4, c->hpin_int + 14);
                st.pat16_gen = c->mesh_gen;
                pat = st.pat16;
            } else {
                pat = build_sell16_struct(s, ptr, col, n, c->hpin_int + 4, c->hpin_int + 14);
            }
            if (c->prm.precision == SEMO_PREC_MIXED)
                prepare_cycle(c, c->amg32, st.cy32, pat);
            else
                prepare_cycle(c, c->amg64, st.cy64, pat);
            fill_sell16<double, double>(s, ptr, val, pat, st.outer.s16);
            st.src_prec = -1;
            if (may_reuse && c->prm.reuse_hierarchy) {
                st.src_val.alloc(nnz, s);
                SEMO_CUDA(cudaMemcpyAsync(st.src_val.p, val, sizeof(double) * nnz, cudaMemcpyDeviceToDevice, s));
                st.src_n = n;
                st.src_nnz = nnz;
                st.src_prec = c->prm.precision;
            }
        }
        if (mesh_matrix) st.of_gen = c->matrix_gen;
    }
    SEMO_CUDA(cudaEventRecord(c->setup_ev[1], s));   // setup_ms is read from setup_ev after the solve
    (void)info;
}

void solve_system(semo_ctx* c, const int* ptr, const int* col, const double* val, int n, int64_t nnz,
                  const double* b, double* x, semo_solve_info* info, bool zero_guess, bool may_reuse) {
    cudaStream_t s = c->stream;
    // with matrix_prebuilt the hierarchy is being built beside this thread's
    // work; before_solve joins that setup and makes this stream wait for it
    if (c->before_solve) {
        auto f = std::move(c->before_solve);
        c->before_solve = nullptr;
        f();
    }
    ApplyState& st = apply_state(c);
    c->flag.zero();
    if (!c->matrix_prebuilt) pressure_setup(c, ptr, col, val, n, nnz, may_reuse, info);
    SEMO_CUDA(cudaEventRecord(c->ev[2], s));
    {
        StageScope sc(c, ST_PCG);
        if (c->prm.precision == SEMO_PREC_MIXED) {
            pcg<float>(c, c->amg32, st.cy32, st.outer, true, ptr, col, val, n, b, x, zero_guess, info);
            fill_info(c->amg32, nnz, info);
        } else {
            pcg<double>(c, c->amg64, st.cy64, st.outer, true, ptr, col, val, n, b, x, zero_guess, info);
            fill_info(c->amg64, nnz, info);
        }
    }
    SEMO_CUDA(cudaEventRecord(c->ev[3], s));
    SEMO_CUDA(cudaEventSynchronize(c->ev[3]));
    float t0 = 0, t1 = 0;
    if (c->matrix_prebuilt) {
        t0 = (float)c->side_setup_ms;   // the setup shared the GPU with the momentum pass
    } else {
        SEMO_CUDA(cudaEventSynchronize(c->setup_ev[1]));
        SEMO_CUDA(cudaEventElapsedTime(&t0, c->setup_ev[0], c->setup_ev[1]));
    }
    SEMO_CUDA(cudaEventElapsedTime(&t1, c->ev[2], c->ev[3]));
    info->setup_ms = t0;
    info->solve_ms = t1;
}

namespace {

// The CSR pattern a batched BiCGStab solve runs on: the context's mesh
// pattern (gen = the mesh generation, so its SELL layout is kept across
// solves) or a caller's matrix (gen < 0: the layout is built for this solve).
struct KrylovPattern {
    int n;
    const int* ptr;
    const int* col;
    const int* dig;   // position of each row's diagonal
    int gen;
};
KrylovPattern mesh_pattern(semo_ctx* c) { return KrylovPattern{c->nc, c->A_ptr, c->A_col, c->A_dig, c->mesh_gen}; }

// Jacobi-preconditioned BiCGStab on NR right-hand sides (planes of b, x) of
// the matrix with values val on the pattern pat, from x = 0.
template <int NR>
semo_status bicgstab_jacobi(semo_ctx* c, int stage, const KrylovPattern& pat, const double* val, const double* b,
                            double* x, semo_solve_info* info) {
    StageScope scope(c, stage);
    cudaStream_t s = c->stream;
    const int n = pat.n;
    const size_t N = n;
    const BiGrid gm = bi_grid(n, kBiThreads), gs = bi_grid(n, kBiStream);
    MomState& st = mom_state(c);
    st.dinv.alloc(N, s);
    st.vec.alloc(5 * 3 * N, s);       // r, p, v, t, xh (room for 3 systems)
    st.part.alloc((size_t)(6 + 6) * kBiBlocks, s);
    st.scal.alloc(4 * kMomScal, s);
    double* r = st.vec.p;
    double* p = r + NR * N;
    double* v = p + NR * N;
    double* t = v + NR * N;
    double* xh = t + NR * N;
    double* const prr = st.part.p + 6 * kBiBlocks;
    // the recurrence residual is driven to half the tolerance so that the true
    // residual, checked at the end, lands under it
    const double tol2 = 0.25 * c->prm.mom_tol * c->prm.mom_tol;
    SEMO_CUDA(cudaEventRecord(c->ev[0], s));
    const bool fresh = pat.gen < 0 || st.gen != pat.gen;   // the mesh's layout is kept
    if (fresh) {
        st.gen = -1;
        build_offdiag(s, pat.ptr, n, st.B, c->hpin_scan);
    }
    k_bi_init<NR><<<gs.blocks, gs.threads, 0, s>>>(n, pat.dig, val, b, st.dinv, xh, r, p, st.part);
    SEMO_CHECK_LAUNCH();
    k_off_fill<<<blocks((int64_t)st.B.nslices * 32, 256), 256, 0, s>>>(n, pat.ptr, pat.col, pat.dig, val, st.dinv,
                                                                       st.B.sptr, st.B.width,
                                                                       fresh ? st.B.col.p : nullptr, st.B.val);
    SEMO_CHECK_LAUNCH();
    st.gen = pat.gen;
    SEMO_CUDA(cudaEventRecord(c->ev[1], s));
    k_bi_fin0<NR><<<1, 32 * NR, 0, s>>>(st.part, gs.blocks, st.scal, tol2);
    SEMO_CHECK_LAUNCH();
    // The iterations run as one graph: a conditional WHILE node around one
    // iteration (5 kernels and k_bi_check), launched without a host round trip
    // first: systems whose right-hand side is zero, already converged or not
    // finite start inactive (k_bi_fin0), every kernel skips them, and the
    // host reads the outcome once, after the true residuals.
    BiGraph& G = st.graph[NR == 1 ? 0 : 1];
    BiGraphKey key;
    key.nr = NR;
    key.n = n;
    key.max_iter = c->prm.mom_max_iter;
    key.tol2 = tol2;
    key.width = st.B.width;
    const void* kp[8] = {st.B.sptr.p, st.B.col.p, st.B.val.p, st.vec.p, st.part.p, st.scal.p, b, nullptr};
    std::copy(kp, kp + 8, key.ptrs);
    if (!G.e || !(G.key == key)) {
        G.reset();
        SEMO_CUDA(cudaGraphCreate(&G.g, 0));
        cudaGraphConditionalHandle handle;
        SEMO_CUDA(cudaGraphConditionalHandleCreate(&handle, G.g, 1, cudaGraphCondAssignDefault));
        cudaGraphNodeParams cp = {};
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = handle;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        cudaGraphNode_t loop;
        SEMO_CUDA(cudaGraphAddNode(&loop, G.g, nullptr, nullptr, 0, &cp));
        cudaGraph_t body = cp.conditional.phGraph_out[0];
        const long long before = __atomic_load_n(&g_kernel_launches, __ATOMIC_RELAXED);
        SEMO_CUDA(cudaStreamBeginCaptureToGraph(s, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
        try {
            st.B.with([&](auto B) {
                launch_pdl(k_bi_mv1<NR, decltype(B)>, gm.blocks, gm.threads, s, B, p, v, b, st.scal.p, st.part.p);
            });
            launch_pdl(k_bi_s<NR>, gs.blocks, gs.threads, s, n, r, v, st.scal.p, st.part.p, gm.blocks);
            st.B.with([&](auto B) {
                launch_pdl(k_bi_mv2<NR, decltype(B)>, gm.blocks, gm.threads, s, B, r, t, st.scal.p, st.part.p);
            });
            launch_pdl(k_bi_xr<NR>, gs.blocks, gs.threads, s, n, xh, p, r, t, b, st.scal.p, st.part.p, gm.blocks,
                       prr);
            launch_pdl(k_bi_check<NR>, 1, 32 * NR, s, handle, st.scal.p, prr, gs.blocks, tol2,
                       c->prm.mom_max_iter);
            launch_pdl(k_bi_p<NR>, gs.blocks, gs.threads, s, n, p, r, v, st.scal.p);
        } catch (...) {
            cudaGraph_t junk = nullptr;
            cudaStreamEndCapture(s, &junk);
            G.reset();
            throw;
        }
        cudaGraph_t captured = nullptr;
        SEMO_CUDA(cudaStreamEndCapture(s, &captured));
        __atomic_store_n(&g_kernel_launches, before, __ATOMIC_RELAXED);
        SEMO_CUDA(cudaGraphInstantiate(&G.e, G.g, 0));
        G.key = key;
    }
    SEMO_CUDA(cudaGraphLaunch(G.e, s));
    // the solutions, and their true FP64 residuals (in scal's last places of the third system)
    k_bi_x<NR><<<blocks(n, 256), 256, 0, s>>>(n, xh, st.dinv, st.scal, x);
    SEMO_CHECK_LAUNCH();
    k_bi_res<NR><<<gs.blocks, gs.threads, 0, s>>>(n, pat.ptr, pat.col, val, x, b, st.part);
    SEMO_CHECK_LAUNCH();
    k_bi_fin_res<NR><<<1, 32 * NR, 0, s>>>(st.part, gs.blocks, st.scal.p + 3 * kMomScal - 3);
    SEMO_CHECK_LAUNCH();
    // pinned: the systems' scalars, the residuals and the iteration count
    double* const hs = c->hpin;
    double* const tr = hs + 3 * kMomScal - 3;
    SEMO_CUDA(cudaMemcpyAsync(hs, st.scal.p, sizeof(double) * 4 * kMomScal, cudaMemcpyDeviceToHost, s));
    SEMO_CUDA(cudaEventRecord(c->ev[2], s));
    SEMO_CUDA(cudaEventSynchronize(c->ev[2]));
    const int it = (int)hs[3 * kMomScal];
    __atomic_add_fetch(&g_kernel_launches, 6LL * it, __ATOMIC_RELAXED);
    int iters[NR] = {};
    for (int j = 0; j < NR; ++j) {
        if (!std::isfinite(hs[kMomScal * j + 8])) throw Error(SEMO_ERR_NAN, "non-finite right-hand side");
        if (!std::isfinite(hs[kMomScal * j + 7])) throw Error(SEMO_ERR_NAN, "NaN/Inf in the BiCGStab residual");
        // systems converge one after another; each counts the iterations it was active
        iters[j] = (int)hs[kMomScal * j + 11];
    }
    float t0 = 0, t1 = 0;
    SEMO_CUDA(cudaEventElapsedTime(&t0, c->ev[0], c->ev[1]));
    SEMO_CUDA(cudaEventElapsedTime(&t1, c->ev[1], c->ev[2]));
    semo_status worst = SEMO_OK;
    for (int j = 0; j < NR; ++j) {
        const double bb = hs[kMomScal * j + 8];
        const double rel = (bb > 0.0) ? std::sqrt(tr[j] / bb) : 0.0;
        if (info) {
            info[j] = semo_solve_info{};
            info[j].iterations = iters[j];
            info[j].rel_residual = rel;
            info[j].levels = 1;
            info[j].coarse_size = n;
            info[j].operator_complexity = 1.0;
            info[j].setup_ms = t0;
            info[j].solve_ms = t1;
        }
        if (hs[kMomScal * j + 10] != 0.0 && !(rel <= c->prm.mom_tol)) worst = SEMO_ERR_BREAKDOWN;
        else if (!(rel <= c->prm.mom_tol) && worst == SEMO_OK) worst = SEMO_ERR_NOT_CONVERGED;
    }
    return worst;
}

}  // namespace

semo_status solve_momentum(semo_ctx* c, semo_solve_info* info) {
    c->xm.alloc(3 * (size_t)c->nc, c->stream);
    return bicgstab_jacobi<3>(c, ST_MSOLVE, mesh_pattern(c), c->Am_val, c->bm, c->xm, info);
}

semo_status solve_vof(semo_ctx* c, semo_solve_info* info) {
    c->xvf.alloc((size_t)c->nc, c->stream);
    return bicgstab_jacobi<1>(c, ST_VSOLVE, mesh_pattern(c), c->Av_val, c->bvf, c->xvf, info);
}

semo_status solve_csr_multi(semo_ctx* c, int n, const int* ptr, const int* col, const int* dig, const double* val,
                            int nrhs, const double* b, double* x, bool guess, semo_solve_info* info) {
    cudaStream_t s = c->stream;
    const size_t N = n;
    const KrylovPattern pat{n, ptr, col, dig, -1};
    // with an initial guess x0: solve A d = b - A x0 from d = 0, then x = x0 + d
    DBuf<double> rb, d;
    const double* rhs = b;
    double* sol = x;
    if (guess) {
        rb.alloc(N * nrhs, s);
        d.alloc(N * nrhs, s);
        const CsrView<double, 8> A8{ptr, col, val, n};
        for (int j = 0; j < nrhs; ++j) {
            k_res64<<<blocks((int64_t)n * 8, 256), 256, 0, s>>>(A8, x + j * N, b + j * N, rb.p + j * N);
            SEMO_CHECK_LAUNCH();
        }
        rhs = rb.p;
        sol = d.p;
    }
    semo_status worst = SEMO_OK;
    auto merge = [&](semo_status st) {
        if (st == SEMO_ERR_BREAKDOWN || (st != SEMO_OK && worst == SEMO_OK)) worst = st;
    };
    if (nrhs == 3) {
        merge(bicgstab_jacobi<3>(c, ST_MSOLVE, pat, val, rhs, sol, info));
    } else {
        for (int j = 0; j < nrhs; ++j)
            merge(bicgstab_jacobi<1>(c, ST_MSOLVE, pat, val, rhs + j * N, sol + j * N, info ? info + j : nullptr));
    }
    if (guess) {
        k_axpy1<double><<<blocks((int64_t)N * nrhs, 256), 256, 0, s>>>((int)(N * nrhs), d.p, x);
        SEMO_CHECK_LAUNCH();
    }
    SEMO_CUDA(cudaStreamSynchronize(s));
    return worst;
}

// Adjoint solve on the hierarchy of the last forward solve (the pressure
// matrix is symmetric, so A^T = A and the same preconditioner applies).  The
// matrix may have been assembled anew since, or the last solve a caller's
// system: one of another size is refused, and otherwise the residual is that of
// the assembled matrix, so that the solve of another one does not converge.
void solve_transpose_reuse(semo_ctx* c, const double* g, double* lam, semo_solve_info* info) {
    const int n = c->nc;
    ApplyState& st = apply_state(c);
    auto check = [&](const auto& h) {
        if (!h.ready) throw Error(SEMO_ERR_STATE, "no hierarchy: run a forward solve first");
        if (h.lev[0].A.n != n)
            throw Error(SEMO_ERR_STATE, "the last solve was of a system of another size: run a forward solve first");
    };
    if (c->prm.precision == SEMO_PREC_MIXED) check(c->amg32);
    else check(c->amg64);
    const bool same = st.of_gen == c->matrix_gen;
    SEMO_CUDA(cudaEventRecord(c->ev[1], c->stream));
    if (c->prm.precision == SEMO_PREC_MIXED) {
        pcg<float>(c, c->amg32, st.cy32, st.outer, same, c->A_ptr, c->A_col, c->A_val, n, g, lam, true, info);
        fill_info(c->amg32, c->nnz, info);
    } else {
        pcg<double>(c, c->amg64, st.cy64, st.outer, same, c->A_ptr, c->A_col, c->A_val, n, g, lam, true, info);
        fill_info(c->amg64, c->nnz, info);
    }
    SEMO_CUDA(cudaEventRecord(c->ev[2], c->stream));
    SEMO_CUDA(cudaEventSynchronize(c->ev[2]));
    float t1 = 0;
    SEMO_CUDA(cudaEventElapsedTime(&t1, c->ev[1], c->ev[2]));
    info->setup_ms = 0.0;
    info->solve_ms = t1;
}

// ---- measurement hooks on the last pressure hierarchy ----------------------
namespace {
template <class V>
Amg<V>& pressure_amg(semo_ctx* c);
template <> Amg<float>& pressure_amg<float>(semo_ctx* c) { return c->amg32; }
template <> Amg<double>& pressure_amg<double>(semo_ctx* c) { return c->amg64; }
template <class V>
Cycle<V>& pressure_cycle(ApplyState& st);
template <> Cycle<float>& pressure_cycle<float>(ApplyState& st) { return st.cy32; }
template <> Cycle<double>& pressure_cycle<double>(ApplyState& st) { return st.cy64; }

// reps launches of y = A x with A the finest level's operator in the layout
// the V-cycle uses (which = 0) or the FP64 outer operator (which = 1)
template <class V>
double time_spmv(semo_ctx* c, int which, int reps) {
    ApplyState& st = apply_state(c);
    Amg<V>& h = pressure_amg<V>(c);
    if (!h.ready || h.lev.empty()) throw Error(SEMO_ERR_STATE, "no pressure hierarchy: run a pressure solve first");
    cudaStream_t s = c->stream;
    const int n = h.lev[0].A.n;
    if (which == 0 && h.lev.size() < 2) throw Error(SEMO_ERR_STATE, "single-level hierarchy: no V-cycle operator");
    if (which == 1 && (c->kp.n < (size_t)n || c->kq.n < (size_t)n)) throw Error(SEMO_ERR_STATE, "no Krylov vectors");
    cudaEvent_t e0, e1;
    SEMO_CUDA(cudaEventCreate(&e0));
    SEMO_CUDA(cudaEventCreate(&e1));
    float ms = 0.f;
    try {
        SEMO_CUDA(cudaEventRecord(e0, s));
        for (int k = 0; k < reps; ++k) {
            if (which == 0) {
                AmgLevel<V>& L = h.lev[0];
                with_A(pressure_cycle<V>(st).lev[0], L.A,
                       [&](auto A) { k_mv<<<grid_for(A), 256, 0, s>>>(A, L.x.p, L.r.p, FirstIterate<V>{}); });
            } else {
                st.outer.with([&](auto A) { k_mv<<<grid_for(A), 256, 0, s>>>(A, c->kp.p, c->kq.p, FirstIterate<double>{}); });
            }
            SEMO_CHECK_LAUNCH();
        }
        SEMO_CUDA(cudaEventRecord(e1, s));
        SEMO_CUDA(cudaEventSynchronize(e1));
        SEMO_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    } catch (...) {
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        throw;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return ms / reps;
}

template <class V>
int levels_of(semo_ctx* c, int64_t* out, int max_levels) {
    ApplyState& st = apply_state(c);
    Amg<V>& h = pressure_amg<V>(c);
    if (!h.ready) throw Error(SEMO_ERR_STATE, "no pressure hierarchy: run a pressure solve first");
    const int nl = (int)h.lev.size();
    Cycle<V>& cy = pressure_cycle<V>(st);
    for (int l = 0; l < nl && l < max_levels; ++l) {
        const AmgLevel<V>& L = h.lev[l];
        int64_t* o = out + 6 * l;
        o[0] = L.A.n;
        o[1] = L.A.nnz;
        o[2] = L.P.nnz;
        o[3] = L.R.nnz;
        o[4] = (l + 1 < nl && l < (int)cy.lev.size()) ? (cy.lev[l].a16 ? 2 : (cy.lev[l].a ? 1 : 0)) : -1;
        o[5] = (int64_t)sizeof(V);
    }
    return nl;
}
}  // namespace

double time_pressure_spmv(semo_ctx* c, int which, int reps) {
    return c->prm.precision == SEMO_PREC_MIXED ? time_spmv<float>(c, which, reps) : time_spmv<double>(c, which, reps);
}

int pressure_levels(semo_ctx* c, int64_t* out, int max_levels) {
    return c->prm.precision == SEMO_PREC_MIXED ? levels_of<float>(c, out, max_levels)
                                               : levels_of<double>(c, out, max_levels);
}

// ---- AMG on the pressure equation of the coupled system (first stage of its
// two-stage preconditioner).  A hierarchy of its own, so the pressure
// equation's hierarchy is left as it is.
struct CprState {
    Amg<float> h32;
    Cycle<float> cy32;
    Amg<double> h64;
    Cycle<double> cy64;
};
CprState& cpr_state(semo_ctx* c) {
    if (!c->cpr) c->cpr = std::shared_ptr<void>(new CprState(), [](void* p) { delete (CprState*)p; });
    return *(CprState*)c->cpr.get();
}
template <class V> Amg<V>& cpr_h(CprState& S);
template <> Amg<float>& cpr_h<float>(CprState& S) { return S.h32; }
template <> Amg<double>& cpr_h<double>(CprState& S) { return S.h64; }
template <class V> Cycle<V>& cpr_cy(CprState& S);
template <> Cycle<float>& cpr_cy<float>(CprState& S) { return S.cy32; }
template <> Cycle<double>& cpr_cy<double>(CprState& S) { return S.cy64; }

template <class V>
void cpr_setup(semo_ctx* c, const int* ptr, const int* col, const double* val, int n, int64_t nnz) {
    CprState& S = cpr_state(c);
    build_hierarchy<V>(c, cpr_h<V>(S), ptr, col, val, n, nnz);
    prepare_cycle(c, cpr_h<V>(S), cpr_cy<V>(S));
}

// x = one V-cycle (zero start, both smoothing sweeps on every level) applied to b
template <class V>
V* cpr_rhs(semo_ctx* c) { return cpr_h<V>(cpr_state(c)).lev[0].b.p; }
template <class V>
const V* cpr_vcycle(semo_ctx* c) {
    CprState& S = cpr_state(c);
    Amg<V>& h = cpr_h<V>(S);
    Cycle<V>& cy = cpr_cy<V>(S);
    cudaStream_t s = c->stream;
    AmgLevel<V>& L = h.lev[0];
    vcycle_from(c, h, cy, 0);
    if (h.lev.size() > 1 && c->prm.cheb_degree == 2 && !cy.lev[0].gs) {
        // the last step vcycle_from leaves to the fused CG kernels on the finest level
        const ChebCoef cc = cheb2(L.lam_max);
        with_A(cy.lev[0], L.A, [&](auto A) {
            k_post1<<<grid_for(A), 256, 0, s>>>(A, L.dinv.p, L.b.p, (V)cc.c1, (V)cc.c2, L.r.p, L.t.p, L.x.p);
        });
        SEMO_CHECK_LAUNCH();
    }
    return L.x.p;
}
template void cpr_setup<float>(semo_ctx*, const int*, const int*, const double*, int, int64_t);
template void cpr_setup<double>(semo_ctx*, const int*, const int*, const double*, int, int64_t);
template float* cpr_rhs<float>(semo_ctx*);
template double* cpr_rhs<double>(semo_ctx*);
template const float* cpr_vcycle<float>(semo_ctx*);
template const double* cpr_vcycle<double>(semo_ctx*);

}  // namespace semo
