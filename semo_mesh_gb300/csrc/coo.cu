// A caller's COO triple to CSR on the device (semo_solve_coo, semo_solve_coo_multi).
//
// Replaces the COO -> CSR counting sort at the head of SEMO's solveAMGCL
// (src/solvers/solveAMGCL.cpp:206-251, :1129-1172): entries of a row keep
// their COO order.  The checks that go with it (indices in range, finite
// values, each row's diagonal, finite right-hand sides) run in the same
// kernels; the host waits once, and an error is the one a serial walk over
// the entries, then the rows, then the vectors would meet first.
//
// What bounds it: the copies of the caller's (pageable) arrays.  The serial
// host conversion this replaced took most of the call: 26.9 ms for a system
// of 115,056 rows and 795,936 entries and 21.3 ms for the three-right-hand-
// side solve of 67,080 rows, against 4.8 and 1.2 ms now (whole calls).
//
// An entry is first placed anywhere in its row (atomic counter), then every
// row is put in COO order: an entry's place is the number of its row's entries
// with a smaller COO index, counted by 8 lanes a row.  That is quadratic in
// the row length, so a system with a row of more than kCooMaxRow entries is
// converted on the host instead (one such row of 512 entries costs its lanes
// 32k comparisons, ~20 us; mesh systems have 7 to 30).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <string>
#include <vector>

#include "index.h"
#include "semo_internal.h"

namespace semo {
namespace {

constexpr int kCooMaxRow = 512;
constexpr int kCooLanes = 8;
inline int blocks(int64_t n, int t) { return (int)((n + t - 1) / t); }

// What the checks found: the smallest 2 k + kind of a bad entry (kind 0 index
// out of range, 1 value not finite), the same for a bad row (0 no diagonal
// entry, 1 zero diagonal), the longest row, and the vectors' flags (bit 0 a
// value that is not finite, bit 1 a guess that is not zero).
struct CooFound {
    unsigned long long entry, row;
    int longest, vec;
};

__global__ void k_coo_init(CooFound* f) {
    f->entry = f->row = ~0ull;
    f->longest = f->vec = 0;
}

__global__ void k_coo_count(int64_t nnz, int n, const int* __restrict__ rows, const int* __restrict__ cols,
                            const double* __restrict__ vals, int* __restrict__ cnt, CooFound* __restrict__ f) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nnz) return;
    const int r = rows[k], c = cols[k];
    if (r < 0 || r >= n || c < 0 || c >= n) {
        atomicMin(&f->entry, 2ull * (unsigned long long)k);
        return;
    }
    if (!isfinite(vals[k])) atomicMin(&f->entry, 2ull * (unsigned long long)k + 1ull);
    atomicAdd(cnt + r, 1);
}

__global__ void k_coo_longest(int n, const int* __restrict__ cnt, CooFound* __restrict__ f) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int m = __reduce_max_sync(0xffffffffu, i < n ? cnt[i] : 0);
    if ((threadIdx.x & 31) == 0) atomicMax(&f->longest, m);
}

// ord[p]: COO index of the entry at place p (a row's entries in any order);
// entries out of range are left out, as the count left them out
__global__ void k_coo_place(int64_t nnz, int n, const int* __restrict__ rows, const int* __restrict__ cols,
                            int* __restrict__ fill, int* __restrict__ ord) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nnz) return;
    const int r = rows[k], c = cols[k];
    if (r < 0 || r >= n || c < 0 || c >= n) return;
    ord[atomicAdd(fill + r, 1)] = (int)k;
}

// rows into COO order; dig (if given): place of each row's first diagonal entry
__global__ void k_coo_rows(int n, const int* __restrict__ ptr, const int* __restrict__ ord,
                           const int* __restrict__ cols, const double* __restrict__ vals, int* __restrict__ col,
                           double* __restrict__ val, int* __restrict__ dig, CooFound* __restrict__ f) {
    if (f->longest > kCooMaxRow) return;   // the host converts it
    const int64_t row = row_of(blockIdx.x, blockDim.x, threadIdx.x, kCooLanes);
    const bool live = row < n;
    const int i = live ? (int)row : 0, lane = threadIdx.x % kCooLanes;
    const int rb = live ? ptr[i] : 0, re = live ? ptr[i + 1] : 0;
    int first = INT_MAX;
    for (int e = rb + lane; e < re; e += kCooLanes) {
        const int k = ord[e];
        int rank = 0;
        for (int u = rb; u < re; ++u) rank += ord[u] < k;
        const int c = cols[k];
        col[rb + rank] = c;
        val[rb + rank] = vals[k];
        if (c == i) first = min(first, rb + rank);
    }
    if (!dig) return;
#pragma unroll
    for (int o = kCooLanes / 2; o > 0; o >>= 1) first = min(first, __shfl_xor_sync(0xffffffffu, first, o, kCooLanes));
    if (!live || lane != 0) return;
    if (first == INT_MAX) {
        atomicMin(&f->row, 2ull * (unsigned long long)i);
        first = rb;
    }
    dig[i] = first;
}

// after k_coo_rows has written every value
__global__ void k_coo_diagonal(int n, const int* __restrict__ ptr, const int* __restrict__ dig,
                               const double* __restrict__ val, CooFound* __restrict__ f) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || f->longest > kCooMaxRow || ptr[i] == ptr[i + 1]) return;
    if (val[dig[i]] == 0.0) atomicMin(&f->row, 2ull * (unsigned long long)i + 1ull);
}

__global__ void k_coo_vectors(int64_t n, const double* __restrict__ b, const double* __restrict__ x,
                              CooFound* __restrict__ f) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int v = 0;
    if (i < n) v = ((isfinite(b[i]) && isfinite(x[i])) ? 0 : 1) | (x[i] != 0.0 ? 2 : 0);
    v = __reduce_or_sync(0xffffffffu, v);
    if (v && (threadIdx.x & 31) == 0) atomicOr(&f->vec, v);
}

// the same conversion on the host, for systems with very long rows
void coo_on_host(semo_ctx* c, int n, int64_t nnz, const int32_t* rows, const int32_t* cols, const double* vals,
                 bool want_dig, CooSystem& S, CooFound& f) {
    std::vector<int> ptr(n + 1, 0), col(nnz), dig(want_dig ? n : 0, -1);
    std::vector<double> val(nnz);
    for (int64_t k = 0; k < nnz; ++k) ptr[rows[k]]++;
    for (int i = 0, t = 0; i < n; ++i) { const int u = ptr[i]; ptr[i] = t; t += u; }
    ptr[n] = (int)nnz;
    for (int64_t k = 0; k < nnz; ++k) {
        const int d = ptr[rows[k]]++;
        col[d] = cols[k];
        val[d] = vals[k];
        if (want_dig && cols[k] == rows[k] && dig[rows[k]] < 0) dig[rows[k]] = d;
    }
    for (int i = 0, last = 0; i <= n; ++i) { const int t = ptr[i]; ptr[i] = last; last = t; }
    if (want_dig)
        for (int i = 0; i < n && f.row == ~0ull; ++i) {
            if (dig[i] < 0) f.row = 2ull * (unsigned long long)i;
            else if (val[dig[i]] == 0.0) f.row = 2ull * (unsigned long long)i + 1ull;
        }
    cudaStream_t s = c->stream;
    S.ptr.upload(ptr.data(), n + 1, s);
    S.col.upload(col.data(), nnz, s);
    S.val.upload(val.data(), nnz, s);
    if (want_dig) S.dig.upload(dig.data(), n, s);
    SEMO_CUDA(cudaStreamSynchronize(s));   // the host vectors are freed on return
}

}  // namespace

bool coo_system(semo_ctx* c, int n, int64_t nnz, const int32_t* rows, const int32_t* cols, const double* vals,
                int nrhs, const double* b, const double* x, bool want_dig, CooSystem& S) {
    cudaStream_t s = c->stream;
    const int64_t nv = (int64_t)nrhs * n;
    DBuf<int> dr, dc, fill, ord;
    DBuf<double> dv;
    DBuf<CooFound> found;
    found.alloc(1, s);
    k_coo_init<<<1, 1, 0, s>>>(found.p);
    SEMO_CHECK_LAUNCH();
    dr.upload(rows, nnz, s);
    dc.upload(cols, nnz, s);
    dv.upload(vals, nnz, s);
    S.ptr.alloc(n + 1, s);
    S.ptr.zero();
    k_coo_count<<<blocks(nnz, 256), 256, 0, s>>>(nnz, n, dr, dc, dv, S.ptr, found.p);
    SEMO_CHECK_LAUNCH();
    k_coo_longest<<<blocks(n, 256), 256, 0, s>>>(n, S.ptr, found.p);
    SEMO_CHECK_LAUNCH();
    device_scan_async(s, S.ptr.p, n + 1);
    fill.alloc(n + 1, s);
    SEMO_CUDA(cudaMemcpyAsync(fill.p, S.ptr.p, sizeof(int) * (n + 1), cudaMemcpyDeviceToDevice, s));
    ord.alloc(nnz, s);
    k_coo_place<<<blocks(nnz, 256), 256, 0, s>>>(nnz, n, dr, dc, fill, ord);
    SEMO_CHECK_LAUNCH();
    S.col.alloc(nnz, s);
    S.val.alloc(nnz, s);
    if (want_dig) S.dig.alloc(n, s);
    k_coo_rows<<<blocks((int64_t)n * kCooLanes, 256), 256, 0, s>>>(n, S.ptr, ord, dc, dv, S.col, S.val,
                                                                  want_dig ? S.dig.p : nullptr, found.p);
    SEMO_CHECK_LAUNCH();
    if (want_dig) {
        k_coo_diagonal<<<blocks(n, 256), 256, 0, s>>>(n, S.ptr, S.dig, S.val, found.p);
        SEMO_CHECK_LAUNCH();
    }
    S.b.upload(b, nv, s);
    S.x.upload(x, nv, s);
    k_coo_vectors<<<blocks(nv, 256), 256, 0, s>>>(nv, S.b, S.x, found.p);
    SEMO_CHECK_LAUNCH();
    static_assert(sizeof(CooFound) <= kHostScalars * sizeof(double), "pinned scalars");
    CooFound& f = *reinterpret_cast<CooFound*>(c->hpin);
    SEMO_CUDA(cudaMemcpyAsync(&f, found.p, sizeof(CooFound), cudaMemcpyDeviceToHost, s));
    SEMO_CUDA(cudaStreamSynchronize(s));
    if (f.entry != ~0ull) {
        if (f.entry & 1ull) throw Error(SEMO_ERR_NAN, "non-finite matrix value");
        throw Error(SEMO_ERR_ARGUMENT, "COO index out of range");
    }
    if (f.longest > kCooMaxRow) coo_on_host(c, n, nnz, rows, cols, vals, want_dig, S, f);
    if (f.row != ~0ull)
        throw Error(SEMO_ERR_ARGUMENT, "row " + std::to_string(f.row >> 1) +
                                           ((f.row & 1ull) ? " has a zero diagonal" : " has no diagonal entry"));
    if (f.vec & 1) throw Error(SEMO_ERR_NAN, "non-finite rhs/guess");
    return (f.vec & 2) != 0;
}

}  // namespace semo
