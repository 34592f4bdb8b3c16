// Smoothed-aggregation setup of small levels in one cooperative kernel.
//
// amg_setup.cu builds a level with ~60 launches and six host waits, which is
// what a small level costs: a level of 3,053 rows takes as long as one of
// 30,000.  Here one kernel builds every level from a small one down to the
// coarsest: the steps are those of amg_setup.cu (strength, MIS(2), joining,
// prolongation, its transpose, A P, R (A P)), each a loop of the whole grid,
// with a grid barrier where a step reads what other blocks wrote (14 and two
// a MIS round; ~1.3 us each with a block on every multiprocessor), and the
// sizes of the next level never leave the device.  The host waits once, for
// the records of all levels.
//
// What bounds it: the barriers and the latency of the dependent loads between
// them; the levels it takes fit in L2 (ncu: of a warp's clocks between two issues
// 15 to 29 are spent at a barrier and 5 on a load; 26 % of the issue slots of a
// 64^3 box used, 9 % of a 32^3 box).
//   setup of a 32^3 box (32,768 rows and below)    2.60 -> 0.78 ms
//   setup of a 14^3 box (2,744 rows and below)     1.42 -> 0.45 ms
// Above kSmallRows rows or kSmallNnz entries the level-by-level kernels, which
// fill the multiprocessors, are as fast: with the second level of a 128^3 box
// (188,670 rows, 6.3M entries) taken too, an outer iteration was 23.5 ms
// against 22.1; with the finest level of a 64^3 box (262,144 rows, 1.8M
// entries) the gradient call was 7.33 ms against 7.57.  Beside the momentum
// pass the line is lower, since a block here keeps a multiprocessor to
// itself: with the finest level of a 47^3 box (103,823 rows) a time step was
// 5.32 ms against 4.90, with the second level of an 80^3 box (46,686 rows,
// 1.5M entries) 9.3 against 10.3.  The two ways differ by rounding, and a
// hierarchy of the mesh's pressure matrix may be built beside the momentum pass
// in one call, alone in the next, or kept from either, with the same result, so
// that matrix takes the lower line always (a setup alone 1.4 instead of 1.0 ms at
// 48^3, 1.8 instead of 1.4 at 64^3); the higher one is for the systems that
// are never set up beside others (a caller's, the coupled system's pressure
// stage).  For the first reason a block takes
// kNnzPerBlock entries or more: 72 blocks instead of 152 at 32^3 made the
// outer iteration 2.33 ms instead of 2.65.
//
// Sums are in a fixed order (lane-strided partial sums and shuffle trees for
// a row's FP64 sums, exact integers in the products), so the hierarchy is the
// same bits run to run; a row's sums differ from amg_setup.cu's by rounding.
//
// Every wait is bounded: a barrier that is not reached within kSpinLimit polls
// sets an error flag and the kernel ends.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <string>
#include <utility>

#include "amg_rows.cuh"
#include "semo_internal.h"

namespace semo {
namespace {

using namespace semo::amg;

constexpr int kT = 1024, kWarps = kT / 32;
constexpr int kSlots = 128;        // table slots of a warp
constexpr int kBigSlots = kWarps * kSlots;   // of the rows that the whole block sums
constexpr int kTableBytes = kWarps * kSlots * kTableSlotBytes;
constexpr int kListed = kSlots * kTableSlotBytes / 32 / 12;   // places a thread in prolongation rows
constexpr int kBlockProducts = 768;   // products from which the whole block sums a row
// the largest levels taken (see above): of a system that is set up alone, and of
// the mesh's pressure matrix
constexpr int kSmallRows = 262144, kBesideRows = 65536;
constexpr int64_t kSmallNnz = 2000000, kBesideNnz = 1700000;
constexpr int kMostBlocks = 152, kNnzPerBlock = 3072;
constexpr int kMaxBlocks = 256, kMaxLevels = 64, kMaxRounds = 200, kRoundSlots = 1024;
// Scratch that may stay with a hierarchy: what a finished arena holds beyond it is
// given back by a copy of the levels (an arena has 56 MB at 64,000 rows of 7
// entries; the calls on such systems take as long as before)
constexpr long long kSpareBytes = 16ll << 20;
constexpr int kGjMax = 64;         // rows of the largest coarsest level inverted by k_small_inverse
constexpr unsigned kSpinLimit = 1u << 23;
// Levels this small are built by one block: its barrier costs some 30 ns
// where the grid's costs 2 us, and what it wrote is in its own L1.
constexpr int kSoloRows = 64, kSoloNnz = 1024;

struct SmallRec {
    int n, nnz, nagg, nnzP;
    int runA, runP, runR;     // entries of the longest cluster run of rows
    long long dinv, Pptr, Pcol, Pval, Rptr, Rcol, Rval, Aptr, Acol, Aval;   // arena offsets (bytes)
    unsigned long long lam;   // bits of the Gershgorin bound
};
enum SmallStatus { SMALL_OK = 0, SMALL_NO_ROOM = 1, SMALL_NO_MIS = 2, SMALL_LONG_ROW = 3 };
struct SmallCtl {
    int status, nlev, zero_diag, non_finite, singular, abort;
    long long cinv, kept;   // kept: bytes of the arena that the hierarchy needs
    SmallRec lev[kMaxLevels];
    // below: not read by the host
    unsigned arrived;
    unsigned long long bump[kMaxLevels];
    int undecided[kRoundSlots];
    int part[kMaxBlocks];
};

template <class V>
struct SmallArgs {
    const int *ptr, *col;
    const V* val;
    int n, nnz;
    float eps;
    int coarse_enough, max_levels;
    double omega;
    unsigned char* arena;
    long long cap;
    int* scol;             // row slots of the products
    V* sval;
    long long slots;
    SmallCtl* ctl;
};

// All blocks of the (cooperative) grid; false when a wait ran out, here or
// in another block, and the kernel has to end.
__device__ bool grid_sync(SmallCtl* ctl, int blocks, unsigned& epoch, int* ok) {
    __syncthreads();
    if (blocks == 1) return true;   // one block left
    epoch += blocks;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&ctl->arrived, 1u);
        int good = 1;
        for (unsigned spins = 0;; ++spins) {
            unsigned got;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(got) : "l"(&ctl->arrived) : "memory");
            if (got >= epoch) break;
            if (spins >= kSpinLimit || ((spins & 63u) == 63u && *(volatile int*)&ctl->abort)) {
                atomicExch(&ctl->abort, 1);
                good = 0;
                break;
            }
        }
        *ok = good;   // the acquire and the barrier below order what follows
    }
    __syncthreads();
    return *ok != 0;
}

// exclusive sum over the block; *total gets the sum (both for every thread)
__device__ int block_scan(int v, int* sh, int* total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    __syncthreads();
    if (lane == 31) sh[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        int w = lane < kWarps ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        if (lane < kWarps) sh[lane] = w;
    }
    __syncthreads();
    *total = sh[kWarps - 1];
    return incl - v + (wid ? sh[wid - 1] : 0);
}
// sum of the blocks' parts before this one's; *total: of all
__device__ int parts_before(const SmallCtl* ctl, int G, int* sh, int* total) {
    const int me = blockIdx.x;
    const int t = threadIdx.x;
    const int v = t < G ? ctl->part[t] : 0;   // at most kMaxBlocks <= kT blocks
    int all;
    block_scan(t < me ? v : 0, sh, &all);
    const int before = all;
    block_scan(v, sh, total);
    return before;
}
static_assert(kWarps == 32 && kBigSlots == 4096, "hash_row_block");
static_assert(kMaxBlocks <= kT, "parts_before reads a part a thread");

template <class T>
__device__ __forceinline__ T group_sum(T v, int vs) {
    for (int o = vs >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ unsigned long long group_max(unsigned long long v, int vs) {
    for (int o = vs >> 1; o > 0; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, v, o);
        v = t > v ? t : v;
    }
    return v;
}

// lanes a row: the row length's power of two, while the grid has lanes to spare
__device__ __forceinline__ int lanes_for(int n, int nnz, int threads) {
    int vs = 1;
    while (vs < 32 && (long long)vs * n < nnz && 2ll * vs * n <= 2ll * threads) vs <<= 1;
    return vs;
}

// sum of |values| of a row, by a warp
template <class V>
__device__ Mag row_size(const V* v, int m, int lane) {
    Mag s{0.0f, kMagNone};
    for (int e = lane; e < m; e += 32) mag_add(s, mag_of(v[e]));
    return mag_warp_sum(s);
}

// One row of C = A B summed by the whole block in one table of kBigSlots (the
// sums are exact integers, so it gives hash_row's bits): the row's A entries
// go round the warps.  Returns its length, or -1 when more than 3/4 of the
// table is taken (every thread); *size gets the sum of |values|.
template <class V>
__device__ int hash_row_block(RowTable tb, Mag* shm, int* cnt2, int ab, int ae, const int* acol, const V* aval,
                              RowSpan rb, const int* bcol, const V* bval, const Mag* bmag, int* ocol, V* oval,
                              Mag* size) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int t = threadIdx.x; t < kBigSlots; t += kT) { tb.keys[t] = -1; tb.vals[t] = 0ull; }
    Mag bound{0.0f, kMagNone};
    for (int ka = ab + threadIdx.x; ka < ae; ka += kT) mag_add(bound, mag_mul(mag_of(aval[ka]), bmag[acol[ka]]));
    bound = mag_warp_sum(bound);
    if (lane == 0) shm[wid] = bound;
    if (threadIdx.x < 2) cnt2[threadIdx.x] = 0;
    __syncthreads();
    const int sc = mag_scale(mag_warp_sum(shm[lane]));   // kWarps == 32: the same tree in every warp
    for (int k = ab + wid; k < ae; k += kWarps) {
        const int a = acol[k], b0 = rb.begin(a), b1 = b0 + rb.count(a);
        const V av = aval[k];
        for (int q = b0 + lane; q < b1; q += 32) {
            const int c = bcol[q];
            uint32_t h = hash_u32((uint32_t)c) & (kBigSlots - 1);
            for (int probe = 0; probe < kBigSlots; ++probe) {   // a full table ends the probing
                const int prev = atomicCAS(tb.keys + h, -1, c);
                if (prev == -1) atomicAdd(cnt2, 1);
                if (prev == -1 || prev == c) {
                    shared_add64(tb.vals + h, (unsigned long long)fixed_product(av, bval[q], sc));
                    break;
                }
                h = (h + 1) & (kBigSlots - 1);
            }
            if (*(volatile int*)cnt2 > kBigSlots * 3 / 4) break;
        }
    }
    __syncthreads();
    const int m = cnt2[0];
    if (m > kBigSlots * 3 / 4) return -1;
    for (int t = threadIdx.x; t < kBigSlots; t += kT)
        if (tb.keys[t] >= 0) {   // in any order: the ranks below sort them
            const int pos = atomicAdd(cnt2 + 1, 1);
            tb.ckeys[pos] = tb.keys[t];
            tb.cvals[pos] = tb.vals[t];
        }
    __syncthreads();
    for (int x = threadIdx.x; x < m; x += kT) {
        const int ce = tb.ckeys[x];
        int rank = 0;
        for (int u = 0; u < m; ++u) rank += tb.ckeys[u] < ce;
        ocol[rank] = ce;
        oval[rank] = fixed_value((long long)tb.cvals[x], sc, V(0));
    }
    __syncthreads();
    if (size && wid == 0) {   // in column order, as a warp's row
        const Mag t = row_size(oval, m, lane);
        if (lane == 0) *size = t;
    }
    __syncthreads();
    return m;
}

// Products of rows [c0, c1) of A B into slots taken from this level's bump
// counter: start[i], cnt[i], size[i] (sum of |values|) per
// row.  A warp sums a row; rows of many products, and rows that fill a warp's
// table, are summed by the whole block afterwards.  Sets ctl->status when
// there is no room or a row is too long.
template <class V>
__device__ void block_product(const SmallArgs<V>& a, int level, int c0, int c1, const int* aptr, const int* acol,
                              const V* aval, RowSpan rb, const int* bcol, const V* bval, const Mag* bmag,
                              int* start, int* cnt, Mag* size, int* later, unsigned char* sm, int* sh, Mag* shm,
                              int* nlater, long long* base) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    SmallCtl* ctl = a.ctl;
    // slots: the rows' product counts, a warp a row, then scanned over the
    // chunk.  A count stops at kMostProducts, so that a tile's sum fits an int;
    // a chunk with such a row has no room.
    constexpr int kMostProducts = 1 << 21;
    bool many = false;
    // short rows (a mesh's): 8 lanes a row, here and in the sums.  Up to 8 entries
    // a row one step of the lanes holds a row; longer ones fill a warp by themselves
    const bool brief = c1 > c0 && (long long)aptr[c1] - aptr[c0] <= (long long)kGroup * (c1 - c0);
    const int vs = brief ? kGroup : 32, rpw = 32 / vs, sub = lane & (vs - 1);
    for (int r0 = c0 + wid * rpw; r0 < c1; r0 += kWarps * rpw) {
        const int i = r0 + lane / vs;
        long long p = 0;
        if (i < c1)
            for (int k = aptr[i] + sub; k < aptr[i + 1]; k += vs) p += rb.count(acol[k]);
        p = group_sum(p, vs);
        many |= p >= kMostProducts;
        if (i < c1 && sub == 0) cnt[i] = (int)min(p, (long long)kMostProducts);
    }
    __syncthreads();
    long long chunk = 0;
    for (int r0 = c0; r0 < c1; r0 += kT) {
        const int i = r0 + threadIdx.x;
        int total;
        const int off = block_scan(i < c1 ? cnt[i] : 0, sh, &total);
        if (i < c1) start[i] = (int)min(chunk + off, 0x7fffffffll);
        chunk += total;
    }
    many = __syncthreads_or(many);
    if (threadIdx.x == 0) {
        *nlater = 0;
        *base = -1;
        if (!many && chunk <= a.slots) {
            const long long at = (long long)atomicAdd(&ctl->bump[level], (unsigned long long)chunk);
            if (at + chunk <= a.slots && at + chunk <= 0x7fffffffll) *base = at;
        }
        if (*base < 0) atomicExch(&ctl->status, SMALL_NO_ROOM);
    }
    __syncthreads();
    if (*base < 0) return;
    const int b0 = (int)*base;
    RowTable tb;
    tb.keys = reinterpret_cast<int*>(sm + (size_t)wid * kSlots * kTableSlotBytes);
    tb.ckeys = tb.keys + kSlots;
    tb.vals = reinterpret_cast<unsigned long long*>(tb.ckeys + kSlots);
    tb.cvals = tb.vals + kSlots;
    // rows from which the block does better together: few rows leave most warps idle
    const int alone = c1 - c0 >= kWarps / 4 ? kBlockProducts : 128;
    RowTable tg = tb;   // the lane's group's part
    tg.keys += (lane / kGroup) * kGroupSlots;
    tg.ckeys += (lane / kGroup) * kGroupSlots;
    tg.vals += (lane / kGroup) * kGroupSlots;
    tg.cvals += (lane / kGroup) * kGroupSlots;
    for (int r0 = c0 + wid * rpw; r0 < c1; r0 += kWarps * rpw) {
        unsigned wide = 1u;   // rows from r0 on that the whole warp sums
        if (brief) {
            const int i = r0 + lane / kGroup;
            const bool mine = i < c1;
            const int s = mine ? b0 + start[i] : 0, ab = mine ? aptr[i] : 0, ae = mine ? aptr[i + 1] : 0;
            __syncwarp();   // every lane has read the row's places before they are written
            Mag t;
            const int m = hash_rows_short<V>(lane, tg, ab, ae, acol, aval, rb, bcol, bval, bmag, a.scol + s,
                                             a.sval + s, &t);
            if (mine && sub == 0 && m >= 0) {
                start[i] = s;
                cnt[i] = m;
                if (size) size[i] = t;
            }
            const unsigned failed = __ballot_sync(0xffffffffu, m < 0);
            wide = (failed & 1u) | (failed >> 8 & 1u) << 1 | (failed >> 16 & 1u) << 2 | (failed >> 24 & 1u) << 3;
        }
        for (; wide; wide &= wide - 1) {
            const int i = r0 + __ffs(wide) - 1;
            const int s = b0 + start[i], most = cnt[i];
            __syncwarp();   // every lane has read the row's places before lane 0 writes them
            const int m = most > alone ? -1
                                       : hash_row<V>(lane, table_size(most, kSlots), tb, aptr[i], aptr[i + 1], acol,
                                                     aval, rb, bcol, bval, bmag, a.scol + s, a.sval + s);
            if (m < 0) {
                if (lane == 0) later[c0 + atomicAdd(nlater, 1)] = i;
                continue;
            }
            Mag t{0.0f, kMagNone};
            if (size) {
                __syncwarp();
                t = row_size(a.sval + s, m, lane);
            }
            if (lane == 0) { start[i] = s; cnt[i] = m; if (size) size[i] = t; }
        }
    }
    __syncthreads();
    const int todo = *nlater;
    tb.keys = reinterpret_cast<int*>(sm);
    tb.ckeys = tb.keys + kBigSlots;
    tb.vals = reinterpret_cast<unsigned long long*>(tb.ckeys + kBigSlots);
    tb.cvals = tb.vals + kBigSlots;
    for (int q = 0; q < todo; ++q) {
        const int i = later[c0 + q];
        const int s = b0 + start[i];
        int m = hash_row_block<V>(tb, shm, sh, aptr[i], aptr[i + 1], acol, aval, rb, bcol, bval, bmag, a.scol + s,
                                  a.sval + s, size ? size + i : nullptr);
        __syncthreads();
        if (threadIdx.x == 0) {
            if (m < 0) {
                atomicExch(&ctl->status, SMALL_LONG_ROW);
                m = 0;
                if (size) size[i] = Mag{0.0f, kMagNone};
            }
            start[i] = s;
            cnt[i] = m;
        }
    }
    __syncthreads();
}

// *most = entries of the longest cluster run of n rows
__device__ __forceinline__ void longest_run(int n, const int* ptr, int* most) {
    const int k = blockIdx.x * kT + threadIdx.x, ch = cluster_run(n);
    if (k < kClusterBlocks) atomicMax(most, ptr[min(n, (k + 1) * ch)] - ptr[min(n, k * ch)]);
}

template <class V>
__global__ void __launch_bounds__(kT, 1) k_small_setup(SmallArgs<V> a) {
    extern __shared__ unsigned long long sm64[];
    unsigned char* const sm = reinterpret_cast<unsigned char*>(sm64);
    __shared__ int sh[32], ok, nlater;
    __shared__ Mag shm[32];
    __shared__ long long base;
    SmallCtl* const ctl = a.ctl;
    int G = gridDim.x, GW = G * kWarps, GT = G * kT;
    const int cta = blockIdx.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int gw = cta * kWarps + wid, gt = cta * kT + threadIdx.x;
    const bool first = gt == 0;
    unsigned epoch = 0;
    int round = 0;
    float eps = a.eps;
    const int* ptr = a.ptr;
    const int* col = a.col;
    const V* val = a.val;
    int n = a.n, nnz = a.nnz;
    // the arena: what stays grows from the bottom, a level's scratch comes
    // from the top; every block makes the same allocations
    long long lo = 0, hi = a.cap;
    auto keep = [&](long long bytes) { const long long o = lo; lo += (bytes + 255) & ~255ll; return o; };
    auto temp = [&](long long bytes) { hi -= (bytes + 255) & ~255ll; return hi; };
#define SMALL_ROOM()                                      \
    do {                                                  \
        if (lo > hi) {                                    \
            if (first) atomicExch(&ctl->status, SMALL_NO_ROOM); \
            return;                                       \
        }                                                 \
    } while (0)
#define SMALL_SYNC()                                      \
    do {                                                  \
        if (!grid_sync(ctl, G, epoch, &ok)) return;       \
    } while (0)
    for (int l = 0;; ++l) {
        if (G > 1 && n <= kSoloRows && nnz <= kSoloNnz) {   // block 0 goes on alone
            if (cta != 0) return;
            G = 1;
            GW = kWarps;
            GT = kT;
        }
        SmallRec& rec = ctl->lev[l];
        hi = a.cap;
        const long long o_dinv = keep((long long)n * sizeof(V));
        V* const dinv = reinterpret_cast<V*>(a.arena + o_dinv);
        V* const dia = reinterpret_cast<V*>(a.arena + temp((long long)n * sizeof(V)));
        SMALL_ROOM();
        if (first) { rec.n = n; rec.nnz = nnz; rec.dinv = o_dinv; }
        longest_run(n, ptr, &rec.runA);
        const int vs = lanes_for(n, nnz, GT), rpw = 32 / vs, sub = lane % vs;
        // diagonal, its reciprocal, the Gershgorin bound of D^-1 A
        double ratio = 0.0;
        for (int r0 = gw * rpw; r0 < n; r0 += GW * rpw) {
            const int i = r0 + lane / vs;
            double rs = 0.0;
            unsigned long long at = 0;   // 1 + the last entry on the diagonal
            if (i < n)
                for (int k = ptr[i] + sub; k < ptr[i + 1]; k += vs) {
                    rs += fabs((double)val[k]);
                    if (col[k] == i) at = (unsigned long long)k + 1ull;
                }
            rs = group_sum(rs, vs);
            at = group_max(at, vs);
            if (i < n && sub == 0) {
                const double d = at ? (double)val[at - 1] : 0.0;
                if (!(d > 0.0) && !(d < 0.0)) atomicExch(&ctl->zero_diag, 1);
                if (!isfinite(d) || !isfinite(rs)) atomicExch(&ctl->non_finite, 1);
                dia[i] = (V)d;
                dinv[i] = (V)(1.0 / d);
                ratio = fmax(ratio, rs / fabs(d));
            }
        }
        {
            const unsigned long long m = group_max((unsigned long long)__double_as_longlong(ratio), 32);
            if (lane == 0 && m) atomicMax(&rec.lam, m);
        }
        SMALL_SYNC();
        if (ctl->zero_diag || ctl->non_finite || n <= a.coarse_enough || l == a.max_levels - 1) {
            if (first) ctl->nlev = l + 1;
            break;
        }
        // strength, and what the rounds start from
        unsigned char* const strong = a.arena + temp(nnz);
        unsigned char* const need = a.arena + temp(n);
        int* const prow = reinterpret_cast<int*>(a.arena + temp(4ll * nnz));
        V* const pnew = reinterpret_cast<V*>(a.arena + temp((long long)nnz * sizeof(V)));
        unsigned long long* const m1 = reinterpret_cast<unsigned long long*>(a.arena + temp(8ll * n));
        Mag* const psize = reinterpret_cast<Mag*>(a.arena + temp(8ll * n));
        Mag* const apsize = reinterpret_cast<Mag*>(a.arena + temp(8ll * n));
        int* const state = reinterpret_cast<int*>(a.arena + temp(4ll * n));
        int* const agg = reinterpret_cast<int*>(a.arena + temp(4ll * n));
        int* const agg2 = reinterpret_cast<int*>(a.arena + temp(4ll * n));
        int* const colcnt = reinterpret_cast<int*>(a.arena + temp(4ll * n));
        int* const fill = reinterpret_cast<int*>(a.arena + temp(4ll * n));
        int* const pcnt = reinterpret_cast<int*>(a.arena + temp(4ll * n));
        int* const apstart = reinterpret_cast<int*>(a.arena + temp(4ll * n));
        int* const apcnt = reinterpret_cast<int*>(a.arena + temp(4ll * n));
        int* const cstart = reinterpret_cast<int*>(a.arena + temp(4ll * n));
        int* const ccnt = reinterpret_cast<int*>(a.arena + temp(4ll * n));
        int* const later = reinterpret_cast<int*>(a.arena + temp(4ll * n));
        SMALL_ROOM();
        const double eps2 = (double)(eps * eps);
        eps *= 0.5f;
        for (int r0 = gw * rpw; r0 < n; r0 += GW * rpw) {
            const int i = r0 + lane / vs;
            int has = 0;
            if (i < n) {
                const V ed = (V)(eps2 * (double)dia[i]);
                for (int k = ptr[i] + sub; k < ptr[i + 1]; k += vs) {
                    const int j = col[k];
                    const V v = val[k];
                    const unsigned char s = (j != i) && (ed * dia[j] < v * v);
                    strong[k] = s;
                    has |= s;
                }
            }
            has = group_sum(has, vs);
            if (i < n && sub == 0) { state[i] = has ? 1 : -1; need[i] = 1; colcnt[i] = 0; }
        }
        SMALL_SYNC();
        // MIS(2): see amg_setup.cu for the round and its need flags
        bool settled = false;
        for (int it = 0; it < kMaxRounds && round < kRoundSlots; ++it, ++round) {
            for (int r0 = gw * rpw; r0 < n; r0 += GW * rpw) {
                const int i = r0 + lane / vs;
                const bool go = i < n && need[i];
                unsigned long long m = 0;
                if (go) {
                    if (sub == 0) m = mis_key(state[i], i);
                    for (int k = ptr[i] + sub; k < ptr[i + 1]; k += vs)
                        if (strong[k]) {
                            const int j = col[k];
                            const unsigned long long t = mis_key(state[j], j);
                            m = (t > m) ? t : m;
                        }
                }
                m = group_max(m, vs);
                if (go && sub == 0) { m1[i] = m; need[i] = 0; }
            }
            SMALL_SYNC();
            int left = 0;
            for (int r0 = gw * rpw; r0 < n; r0 += GW * rpw) {
                const int i = r0 + lane / vs;
                const bool active = i < n && state[i] == 1;
                unsigned long long m = 0;
                if (active) {
                    if (sub == 0) m = m1[i];
                    for (int k = ptr[i] + sub; k < ptr[i + 1]; k += vs)
                        if (strong[k]) { const unsigned long long t = m1[col[k]]; m = (t > m) ? t : m; }
                }
                m = group_max(m, vs);
                if (!active) continue;
                const bool root = m == mis_key(1, i);
                const bool covered = !root && (m >> 62) == 2ull;
                if (sub == 0) {
                    if (root) state[i] = 2;
                    else if (covered) state[i] = 0;
                    else ++left;
                }
                if (root || covered) continue;
                if (sub == 0) need[i] = 1;
                for (int k = ptr[i] + sub; k < ptr[i + 1]; k += vs)
                    if (strong[k]) need[col[k]] = 1;
            }
            __syncwarp();
            left = group_sum(left, 32);
            if (lane == 0 && left) atomicAdd(&ctl->undecided[round], left);
            SMALL_SYNC();
            if (*(volatile int*)&ctl->undecided[round] == 0) { settled = true; ++round; break; }
        }
        if (!settled) {
            if (first) atomicExch(&ctl->status, SMALL_NO_MIS);
            return;
        }
        // aggregates: roots numbered in row order; a block takes a run of rows
        const int ch = (n + G - 1) / G, c0 = min(n, cta * ch), c1 = min(n, c0 + ch);
        {
            int mine = 0;
            for (int i = c0 + threadIdx.x; i < c1; i += kT) mine += state[i] == 2;
            int total;
            block_scan(mine, sh, &total);
            if (threadIdx.x == 0) ctl->part[cta] = total;
        }
        SMALL_SYNC();
        int nagg;
        {
            int run = parts_before(ctl, G, sh, &nagg);
            for (int r0 = c0; r0 < c1; r0 += kT) {
                const int i = r0 + threadIdx.x;
                const int f = i < c1 && state[i] == 2;
                int total;
                const int off = block_scan(f, sh, &total);
                if (i < c1) agg[i] = f ? run + off : -1;
                run += total;
            }
        }
        SMALL_SYNC();
        if (nagg == 0 || nagg >= n) {
            if (first) ctl->nlev = l + 1;
            break;
        }
        // two passes of joining the strong neighbour with the largest key
        for (int pass = 0; pass < 2; ++pass) {
            const int* const in = pass ? agg2 : agg;
            int* const out = pass ? agg : agg2;
            for (int r0 = gw * rpw; r0 < n; r0 += GW * rpw) {
                const int i = r0 + lane / vs;
                const bool look = i < n && in[i] < 0 && state[i] >= 0;
                unsigned long long best = 0;   // key + 1; 0 = none
                if (look)
                    for (int k = ptr[i] + sub; k < ptr[i + 1]; k += vs) {
                        const int j = col[k];
                        if (!strong[k] || in[j] < 0) continue;
                        const unsigned long long kj =
                            (((unsigned long long)hash_u32((uint32_t)j) << 32) | (unsigned long long)j) + 1;
                        best = (kj > best) ? kj : best;
                    }
                best = group_max(best, vs);
                if (i < n && sub == 0) out[i] = look ? (best ? in[(int)((best - 1) & 0xffffffffull)] : -1) : in[i];
            }
            SMALL_SYNC();
        }
        // prolongation, a thread a row (its FP64 sums then fill the lanes of the
        // FP64 unit): the row's aggregates and their sums, in entry order, in a
        // list whose first kListed places are in shared memory and the others
        // at the row's place in A (it has no more aggregates than entries),
        // where the row ends up sorted
        {
            int* const sagg = reinterpret_cast<int*>(sm) + threadIdx.x;
            V* const ssum = reinterpret_cast<V*>(sm + sizeof(int) * kListed * kT) + threadIdx.x;
            int mine = 0;
            for (int i = c0 + threadIdx.x; i < c1; i += kT) {
                const int rb = ptr[i], re = ptr[i + 1];
                // entries are loaded kAhead at a time: one at a time, every entry
                // is two dependent round trips to L2
                constexpr int kAhead = sizeof(V) == 4 ? 8 : 4;
                int j[kAhead];
                V x[kAhead];
                bool st[kAhead];
                auto load = [&](int k0) {
#pragma unroll
                    for (int u = 0; u < kAhead; ++u) {
                        const int k = min(k0 + u, re - 1);
                        j[u] = col[k];
                        x[u] = val[k];
                        st[u] = strong[k] != 0;
                    }
                };
                double df = 0.0;
                for (int k0 = rb; k0 < re; k0 += kAhead) {
                    load(k0);
#pragma unroll
                    for (int u = 0; u < kAhead; ++u)
                        if (k0 + u < re && (j[u] == i || !st[u])) df += (double)x[u];
                }
                df = -a.omega * (1.0 / df);
                int m = 0;
                int* const lagg = prow + rb;
                V* const lsum = pnew + rb;
                for (int k0 = rb; k0 < re; k0 += kAhead) {
                    load(k0);
                    int g[kAhead];
#pragma unroll
                    for (int u = 0; u < kAhead; ++u)
                        g[u] = (k0 + u < re && (j[u] == i || st[u])) ? agg[j[u]] : -1;
#pragma unroll
                    for (int u = 0; u < kAhead; ++u) {
                        if (g[u] < 0) continue;
                        const double v = (j[u] == i) ? (1.0 - a.omega) : df * (double)x[u];
                        int t = 0;
                        while (t < m && (t < kListed ? sagg[t * kT] : lagg[t]) != g[u]) ++t;
                        V* const at = t < kListed ? ssum + t * kT : lsum + t;
                        if (t < m) { *at = (V)((double)*at + v); continue; }
                        (t < kListed ? sagg[t * kT] : lagg[t]) = g[u];
                        *at = (V)v;
                        ++m;
                    }
                }
                Mag size{0.0f, kMagNone};
                if (m <= kListed) {
                    for (int e = 0; e < m; ++e) {
                        const int g = sagg[e * kT];
                        const V v = ssum[e * kT];
                        int rank = 0;
                        for (int u = 0; u < m; ++u) rank += sagg[u * kT] < g;
                        lagg[rank] = g;
                        lsum[rank] = v;
                        mag_add(size, mag_of(v));
                        atomicAdd(colcnt + g, 1);
                    }
                } else {
                    for (int e = 0; e < kListed; ++e) { lagg[e] = sagg[e * kT]; lsum[e] = ssum[e * kT]; }
                    for (int e = 0; e < m; ++e) {   // insertion sort by aggregate
                        const int g = lagg[e];
                        const V v = lsum[e];
                        int t = e - 1;
                        while (t >= 0 && lagg[t] > g) { lagg[t + 1] = lagg[t]; lsum[t + 1] = lsum[t]; --t; }
                        lagg[t + 1] = g;
                        lsum[t + 1] = v;
                        mag_add(size, mag_of(v));
                        atomicAdd(colcnt + g, 1);
                    }
                }
                pcnt[i] = m;
                psize[i] = size;
                mine += m;
            }
            int total;
            block_scan(mine, sh, &total);
            if (threadIdx.x == 0) ctl->part[cta] = total;
        }
        SMALL_SYNC();
        int nnzP;
        int run = parts_before(ctl, G, sh, &nnzP);
        const long long o_pptr = keep(4ll * (n + 1)), o_pcol = keep(4ll * nnzP), o_pval = keep((long long)nnzP * sizeof(V));
        const long long o_rptr = keep(4ll * (nagg + 1)), o_rcol = keep(4ll * nnzP), o_rval = keep((long long)nnzP * sizeof(V));
        int* const tcol = reinterpret_cast<int*>(a.arena + temp(4ll * nnzP));
        V* const tval = reinterpret_cast<V*>(a.arena + temp((long long)nnzP * sizeof(V)));
        SMALL_ROOM();
        int* const pptr = reinterpret_cast<int*>(a.arena + o_pptr);
        int* const pcol = reinterpret_cast<int*>(a.arena + o_pcol);
        V* const pval = reinterpret_cast<V*>(a.arena + o_pval);
        int* const rptr = reinterpret_cast<int*>(a.arena + o_rptr);
        int* const rcol = reinterpret_cast<int*>(a.arena + o_rcol);
        V* const rval = reinterpret_cast<V*>(a.arena + o_rval);
        if (first) {
            rec.nagg = nagg; rec.nnzP = nnzP;
            rec.Pptr = o_pptr; rec.Pcol = o_pcol; rec.Pval = o_pval;
            rec.Rptr = o_rptr; rec.Rcol = o_rcol; rec.Rval = o_rval;
            pptr[n] = nnzP;
            rptr[nagg] = nnzP;
        }
        for (int r0 = c0; r0 < c1; r0 += kT) {
            const int i = r0 + threadIdx.x;
            int total;
            const int off = block_scan(i < c1 ? pcnt[i] : 0, sh, &total);
            if (i < c1) pptr[i] = run + off;
            run += total;
        }
        __syncthreads();
        for (int i = c0 + threadIdx.x; i < c1; i += kT) {
            const int rb = ptr[i], d = pptr[i], m = pcnt[i];
            for (int e = 0; e < m; ++e) {
                pcol[d + e] = prow[rb + e];
                pval[d + e] = pnew[rb + e];
            }
        }
        SMALL_SYNC();
        longest_run(n, pptr, &rec.runP);
        // R's row counts; A P of the block's rows
        const int qh = (nagg + G - 1) / G, q0 = min(nagg, cta * qh), q1 = min(nagg, q0 + qh);
        {
            int mine = 0;
            for (int q = q0 + threadIdx.x; q < q1; q += kT) mine += colcnt[q];
            int total;
            block_scan(mine, sh, &total);
            if (threadIdx.x == 0) ctl->part[cta] = total;
        }
        block_product<V>(a, l, c0, c1, ptr, col, val, RowSpan{pptr, nullptr}, pcol, pval, psize, apstart, apcnt, apsize,
                         later, sm, sh, shm, &nlater, &base);
        SMALL_SYNC();
        if (*(volatile int*)&ctl->status) return;
        {
            int all;
            int rrun = parts_before(ctl, G, sh, &all);
            for (int r0 = q0; r0 < q1; r0 += kT) {
                const int q = r0 + threadIdx.x;
                int total;
                const int off = block_scan(q < q1 ? colcnt[q] : 0, sh, &total);
                if (q < q1) { rptr[q] = rrun + off; fill[q] = rrun + off; }
                rrun += total;
            }
        }
        SMALL_SYNC();
        longest_run(nagg, rptr, &rec.runR);
        for (int i = gt; i < n; i += GT)
            for (int k = pptr[i]; k < pptr[i + 1]; ++k) {
                const int d = atomicAdd(fill + pcol[k], 1);
                tcol[d] = i;
                tval[d] = pval[k];
            }
        SMALL_SYNC();
        for (int q = gw; q < nagg; q += GW) {   // columns are unique: an entry's place is the number of smaller ones
            const int rb = rptr[q], re = rptr[q + 1];
            constexpr int kStageInts = kSlots * kTableSlotBytes / (int)sizeof(int);   // a warp's share of the tables
            int* const row = reinterpret_cast<int*>(sm) + (size_t)wid * kStageInts;
            const bool staged = re - rb <= kStageInts;
            if (staged)
                for (int e = rb + lane; e < re; e += 32) row[e - rb] = tcol[e];
            __syncwarp();
            const int* const cols = staged ? row : tcol + rb;
            for (int e = rb + lane; e < re; e += 32) {
                const int ce = cols[e - rb];
                int rank = 0;
                for (int u = 0; u < re - rb; ++u) rank += cols[u] < ce;
                rcol[rb + rank] = ce;
                rval[rb + rank] = tval[e];
            }
            __syncwarp();
        }
        SMALL_SYNC();
        // the next level's matrix: R (A P), then its rows to their exact places
        block_product<V>(a, l, q0, q1, rptr, rcol, rval, RowSpan{apstart, apcnt}, a.scol, a.sval, apsize, cstart, ccnt,
                         nullptr, later, sm, sh, shm, &nlater, &base);
        {
            int mine = 0;
            if (base >= 0)
                for (int q = q0 + threadIdx.x; q < q1; q += kT) mine += ccnt[q];
            int total;
            block_scan(mine, sh, &total);
            if (threadIdx.x == 0) ctl->part[cta] = total;
        }
        SMALL_SYNC();
        if (*(volatile int*)&ctl->status) return;
        int nnzC;
        int crun = parts_before(ctl, G, sh, &nnzC);
        const long long o_aptr = keep(4ll * (nagg + 1)), o_acol = keep(4ll * nnzC), o_aval = keep((long long)nnzC * sizeof(V));
        SMALL_ROOM();
        int* const nptr = reinterpret_cast<int*>(a.arena + o_aptr);
        int* const ncol = reinterpret_cast<int*>(a.arena + o_acol);
        V* const nval = reinterpret_cast<V*>(a.arena + o_aval);
        if (first) {
            SmallRec& nx = ctl->lev[l + 1];
            nx.Aptr = o_aptr; nx.Acol = o_acol; nx.Aval = o_aval;
            nptr[nagg] = nnzC;
        }
        for (int r0 = q0; r0 < q1; r0 += kT) {
            const int q = r0 + threadIdx.x;
            int total;
            const int off = block_scan(q < q1 ? ccnt[q] : 0, sh, &total);
            if (q < q1) nptr[q] = crun + off;
            crun += total;
        }
        __syncthreads();
        for (int q = q0 + wid; q < q1; q += kWarps) {
            const int s = cstart[q], d = nptr[q], m = ccnt[q];
            for (int e = lane; e < m; e += 32) {
                ncol[d + e] = a.scol[s + e];
                nval[d + e] = a.sval[s + e];
            }
        }
        SMALL_SYNC();
        ptr = nptr;
        col = ncol;
        val = nval;
        n = nagg;
        nnz = nnzC;
    }
    // the coarsest level's inverse (k_small_inverse)
    if (n <= kGjMax) {
        const long long o_inv = keep(8ll * n * n);
        if (lo > a.cap) {
            if (first) atomicExch(&ctl->status, SMALL_NO_ROOM);
        } else if (first) {
            ctl->cinv = o_inv;
        }
    }
    if (first) ctl->kept = lo;
#undef SMALL_ROOM
#undef SMALL_SYNC
}

// Explicit FP64 inverse of the coarsest level, one block: Gauss-Jordan in place
// with partial pivoting, the rows left where they are (a row is a pivot once).
// A thread holds rows q, q + 16, q + 32, q + 48 of one column in registers; a
// step passes the pivot's column and scaled row through shared memory.  Its bound
// is the FP64 unit of one multiprocessor: n^2 multiply-adds a step.  One thread
// divides: the reciprocal of the pivot in every thread was 2.6 us of each step,
// and matrix and inverse side by side in shared memory twice the multiply-adds.
template <class V>
__global__ void __launch_bounds__(kT, 1) k_small_inverse(SmallArgs<V> a) {
    static_assert(kGjMax == 64 && kT == 1024, "16 threads a column, 4 rows a thread");
    __shared__ double column[2][kGjMax], row[kGjMax], sinv;
    __shared__ int spiv, order[kGjMax], place[kGjMax];   // step -> pivot row; its inverse
    extern __shared__ double dense[];
    SmallCtl* const ctl = a.ctl;
    if (ctl->status || ctl->abort || ctl->nlev < 1) return;
    const int l = ctl->nlev - 1, n = ctl->lev[l].n;
    if (n > kGjMax) return;
    const int* ptr = l ? reinterpret_cast<const int*>(a.arena + ctl->lev[l].Aptr) : a.ptr;
    const int* col = l ? reinterpret_cast<const int*>(a.arena + ctl->lev[l].Acol) : a.col;
    const V* val = l ? reinterpret_cast<const V*>(a.arena + ctl->lev[l].Aval) : a.val;
    for (int t = threadIdx.x; t < n * n; t += kT) dense[t] = 0.0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += kT)
        for (int k = ptr[i]; k < ptr[i + 1]; ++k) dense[i * n + col[k]] = (double)val[k];
    __syncthreads();
    const int k = threadIdx.x & 63, q = threadIdx.x >> 6, lane = threadIdx.x & 31;
    double m[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int r = q + 16 * j;
        m[j] = (k < n && r < n) ? dense[r * n + k] : 0.0;
        if (k == 0) column[0][r] = m[j];
    }
    __syncthreads();
    unsigned long long used = 0;   // pivot rows so far (the first warp's)
    for (int c = 0; c < n; ++c) {
        const double* const f = column[c & 1];
        if (threadIdx.x < 32) {
            // the first largest |a_rc| of the rows left; magnitudes compare as integers
            unsigned long long best = 0;
            int p = n;
            for (int r = lane; r < n; r += 32) {
                const unsigned long long v = (unsigned long long)__double_as_longlong(f[r]) & 0x7fffffffffffffffull;
                if (!(used >> r & 1) && (p == n || v > best)) { best = v; p = r; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int op = __shfl_xor_sync(0xffffffffu, p, o);
                if (op < n && (p == n || ob > best || (ob == best && op < p))) { best = ob; p = op; }
            }
            used |= 1ull << p;   // c < n rows are used, so one is left
            if (lane == 0) {
                const double pv = f[p];
                if (!(fabs(pv) > 0.0)) ctl->singular = 1;
                spiv = p;
                sinv = 1.0 / pv;
                order[c] = p;
                place[p] = c;
            }
        }
        __syncthreads();
        const int p = spiv;
        const double ip = sinv;
        if (f[p] == 0.0) return;
        if (q == (p & 15) && k < n) {
            const double x = p < 32 ? (p < 16 ? m[0] : m[1]) : (p < 48 ? m[2] : m[3]);
            row[k] = k == c ? ip : x * ip;
        }
        __syncthreads();
        if (k < n) {
            const double rk = row[k];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int r = q + 16 * j;
                if (r >= n) continue;
                if (r == p) m[j] = rk;
                else m[j] = (k == c ? 0.0 : m[j]) - f[r] * rk;
                if (k == c + 1) column[(c + 1) & 1][r] = m[j];
            }
        }
        __syncthreads();
    }
    // row order[i] of the array is row i of the inverse, its column c belongs to right-hand side order[c]
    double* const out = reinterpret_cast<double*>(a.arena + ctl->cinv);
    if (k < n)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = q + 16 * j;
            if (r < n) out[place[r] * n + order[k]] = m[j];
        }
}

}  // namespace

size_t small_record_bytes() { return offsetof(SmallCtl, arrived); }

bool small_setup_fits(int n, int64_t nnz, bool mesh_matrix) {
    return n <= (mesh_matrix ? kBesideRows : kSmallRows) && nnz <= (mesh_matrix ? kBesideNnz : kSmallNnz);
}

template <class V>
SmallResult small_setup(semo_ctx* c, Amg<V>& h, float eps, double omega, const int* sflag) {
    cudaStream_t s = setup_stream(c);
    const int first = (int)h.lev.size() - 1;
    const DCsr<V>& A0 = h.lev[first].A;
    const int n = A0.n;
    const int64_t nnz = A0.nnz;
    DBuf<unsigned char> ctl;
    DBuf<int> scol;
    DBuf<V> sval;
    ctl.alloc(sizeof(SmallCtl), s);
    ctl.zero();
    SmallArgs<V> a{};
    a.ptr = A0.ptr; a.col = A0.col; a.val = A0.val;
    a.n = n;
    a.nnz = (int)nnz;
    a.eps = eps;
    a.coarse_enough = c->prm.coarse_enough;
    a.max_levels = std::min(c->prm.max_levels - first, kMaxLevels);
    a.omega = omega;
    // room: a level's scratch is 77 bytes a row and (2 + 12) an entry, what
    // stays at most 24 bytes an entry of P and 12 of the next matrix; the
    // products of mesh levels come to 5-9 an entry.  A matrix that needs more
    // goes to the level-by-level kernels.
    a.cap = 160ll * n + 96ll * nnz + (4ll << 20);
    a.slots = 10ll * nnz + 262144;
    h.arena.alloc((size_t)a.cap, s);
    scol.alloc((size_t)a.slots, s);
    sval.alloc((size_t)a.slots, s);
    a.arena = h.arena.p;
    a.scol = scol.p;
    a.sval = sval.p;
    a.ctl = reinterpret_cast<SmallCtl*>(ctl.p);
    // a block a multiprocessor at most, fewer for the smallest levels (the
    // barrier is then cheaper): about a thousand entries a block
    int grid = (int)std::min<int64_t>(std::min(sm_count(c->device), kMostBlocks), std::max<int64_t>(16, nnz / kNnzPerBlock));
    auto kern = k_small_setup<V>;
    SEMO_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kTableBytes));
    void* args[] = {&a};
    SEMO_CUDA(cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(kT), args, kTableBytes, s));
    SEMO_CHECK_LAUNCH();
    const int gj = kGjMax * kGjMax * (int)sizeof(double);
    k_small_inverse<V><<<1, kT, gj, s>>>(a);
    SEMO_CHECK_LAUNCH();
    SmallCtl& r = *reinterpret_cast<SmallCtl*>(c->hpin_small);
    SEMO_CUDA(cudaMemcpyAsync(&r, ctl.p, small_record_bytes(), cudaMemcpyDeviceToHost, s));
    SEMO_CUDA(cudaStreamSynchronize(s));   // whatever the caller queued before has landed too
    if (r.abort) throw Error(SEMO_ERR_CUDA, "AMG setup: a grid barrier was not reached");
    if (sflag[2]) r.zero_diag = 1;   // the levels above
    else if (sflag[3] && !r.zero_diag) r.non_finite = 1;
    if (r.zero_diag) throw Error(SEMO_ERR_ARGUMENT, "matrix has a zero diagonal entry");
    if (r.non_finite) throw Error(SEMO_ERR_NAN, "non-finite matrix entry");
    if (r.status == SMALL_NO_MIS) throw Error(SEMO_ERR_CUDA, "MIS(2) aggregation did not terminate");
    if (r.status == SMALL_LONG_ROW)
        throw Error(SEMO_ERR_CUDA, "SpGEMM row has more than " + std::to_string(kBigSlots * 3 / 4) + " distinct columns");
    if (r.status == SMALL_NO_ROOM) {
        h.arena.release();
        return SmallResult::no_room;
    }
    if (r.singular) throw Error(SEMO_ERR_BREAKDOWN, "coarsest AMG matrix is singular");
    if (a.cap - r.kept > kSpareBytes) {   // the levels stay, the scratch does not
        DBuf<unsigned char> kept;
        kept.alloc((size_t)r.kept, s);
        SEMO_CUDA(cudaMemcpyAsync(kept.p, h.arena.p, (size_t)r.kept, cudaMemcpyDeviceToDevice, s));
        h.arena = std::move(kept);
    }
    unsigned char* const A = h.arena.p;
    auto ints = [&](DBuf<int>& b, long long off, int64_t count) { b.view(reinterpret_cast<int*>(A + off), (size_t)count); };
    auto vals = [&](DBuf<V>& b, long long off, int64_t count) { b.view(reinterpret_cast<V*>(A + off), (size_t)count); };
    for (int l = 0; l < r.nlev; ++l) {
        const SmallRec& q = r.lev[l];
        if (l > 0) {
            h.lev.emplace_back();
            AmgLevel<V>& L = h.lev.back();
            L.A.n = L.A.m = q.n;
            L.A.nnz = q.nnz;
            ints(L.A.ptr, q.Aptr, q.n + 1);
            ints(L.A.col, q.Acol, q.nnz);
            vals(L.A.val, q.Aval, q.nnz);
        }
        AmgLevel<V>& L = h.lev.back();
        L.A.run = q.runA;
        L.P.run = q.runP;
        L.R.run = q.runR;
        vals(L.dinv, q.dinv, q.n);
        std::memcpy(&L.lam_max, &q.lam, sizeof(double));
        h.total_nnz += q.nnz;
        L.x.alloc(q.n, s); L.b.alloc(q.n, s); L.r.alloc(q.n, s); L.t.alloc(q.n, s);
        if (l + 1 < r.nlev) {
            L.nagg = q.nagg;
            L.P.n = q.n; L.P.m = q.nagg; L.P.nnz = q.nnzP;
            L.R.n = q.nagg; L.R.m = q.n; L.R.nnz = q.nnzP;
            ints(L.P.ptr, q.Pptr, q.n + 1);
            ints(L.P.col, q.Pcol, q.nnzP);
            vals(L.P.val, q.Pval, q.nnzP);
            ints(L.R.ptr, q.Rptr, q.nagg + 1);
            ints(L.R.col, q.Rcol, q.nnzP);
            vals(L.R.val, q.Rval, q.nnzP);
        }
    }
    h.coarse_n = h.lev.back().A.n;
    if (h.coarse_n > kGjMax) return SmallResult::needs_inverse;
    h.cinv.view(reinterpret_cast<double*>(A + r.cinv), (size_t)h.coarse_n * h.coarse_n);
    return SmallResult::done;
}
template SmallResult small_setup<float>(semo_ctx*, Amg<float>&, float, double, const int*);
template SmallResult small_setup<double>(semo_ctx*, Amg<double>&, float, double, const int*);

}  // namespace semo
