// Row-wise pieces of the AMG setup shared by the level-by-level kernels
// (amg_setup.cu) and the single-kernel setup of small levels (amg_small.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace semo {
namespace amg {

__device__ __forceinline__ uint32_t hash_u32(uint32_t x) {
    // integer avalanche mixer (public-domain "lowbias32" constants)
    x ^= x >> 16; x *= 0x7feb352dU; x ^= x >> 15; x *= 0x846ca68bU; x ^= x >> 16;
    return x;
}

__device__ __forceinline__ unsigned long long mis_key(int st, int i) {
    const unsigned long long s = (st < 0) ? 0ull : (unsigned long long)st;
    return (s << 62) | ((unsigned long long)hash_u32((uint32_t)i) << 30) | (unsigned long long)i;
}

// round(a b 2^sc) to the nearest integer (ties to even) for finite floats,
// on the integer pipes: the 24-bit significands multiply exactly into 48
// bits, so this equals __double2ll_rn(((double)a * b) * 2^sc) (the FP64
// product of two floats is exact too) without touching the FP64 unit.
// Requires |a b| 2^sc < 2^62.
__device__ __forceinline__ long long fixed_product(float a, float b, int sc) {
    const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
    int ea = (int)((ua >> 23) & 0xff), eb = (int)((ub >> 23) & 0xff);
    const uint32_t ma = (ua & 0x7fffffu) | (ea ? 0x800000u : 0u);
    const uint32_t mb = (ub & 0x7fffffu) | (eb ? 0x800000u : 0u);
    ea = ea ? ea : 1;
    eb = eb ? eb : 1;
    const unsigned long long m = (unsigned long long)ma * (unsigned long long)mb;   // exact
    const int e = (ea - 150) + (eb - 150) + sc;                                     // |a b| 2^sc = m 2^e
    unsigned long long q;
    if (m == 0ull) {
        q = 0ull;
    } else if (e >= 0) {
        q = (e < 64) ? (m << e) : 0ull;   // e <= 61 whenever the scale bound holds
    } else if (e <= -64) {
        q = 0ull;   // below half a unit (m < 2^48)
    } else {
        const int sh = -e;
        q = m >> sh;
        const unsigned long long rem = m & ((1ull << sh) - 1ull), half = 1ull << (sh - 1);
        if (rem > half || (rem == half && (q & 1ull))) ++q;
    }
    return ((ua ^ ub) >> 31) ? -(long long)q : (long long)q;
}

// A magnitude in FP32 with an exponent of its own: at most m 2^e.  The products'
// fixed-point scales need only the exponent of a row's sum of |products|; in
// FP64 (2 lanes a clock and multiprocessor on GB300, a warp instruction 16
// clocks) those sums, their shuffle trees and the conversions of the results
// cost more than the products: ~25 FP64 instructions a row.
struct Mag {
    float m;
    int e;
};
constexpr int kMagNone = -100000;
__device__ __forceinline__ float pow2_down(int d) {   // 2^d, d <= 0 (0 below 2^-126)
    return d < -126 ? 0.0f : __int_as_float((127 + d) << 23);
}
__device__ __forceinline__ Mag mag_of(float v) {
    const uint32_t u = __float_as_uint(v) & 0x7fffffffu;
    const int ex = (int)(u >> 23);
    if (ex == 0) return Mag{__uint2float_rn(u) * 1.1920928955078125e-07f, -126};   // u 2^-149
    return Mag{__uint_as_float((u & 0x7fffffu) | 0x3f800000u), ex - 127};
}
__device__ __forceinline__ Mag mag_of(double v) {   // rounded up to 20 bits
    const uint32_t hi = (uint32_t)__double2hiint(v) & 0x7fffffffu;
    const int ex = (int)(hi >> 20);
    if (ex == 0) return Mag{(hi | (uint32_t)__double2loint(v)) ? 1.0f : 0.0f, -1022};
    return Mag{__uint_as_float(0x3f800000u | ((hi & 0xfffffu) << 3)) + 9.5367431640625e-07f, ex - 1023};
}
__device__ __forceinline__ void mag_add(Mag& s, Mag x) {
    if (x.e > s.e) { s.m = s.m * pow2_down(s.e - x.e) + x.m; s.e = x.e; }
    else s.m += x.m * pow2_down(x.e - s.e);
}
__device__ __forceinline__ Mag mag_mul(Mag a, Mag b) { return Mag{a.m * b.m, a.e + b.e}; }
// the sum over the warp (every lane gets it)
__device__ __forceinline__ Mag mag_warp_sum(Mag s) {
    const int e = __reduce_max_sync(0xffffffffu, s.e);
    float m = s.m * pow2_down(s.e - e);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
    return Mag{m, e};
}
// fixed-point scale exponent for sums of at most s: s 2^sc < 2^62.  The FP32
// sums above round a few times; 2^-10 covers them.
__device__ __forceinline__ int mag_scale(Mag s) {
    const float m = s.m * 1.0009765625f;
    const int e = m > 0.0f ? s.e + (int)((__float_as_uint(m) >> 23) & 0xff) - 126 : -1022;   // s < 2^e
    return max(-960, min(1000, 62 - e));
}
// q 2^-sc rounded to the nearest V
__device__ __forceinline__ double fixed_value(long long q, int sc, double) {
    return (double)q * __longlong_as_double((long long)(1023 - sc) << 52);
}
__device__ __forceinline__ float fixed_value(long long q, int sc, float) {
    const uint32_t u = __float_as_uint(__ll2float_rn(q));
    if ((u << 1) == 0u) return 0.0f;
    const int ex = (int)((u >> 23) & 0xff) - sc;
    if (ex > 0 && ex < 255) return __uint_as_float((u & 0x807fffffu) | ((uint32_t)ex << 23));
    return (float)fixed_value(q, sc, 0.0);   // under- or overflow
}

// Rows of the right-hand factor of a product: CSR (len null) or slots with a
// start and a length each.
struct RowSpan {
    const int* start;
    const int* len;
    __device__ __forceinline__ int begin(int a) const { return start[a]; }
    __device__ __forceinline__ int count(int a) const { return len ? len[a] : start[a + 1] - start[a]; }
};

// A warp's table in shared memory: open addressing while the row is summed,
// then the occupied slots compacted.
struct RowTable {
    int *keys, *ckeys;
    unsigned long long *vals, *cvals;
};
// *p += x in shared memory as two 32-bit atomic additions, the low word's
// carry going into the high one.  The 64-bit shared atomicAdd is a
// compare-and-swap loop, and a coarse row's 32 products meet in a few columns:
// the loop's retries took ~2 us a step of 32 products.
__device__ __forceinline__ void shared_add64(unsigned long long* p, unsigned long long x) {
    unsigned* const w = reinterpret_cast<unsigned*>(p);
    const unsigned lo = (unsigned)x, old = atomicAdd(w, lo);
    const unsigned hi = (unsigned)(x >> 32) + (old + lo < old ? 1u : 0u);
    if (hi) atomicAdd(w + 1, hi);
}
constexpr int kTableSlotBytes = 2 * (int)(sizeof(int) + sizeof(unsigned long long));

// table size (power of two, 32..limit) for a row with at most `most` distinct columns
__device__ __forceinline__ int table_size(int most, int limit) {
    const int need = (4 * most) / 3 + 2;
    int ht = 32;
    while (ht < need && ht < limit) ht <<= 1;
    return ht;
}

// One row of C = A B, by one warp: row entries acol/aval [ab, ae), rows of B by
// rb, bmag[k] >= sum_j |b_kj|.  Products are consumed in a fixed order (A entries
// in row order, B entries in chunks of 32) and summed as 64-bit fixed-point
// integers (integer addition is associative, so the sums do not depend on the
// order the shared-memory atomics land in): with S = sum_k |a_ik| bmag_k >=
// the row's sum of |products|, each product is scaled by 2^s, S 2^s < 2^62,
// and rounded to an integer -- an error of at most 2^-62 S per product, below
// what FP64 accumulation of the same products incurs (2^-53 S per addition).
// The row is written sorted by column to ocol/oval.  Returns its length, or
// -1 (nothing written) when more than 3/4 of the ht slots are taken.
template <class V>
__device__ int hash_row(int lane, int ht, RowTable tb, int ab, int ae, const int* acol, const V* aval, RowSpan rb,
                        const int* bcol, const V* bval, const Mag* bmag, int* ocol, V* oval) {
    __syncwarp();
    const int hmask = ht - 1;
    for (int t = lane; t < ht; t += 32) { tb.keys[t] = -1; tb.vals[t] = 0ull; }
    Mag bound{0.0f, kMagNone};
    for (int ka = ab + lane; ka < ae; ka += 32) mag_add(bound, mag_mul(mag_of(aval[ka]), bmag[acol[ka]]));
    const int sc = mag_scale(mag_warp_sum(bound));   // the row's scale 2^sc (a fixed tree: deterministic)
    const double up_scale = __longlong_as_double((long long)(1023 + sc) << 52);   // 2^sc (FP64 values)
    __syncwarp();
    int distinct = 0;
    bool full = false;
    // Products in a fixed flattened order: up to 32 A entries at a time,
    // their B rows laid end to end, 32 products per step.
    for (int k0 = ab; k0 < ae && !full; k0 += 32) {
        const int k = k0 + lane;
        const bool ka = k < ae;
        const int a = ka ? acol[k] : 0;
        const V avk = ka ? aval[k] : V(0);
        const int bb = ka ? rb.begin(a) : 0;
        const int blen = ka ? rb.count(a) : 0;
        int incl = blen;   // inclusive scan of the B row lengths over the lanes
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        const int excl = incl - blen;
        for (int t0 = 0; t0 < total; t0 += 32) {
            const int t = t0 + lane;
            const bool act = t < total;
            // owner lane: the last lane whose B-row run starts at or before t
            int j = 0;
#pragma unroll
            for (int step = 16; step >= 1; step >>= 1) {
                const int x = __shfl_sync(0xffffffffu, excl, j + step);
                if (x <= t) j += step;
            }
            const int q = __shfl_sync(0xffffffffu, bb, j) + (t - __shfl_sync(0xffffffffu, excl, j));
            const V av = __shfl_sync(0xffffffffu, avk, j);
            const int c = act ? bcol[q] : -1;
            int slot = -1;
            bool fresh = false;
            if (act) {
                uint32_t h = hash_u32((uint32_t)c) & hmask;
                for (int probe = 0; probe < ht; ++probe) {
                    const int prev = atomicCAS(tb.keys + h, -1, c);
                    if (prev == -1) { slot = (int)h; fresh = true; break; }
                    if (prev == c) { slot = (int)h; break; }
                    h = (h + 1) & hmask;
                }
            }
            distinct += __popc(__ballot_sync(0xffffffffu, fresh));
            const bool lost = __any_sync(0xffffffffu, act && slot < 0);
            if (!lost && act) {
                long long fx;
                if constexpr (sizeof(V) == 4) fx = fixed_product(av, bval[q], sc);
                else fx = __double2ll_rn((av * bval[q]) * up_scale);
                shared_add64(tb.vals + slot, (unsigned long long)fx);   // two's complement: signed sum mod 2^64
            }
            __syncwarp();
            if (lost || distinct > (ht * 3) / 4) { full = true; break; }
        }
    }
    if (full) return -1;
    // compact occupied slots (slot order), then rank by column
    int m = 0;
    for (int t0 = 0; t0 < ht; t0 += 32) {
        const int t = t0 + lane;
        const bool occ = tb.keys[t] >= 0;
        const unsigned bal = __ballot_sync(0xffffffffu, occ);
        if (occ) {
            const int pos = m + __popc(bal & ((1u << lane) - 1u));
            tb.ckeys[pos] = tb.keys[t];
            tb.cvals[pos] = tb.vals[t];
        }
        m += __popc(bal);
    }
    __syncwarp();
    for (int x = lane; x < m; x += 32) {
        const int ce = tb.ckeys[x];
        int rank = 0;
        for (int u = 0; u < m; ++u) rank += (tb.ckeys[u] < ce);
        ocol[rank] = ce;
        oval[rank] = fixed_value((long long)tb.cvals[x], sc, V(0));
    }
    return m;
}

}  // namespace amg
}  // namespace semo
