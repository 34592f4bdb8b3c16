// Row-wise pieces of the AMG setup shared by the level-by-level kernels
// (amg_setup.cu) and the single-kernel setup of small levels (amg_small.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

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
// Requires |a b| 2^sc < 2^63.
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
        q = (e < 64) ? (m << e) : 0ull;   // e <= 62 whenever the scale bound holds
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

// the same for doubles: the 53-bit significands multiply exactly into 106 bits,
// so the product is rounded once, where (a b) 2^sc in FP64 rounds twice and
// takes three instructions of the FP64 unit, 16 clocks a warp each
__host__ __device__ __forceinline__ long long fixed_product(double a, double b, int sc) {
#ifdef __CUDA_ARCH__
    const uint64_t ua = (uint64_t)__double_as_longlong(a), ub = (uint64_t)__double_as_longlong(b);
#else
    uint64_t ua, ub;
    memcpy(&ua, &a, 8);
    memcpy(&ub, &b, 8);
#endif
    int ea = (int)(ua >> 52) & 0x7ff, eb = (int)(ub >> 52) & 0x7ff;
    const uint64_t ma = (ua & 0xfffffffffffffull) | (ea ? 0x10000000000000ull : 0ull);
    const uint64_t mb = (ub & 0xfffffffffffffull) | (eb ? 0x10000000000000ull : 0ull);
    ea = ea ? ea : 1;
    eb = eb ? eb : 1;
    const unsigned __int128 m = (unsigned __int128)ma * mb;
    const uint64_t hi = (uint64_t)(m >> 64), lo = (uint64_t)m;
    const int sh = 2150 - ea - eb - sc;   // |a b| 2^sc = m 2^-sh
    uint64_t q, rem, half;
    if (sh <= 0) {   // m < 2^63 then, by the scale's bound
        q = sh > -64 ? lo << -sh : 0ull;
        rem = 0ull;
        half = 1ull;
    } else if (sh < 64) {
        q = (hi << (64 - sh)) | (lo >> sh);
        rem = lo << (64 - sh);   // the bits below the unit, at the top of a word
        half = 1ull << 63;
    } else if (sh < 128) {
        const int s = sh - 64;
        q = s ? hi >> s : hi;
        rem = s ? (hi << (64 - s)) | (lo >> s) | (lo << (64 - s) ? 1ull : 0ull) : lo;
        half = 1ull << 63;
    } else {
        q = rem = 0ull;   // below half a unit (m < 2^106)
        half = 1ull;
    }
    if (rem > half || (rem == half && (q & 1ull))) ++q;
    return ((ua ^ ub) >> 63) ? -(long long)q : (long long)q;
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
// fixed-point scale exponent for sums of at most s: s 2^sc < 2^63 by 2^-10 of it,
// which covers the roundings of the FP32 sums above (2^-24 an addition, 3,072 in a
// row at most) and of the scaled products (half a unit each)
__device__ __forceinline__ int mag_scale(Mag s) {
    const float m = s.m * 1.0009765625f;
    const int e = m > 0.0f ? s.e + (int)((__float_as_uint(m) >> 23) & 0xff) - 126 : -1022;   // s < 2^e
    return max(-960, min(1000, 63 - e));
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
// the row's sum of |products|, each product is scaled by 2^s, S 2^s < 2^63,
// and rounded to an integer -- an error of at most 2^-63 (S + 2^-10 S) per product, below
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
        // a step's products are fetched while the one before is summed
        int c = -1;
        V av = V(0), bv = V(0);
        auto fetch = [&](int t) {
            // owner lane: the last lane whose B-row run starts at or before t
            int j = 0;
#pragma unroll
            for (int step = 16; step >= 1; step >>= 1) {
                const int x = __shfl_sync(0xffffffffu, excl, j + step);
                if (x <= t) j += step;
            }
            const int q = __shfl_sync(0xffffffffu, bb, j) + (t - __shfl_sync(0xffffffffu, excl, j));
            av = __shfl_sync(0xffffffffu, avk, j);
            c = t < total ? bcol[q] : -1;
            if (t < total) bv = bval[q];
        };
        fetch(lane);
        for (int t0 = 0; t0 < total; t0 += 32) {
            const bool act = c >= 0;
            const int cc = c;
            const V a0 = av, b0 = bv;
            if (t0 + 32 < total) fetch(t0 + 32 + lane);
            int slot = -1;
            bool fresh = false;
            if (act) {
                uint32_t h = hash_u32((uint32_t)cc) & hmask;
                for (int probe = 0; probe < ht; ++probe) {
                    const int prev = atomicCAS(tb.keys + h, -1, cc);
                    if (prev == -1) { slot = (int)h; fresh = true; break; }
                    if (prev == cc) { slot = (int)h; break; }
                    h = (h + 1) & hmask;
                }
            }
            distinct += __popc(__ballot_sync(0xffffffffu, fresh));
            const bool lost = __any_sync(0xffffffffu, act && slot < 0);
            if (!lost && act)   // two's complement: signed sum mod 2^64
                shared_add64(tb.vals + slot, (unsigned long long)fixed_product(a0, b0, sc));
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

// Four short rows by one warp, 8 lanes and a table of 32 slots each (tb: the
// group's, with room for 32 slots): row [ab, ae) of the lane's group, ab == ae
// for none.  The sums are hash_row's.  A row of 26 products leaves a warp's lanes
// idle in all but one step and costs its latency, ~5 us, alone (A P of 262,144
// rows in the single-kernel setup 266 -> 118 us).  Returns the
// length, or -1 (nothing written) when more than 24 slots are taken; *size: the
// sum of |values|.
constexpr int kGroup = 8, kGroupSlots = 32;
__device__ __forceinline__ Mag mag_group_sum(Mag s) {
#pragma unroll
    for (int o = kGroup / 2; o > 0; o >>= 1) {
        const float m = __shfl_xor_sync(0xffffffffu, s.m, o);
        const int e = __shfl_xor_sync(0xffffffffu, s.e, o);
        const int top = max(e, s.e);   // the same in both lanes
        s.m = s.m * pow2_down(s.e - top) + m * pow2_down(e - top);
        s.e = top;
    }
    return s;
}
template <class V>
__device__ int hash_rows_short(int lane, RowTable tb, int ab, int ae, const int* acol, const V* aval, RowSpan rb,
                               const int* bcol, const V* bval, const Mag* bmag, int* ocol, V* oval, Mag* size) {
    const int sub = lane & (kGroup - 1), first = lane & ~(kGroup - 1);
    const unsigned group = ((1u << kGroup) - 1u) << first;
    __syncwarp();
#pragma unroll
    for (int t = sub; t < kGroupSlots; t += kGroup) { tb.keys[t] = -1; tb.vals[t] = 0ull; }
    Mag bound{0.0f, kMagNone};
    for (int ka = ab + sub; ka < ae; ka += kGroup) mag_add(bound, mag_mul(mag_of(aval[ka]), bmag[acol[ka]]));
    const int sc = mag_scale(mag_group_sum(bound));
    __syncwarp();
    int distinct = 0;
    bool full = false;
    for (int k0 = ab; __any_sync(0xffffffffu, k0 < ae && !full); k0 += kGroup) {
        const int k = k0 + sub;
        const bool ka = k < ae && !full;
        const int a = ka ? acol[k] : 0;
        const V avk = ka ? aval[k] : V(0);
        const int bb = ka ? rb.begin(a) : 0;
        const int blen = ka ? rb.count(a) : 0;
        int incl = blen;
#pragma unroll
        for (int o = 1; o < kGroup; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o, kGroup);
            if (sub >= o) incl += t;
        }
        const int total = __shfl_sync(0xffffffffu, incl, kGroup - 1, kGroup);
        const int excl = incl - blen;
        int c = -1;
        V av = V(0), bv = V(0);
        auto fetch = [&](int t) {
            int j = 0;
#pragma unroll
            for (int step = kGroup / 2; step >= 1; step >>= 1) {
                const int x = __shfl_sync(0xffffffffu, excl, j + step, kGroup);
                if (x <= t) j += step;
            }
            const int q = __shfl_sync(0xffffffffu, bb, j, kGroup) + (t - __shfl_sync(0xffffffffu, excl, j, kGroup));
            av = __shfl_sync(0xffffffffu, avk, j, kGroup);
            c = t < total ? bcol[q] : -1;
            if (t < total) bv = bval[q];
        };
        fetch(sub);
        for (int t0 = 0; __any_sync(0xffffffffu, t0 < total && !full); t0 += kGroup) {
            const bool act = c >= 0 && !full;
            const int cc = c;
            const V a0 = av, b0 = bv;
            fetch(t0 + kGroup + sub);
            int slot = -1;
            bool fresh = false;
            if (act) {
                uint32_t h = hash_u32((uint32_t)cc) & (kGroupSlots - 1);
                for (int probe = 0; probe < kGroupSlots; ++probe) {
                    const int prev = atomicCAS(tb.keys + h, -1, cc);
                    if (prev == -1) { slot = (int)h; fresh = true; break; }
                    if (prev == cc) { slot = (int)h; break; }
                    h = (h + 1) & (kGroupSlots - 1);
                }
            }
            distinct += __popc(__ballot_sync(0xffffffffu, fresh) & group);
            const bool lost = (__ballot_sync(0xffffffffu, act && slot < 0) & group) != 0;
            if (act && slot >= 0) shared_add64(tb.vals + slot, (unsigned long long)fixed_product(a0, b0, sc));
            full |= lost || distinct > (kGroupSlots * 3) / 4;
        }
    }
    __syncwarp();
    int m = 0;
#pragma unroll
    for (int t0 = 0; t0 < kGroupSlots; t0 += kGroup) {
        const bool occ = tb.keys[t0 + sub] >= 0;
        const unsigned bal = (__ballot_sync(0xffffffffu, occ) & group) >> first;
        if (occ) {
            const int pos = m + __popc(bal & ((1u << sub) - 1u));
            tb.ckeys[pos] = tb.keys[t0 + sub];
            tb.cvals[pos] = tb.vals[t0 + sub];
        }
        m += __popc(bal);
    }
    __syncwarp();
    Mag sum{0.0f, kMagNone};
    if (!full)
        for (int x = sub; x < m; x += kGroup) {
            const int ce = tb.ckeys[x];
            int rank = 0;
            for (int u = 0; u < m; ++u) rank += (tb.ckeys[u] < ce);
            const V v = fixed_value((long long)tb.cvals[x], sc, V(0));
            ocol[rank] = ce;
            oval[rank] = v;
            mag_add(sum, mag_of(v));
        }
    *size = mag_group_sum(sum);
    return full ? -1 : m;
}

}  // namespace amg
}  // namespace semo
