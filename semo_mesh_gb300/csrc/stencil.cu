// Vertex-stencil pass: least-squares gradients and stencil limits of five cell
// fields (setCellVarMinMax x4 + calcLeastSquare("cellVertex","1st") x5,
// src/solvers/cellVarMinMax.cpp:8-23, src/math/gradient.cpp:761-816, :997-1050,
// :1136-1159).
//
// A gradient is sum_k g_k (phi_k - phi_i) over the vertex neighbours and
// boundary faces, with g_k = M^-1 w_k d_k formed once per mesh, and is summed as
// sum_k g_k phi_k - phi_i sum_k g_k.  The sums run in fixed point on the integer
// pipes: with FP64 multiply-adds (15 an entry) the kernel took 1.59 ms at 128^3
// cells, 94 % of the FP64 unit's issue rate (2 lanes a clock and
// multiprocessor); an exact integer multiply-add of two 28-bit limbs is one
// instruction of 64 lanes a clock.
//   weights  g = (2^28 gh + gl) 2^(Ew - 54) per cell and component, |gh| <= 2^26,
//            gl in [-2^27, 2^27): 54 bits of the cell's largest weight, as two
//            ints, the bytes of the double they stand for
//   values   phi = (2^28 ph + pl) 2^(E - 1077), |ph| <= 2^27, pl in [0, 2^28): 55
//            bits of the stencil's largest |phi| (a first walk over the stencil
//            finds its exponent E)
//   sums     sum gh ph and sum (gh pl + gl ph), exact in 64 bits (the second is
//            carried into the first every 64 entries; a stencil has at most 1,024);
//            gl pl, 2^-54 of the largest product, is left out
// Against __float128 on jittered 26-entry stencils the sum's error is 2.9e-16 of
// the largest product in the rms for fields of the solver's kinds, the FP64
// chain's 3.7e-16 (uniform velocities: 3.0 against 3.7; a volume fraction across
// its interface: 2.3 against 4.2; a pressure of 1e5 with 1 % noise: 1.5 each).
// What bounds it now: integer issue (unpacking a value is ~15 instructions, the
// limits 11, the products 9), then the 1 KB a cell of weights, indices and
// results.  Measured at 128^3: five fields 1.39 ms (1.59 before), U, V, W alone
// 0.81 ms (0.95).
//
// The limits stay bit-exact: they compare order-preserving images of the doubles.
#include <cuda_runtime.h>

#include <algorithm>

#include "face_common.cuh"
#include "semo_internal.h"

namespace {

using namespace semo::face;

constexpr int kW = 54;        // bits of a weight
constexpr int kCarry = 64;    // entries between carries
__device__ __forceinline__ int exp_of(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// Once per mesh: the fixed-point weights of each cell's stencil entries (3
// planes of stn), their exponents Ew (3 planes of nc), the boundary faces'
// weights M^-1 w d (3 planes of nb) and the sums of all weights (3 planes of nc).
__global__ void k_stencil_weights(int nc, int ni, int nb, const int* __restrict__ stp, int64_t stn,
                                  const double* __restrict__ stw, const int* __restrict__ cfp,
                                  const int* __restrict__ cfi, const double* __restrict__ bfw,
                                  const double* __restrict__ minv, int2* __restrict__ stf, int* __restrict__ stfe,
                                  double* __restrict__ bfg, double* __restrict__ sum) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nc) return;
    const size_t N = nc;
    const double m[3][3] = {{minv[i], minv[N + i], minv[2 * N + i]},
                            {minv[N + i], minv[3 * N + i], minv[4 * N + i]},
                            {minv[2 * N + i], minv[4 * N + i], minv[5 * N + i]}};
    int e[3] = {0, 0, 0};
    for (int k = stp[i]; k < stp[i + 1]; ++k) {
        const double w[3] = {stw[3 * (int64_t)k], stw[3 * (int64_t)k + 1], stw[3 * (int64_t)k + 2]};
#pragma unroll
        for (int c = 0; c < 3; ++c) e[c] = max(e[c], exp_of(m[c][0] * w[0] + m[c][1] * w[1] + m[c][2] * w[2]));
    }
    long long s[3] = {0, 0, 0};
#pragma unroll
    for (int c = 0; c < 3; ++c) e[c] -= 1022;   // |g| < 2^e
    for (int k = stp[i]; k < stp[i + 1]; ++k) {
        const double w[3] = {stw[3 * (int64_t)k], stw[3 * (int64_t)k + 1], stw[3 * (int64_t)k + 2]};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const long long q = __double2ll_rn(ldexp(m[c][0] * w[0] + m[c][1] * w[1] + m[c][2] * w[2], kW - e[c]));
            const long long hi = (q + (1ll << 27)) >> 28;
            stf[c * stn + k] = make_int2((int)hi, (int)(q - hi * (1ll << 28)));
            s[c] += q;
        }
    }
    double t[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        stfe[c * N + i] = e[c];
        t[c] = ldexp((double)s[c], e[c] - kW);
    }
    for (int k = cfp[i]; k < cfp[i + 1]; ++k) {
        const int b = (cfi[k] & kFaceMask) - ni;
        if (b < 0) continue;
        const double w[3] = {bfw[b], bfw[nb + b], bfw[2 * nb + b]};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double g = m[c][0] * w[0] + m[c][1] * w[1] + m[c][2] * w[2];
            bfg[(size_t)c * nb + b] = g;
            t[c] += g;
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) sum[c * N + i] = t[c];
}

struct Fields5 {
    const double* p[5];
};

// (hh 2^28 + mid) 2^(28 + ex) in FP64, mid carried
__device__ __forceinline__ double fixed_sum(long long hh, long long mid, int ex) {
    hh += mid >> 28;
    const int lo = (int)(mid & 0xfffffff);
    // as many of lo's bits as fit beside hh in 64
    const int room = min(28, __clzll(hh ^ (hh >> 63)) - 1);
    const double d = __ll2double_rn((hh << room) | (long long)(lo >> (28 - room)));
    const int p = ex + 56 - room, hi = __double2hiint(d);
    const int be = ((hi >> 20) & 0x7ff) + p;   // the exponent is added in place
    if (be <= 0 || be >= 2047 || d == 0.0) return d == 0.0 ? 0.0 : ldexp(d, p);
    return __hiloint2double(hi + p * (1 << 20), __double2loint(d));
}

// fields F0 .. F1 - 1 of (P, U, V, W, VF): gradients (plane 3 q + c of grad) and
// limits (mm planes maxU,minU,maxV,minV,maxW,minW,maxVF,minVF,maxP,minP); the
// other planes are left as they are.  bf: boundary-face values, 5 planes of nb.
template <int F0, int F1>
__global__ void __launch_bounds__(128, 4) k_stencil(int nc, int ni, int nb, const int* __restrict__ stp,
                                                 const int* __restrict__ sti, const int2* __restrict__ stf,
                                                 const int* __restrict__ stfe, int64_t stn,
                                                 const int* __restrict__ cfp, const int* __restrict__ cfi,
                                                 const double* __restrict__ bfg, const double* __restrict__ sum,
                                                 Fields5 F, const double* __restrict__ bf,
                                                 double* __restrict__ grad, double* __restrict__ mm) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nc) return;
    constexpr int n = F1 - F0;
    const size_t N = nc;
    const int kb = stp[i], ke = stp[i + 1];
    // exponent of the largest |phi| of the stencil (hi words: sign off)
    int top[n];
#pragma unroll
    for (int q = 0; q < n; ++q) top[q] = 0;
#pragma unroll 4
    for (int k = kb; k < ke; ++k) {
        const int j = __ldg(sti + k);
#pragma unroll
        for (int q = 0; q < n; ++q)
            top[q] = max(top[q], __ldg(reinterpret_cast<const int*>(F.p[F0 + q]) + 2 * (size_t)j + 1) & 0x7fffffff);
    }
    // at least 64, so that a zero, whose exponent field is 0, is shifted out; a
    // stencil whose values are all below 2^-958 so counts as zero
#pragma unroll
    for (int q = 0; q < n; ++q) top[q] = max(top[q] >> 20, 64);
    long long kmax[n], kmin[n], hh[n][3], mid[n][3];
    double phi[n];
#pragma unroll
    for (int q = 0; q < n; ++q) {
        phi[q] = F.p[F0 + q][i];
        kmax[q] = kmin[q] = okey(phi[q]);
#pragma unroll
        for (int c = 0; c < 3; ++c) hh[q][c] = mid[q][c] = 0;
    }
    // an entry's weights and values are fetched while the one before it is
    // summed, its index two entries ahead
    int jn = 0;
    double vn[n];
    int2 gn[3];
    auto fetch = [&](int k) {   // entry k, its index in jn; then the index of k + 1
#pragma unroll
        for (int q = 0; q < n; ++q) vn[q] = __ldg(F.p[F0 + q] + jn);
#pragma unroll
        for (int c = 0; c < 3; ++c) gn[c] = __ldg(stf + c * stn + k);
        jn = __ldg(sti + min(k + 1, ke - 1));
    };
    if (kb < ke) {
        jn = __ldg(sti + kb);
        fetch(kb);
    }
    for (int k0 = kb; k0 < ke; k0 += kCarry) {
        const int k1 = min(k0 + kCarry, ke);
        for (int k = k0; k < k1; ++k) {
            double val[n];
            int2 g[3];
#pragma unroll
            for (int q = 0; q < n; ++q) val[q] = vn[q];
#pragma unroll
            for (int c = 0; c < 3; ++c) g[c] = gn[c];
            fetch(min(k + 1, ke - 1));
#pragma unroll
            for (int q = 0; q < n; ++q) {
                const double v = val[q];
                const long long t = okey(v);
                kmax[q] = (kmax[q] < t) ? t : kmax[q];
                kmin[q] = (t < kmin[q]) ? t : kmin[q];
                // the key's mantissa, inverted below zero, is a two's complement
                // significand but for its last bit: 1.m 2^62 with the implicit
                // bit (01 or 10) put in front; -0 goes in front as 0 does
                const int kh = (int)(t >> 32), s = kh >> 31;
                const int e = ((kh ^ s) >> 20) & 0x7ff;
                const unsigned lead = (e != 0 && s != 0) ? 0x80000000u : 0x40000000u;
                const unsigned mh = ((unsigned)(t >> 22) & 0x3fffffffu) | lead;
                const long long m = ((long long)(int)mh << 32) | (unsigned)((unsigned)t << 10);
                const int sh = top[q] - e;
                const int ph = (int)mh >> min(sh + 4, 31);
                const int pl = (int)(m >> min(sh + 8, 63)) & 0xfffffff;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    hh[q][c] += (long long)g[c].x * ph;
                    mid[q][c] += (long long)g[c].x * pl;
                    mid[q][c] += (long long)g[c].y * ph;
                }
            }
        }
#pragma unroll
        for (int q = 0; q < n; ++q)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                hh[q][c] += mid[q][c] >> 28;
                mid[q][c] &= 0xfffffff;
            }
    }
    double a[n][3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int ew = stfe[c * N + i];
        const double S = sum[c * N + i];
#pragma unroll
        for (int q = 0; q < n; ++q) {
            // a field that is not finite somewhere in the stencil has no gradient there
            const double g = top[q] == 0x7ff ? __longlong_as_double(0x7ff8000000000000LL)
                                             : fixed_sum(hh[q][c], mid[q][c], ew - kW + top[q] - 1077);
            a[q][c] = fma(-phi[q], S, g);
        }
    }
    // boundary faces (face index >= ni) come last in the ascending list
    int k = cfp[i + 1];
    const int fb = cfp[i];
    while (k > fb && (cfi[k - 1] & kFaceMask) >= ni) {
        --k;
        const int b = (cfi[k] & kFaceMask) - ni;
        const double g[3] = {bfg[b], bfg[nb + b], bfg[2 * (size_t)nb + b]};
#pragma unroll
        for (int q = 0; q < n; ++q) {
            const double v = bf[(size_t)(F0 + q) * nb + b];
#pragma unroll
            for (int c = 0; c < 3; ++c) a[q][c] = fma(g[c], v, a[q][c]);
        }
    }
#pragma unroll
    for (int q = 0; q < n; ++q) {
        // limits: U, V, W, VF, P in that order
        const int f = F0 + q, at = f == 0 ? 8 : (f == 4 ? 6 : 2 * (f - 1));
#pragma unroll
        for (int c = 0; c < 3; ++c) grad[(size_t)(3 * f + c) * N + i] = a[q][c];
        mm[(size_t)at * N + i] = ounkey(kmax[q]);
        mm[(size_t)(at + 1) * N + i] = ounkey(kmin[q]);
    }
}

}  // namespace

namespace semo {

void stencil_weights(semo_ctx* c) {
    cudaStream_t s = c->stream;
    const size_t stn = (size_t)std::max<int64_t>(c->st_nnz, 1), N = c->nc;
    c->stf.alloc(3 * stn, s);
    c->stfe.alloc(3 * N, s);
    c->stfs.alloc(3 * N, s);
    c->bfg.alloc(3 * (size_t)std::max(c->nb, 1), s);
    k_stencil_weights<<<blocks(c->nc, 128), 128, 0, s>>>(c->nc, c->ni, c->nb, c->st_ptr, c->st_nnz, c->stw, c->cf_ptr,
                                                         c->cf_idx, c->bfw, c->minv, c->stf, c->stfe, c->bfg,
                                                         c->stfs);
    SEMO_CHECK_LAUNCH();
}

void lsq_gradients(semo_ctx* c, const double* const* f, const double* bf, double* grad, double* mm, bool uvw_only) {
    Fields5 F;
    for (int q = 0; q < 5; ++q) F.p[q] = f[q];
    auto launch = [&](auto kern) {
        kern<<<blocks(c->nc, 128), 128, 0, c->stream>>>(c->nc, c->ni, c->nb, c->st_ptr, c->st_idx, c->stf, c->stfe,
                                                        c->st_nnz, c->cf_ptr, c->cf_idx, c->bfg, c->stfs, F, bf, grad,
                                                        mm);
        SEMO_CHECK_LAUNCH();
    };
    if (uvw_only) launch(k_stencil<1, 4>);
    else launch(k_stencil<0, 5>);
}

void lsq_gradients5(semo_ctx* c, const double* f0, const double* f1, const double* f2, const double* f3,
                    const double* f4, const double* bf, double* grad, double* mm) {
    const double* const f[5] = {f0, f1, f2, f3, f4};
    lsq_gradients(c, f, bf, grad, mm, false);
}

void stencil_pass(semo_ctx* c, bool full) {
    StageScope sc(c, full ? ST_STENCIL : ST_STENCIL_UVW);
    const double* const f[5] = {c->P, c->U, c->V, c->W, c->VF};
    lsq_gradients(c, f, c->bface, c->grad, c->mm, !full);
}

}  // namespace semo
