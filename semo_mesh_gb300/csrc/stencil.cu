// Vertex-stencil pass: least-squares gradients and stencil limits of five cell
// fields (setCellVarMinMax x4 + calcLeastSquare("cellVertex","1st") x5,
// src/solvers/cellVarMinMax.cpp:8-23, src/math/gradient.cpp:761-816, :997-1050,
// :1136-1159).
//
// One pass over each cell's stencil.  The weight vectors w_k d_k are formed once
// per mesh, and so is their per-cell sum S (stencil and boundary faces): the sum
// sum_k w_k (phi_k - phi_i) is formed as sum_k w_k phi_k - phi_i S, three
// multiply-adds an entry and field instead of a difference and three.  What
// bounds it is the FP64 unit (2 lanes a clock and multiprocessor on GB300): 15
// multiply-adds an entry for five fields, 1.59 ms at 128^3 cells, 94 % of the
// unit's issue rate (0.34 ms at 75^3); U, V, W alone 0.95 ms.  The limits compare order-preserving
// integer images of the doubles, off that unit.
//
// The same sums in fixed point on the integer pipes (54-bit weights, 55-bit values
// with one exponent a cell and field) took 1.39 and 0.81 ms (0.23 at 75^3), but
// their error is relative to the largest weight times the largest value of the
// stencil and not to the largest product: on stretched lattices, and beside values
// 2^20 times a cell's own, it was up to 5,900 times the bound of the sums here.
#include <cuda_runtime.h>

#include "face_common.cuh"
#include "semo_internal.h"

namespace {

using namespace semo::face;

struct Fields5 {
    const double* p[5];
};

// fields F0 .. F1 - 1 of (P, U, V, W, VF): gradients (plane 3 q + c of grad) and
// limits (mm planes maxU,minU,maxV,minV,maxW,minW,maxVF,minVF,maxP,minP); the
// other planes are left as they are.  bf: boundary-face values, 5 planes of nb.
template <int F0, int F1>
__global__ void __launch_bounds__(128) k_stencil(int nc, int ni, int nb, const int* __restrict__ stp,
                                                 const int* __restrict__ sti, const double* __restrict__ stw,
                                                 const int* __restrict__ cfp, const int* __restrict__ cfi,
                                                 const double* __restrict__ bfw, const double* __restrict__ stws,
                                                 const double* __restrict__ minv, Fields5 F,
                                                 const double* __restrict__ bf, double* __restrict__ grad,
                                                 double* __restrict__ mm) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nc) return;
    constexpr int n = F1 - F0;
    const size_t N = nc;
    double phi[n], g[n][3];
    long long kmax[n], kmin[n];
#pragma unroll
    for (int q = 0; q < n; ++q) {
        phi[q] = F.p[F0 + q][i];
        kmax[q] = kmin[q] = okey(phi[q]);
        g[q][0] = g[q][1] = g[q][2] = 0.0;
    }
    const int ke = stp[i + 1];
    for (int k = stp[i]; k < ke; ++k) {
        const int j = __ldg(sti + k);
        const double* const wk = stw + 3 * (int64_t)k;
        const double wx = __ldg(wk), wy = __ldg(wk + 1), wz = __ldg(wk + 2);
        double v[n];
#pragma unroll
        for (int q = 0; q < n; ++q) v[q] = __ldg(F.p[F0 + q] + j);
#pragma unroll
        for (int q = 0; q < n; ++q) {
            g[q][0] = fma(wx, v[q], g[q][0]);
            g[q][1] = fma(wy, v[q], g[q][1]);
            g[q][2] = fma(wz, v[q], g[q][2]);
            const long long t = okey(v[q]);
            kmax[q] = (kmax[q] < t) ? t : kmax[q];
            kmin[q] = (t < kmin[q]) ? t : kmin[q];
        }
    }
    // boundary faces (face index >= ni) come last in the ascending list
    const int fe = cfp[i + 1];
    int kf = fe;
    while (kf > cfp[i] && (cfi[kf - 1] & kFaceMask) >= ni) --kf;
    for (; kf < fe; ++kf) {
        const int b = (cfi[kf] & kFaceMask) - ni;
        const double wx = bfw[b], wy = bfw[nb + b], wz = bfw[2 * (size_t)nb + b];
#pragma unroll
        for (int q = 0; q < n; ++q) {
            const double d = bf[(size_t)(F0 + q) * nb + b];
            g[q][0] = fma(wx, d, g[q][0]);
            g[q][1] = fma(wy, d, g[q][1]);
            g[q][2] = fma(wz, d, g[q][2]);
        }
    }
    const double sx = stws[i], sy = stws[N + i], sz = stws[2 * N + i];
    const double m0 = minv[i], m1 = minv[N + i], m2 = minv[2 * N + i];
    const double m3 = minv[3 * N + i], m4 = minv[4 * N + i], m5 = minv[5 * N + i];
#pragma unroll
    for (int q = 0; q < n; ++q) {
        const double a0 = fma(-phi[q], sx, g[q][0]);
        const double a1 = fma(-phi[q], sy, g[q][1]);
        const double a2 = fma(-phi[q], sz, g[q][2]);
        // limits: U, V, W, VF, P in that order
        const int f = F0 + q, at = f == 0 ? 8 : (f == 4 ? 6 : 2 * (f - 1));
        grad[(size_t)(3 * f) * N + i] = fma(m2, a2, fma(m1, a1, fma(m0, a0, 0.0)));
        grad[(size_t)(3 * f + 1) * N + i] = fma(m4, a2, fma(m3, a1, fma(m1, a0, 0.0)));
        grad[(size_t)(3 * f + 2) * N + i] = fma(m5, a2, fma(m4, a1, fma(m2, a0, 0.0)));
        mm[(size_t)at * N + i] = ounkey(kmax[q]);
        mm[(size_t)(at + 1) * N + i] = ounkey(kmin[q]);
    }
}

}  // namespace

namespace semo {

void lsq_gradients(semo_ctx* c, const double* const* f, const double* bf, double* grad, double* mm, bool uvw_only) {
    Fields5 F;
    for (int q = 0; q < 5; ++q) F.p[q] = f[q];
    auto launch = [&](auto kern) {
        kern<<<blocks(c->nc, 128), 128, 0, c->stream>>>(c->nc, c->ni, c->nb, c->st_ptr, c->st_idx, c->stw, c->cf_ptr,
                                                        c->cf_idx, c->bfw, c->stws, c->minv, F, bf, grad, mm);
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
