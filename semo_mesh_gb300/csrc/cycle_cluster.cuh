// The V-cycle's smallest levels in one block, and whole CG solves of small
// systems in a thread-block cluster (part of cycle.cu).
//
// A small level costs a launch a step whatever its size: ~2.75 us a kernel of
// the CG loop's graph at 14^3 cells (19 kernels, 52 us an iteration), with the
// multiprocessors nearly idle.
//   k_local_cycle     levels l0.. of the V-cycle from b to x by one block, the
//                     matrices (16-bit columns) and vectors in shared memory: a
//                     step is a block barrier and shared-memory reads.  What
//                     bounds it is one multiprocessor's shared memory, so it
//                     takes levels of up to kLocalNnz entries: with 13k entries
//                     (the third level at 47^3) it took as long as the six
//                     kernels, with 3k it took 3 % off an outer iteration at
//                     32^3.
//   k_cluster_cg      the whole preconditioned CG of cg_iteration, loop
//                     included, by 8 blocks: no graph is captured or
//                     instantiated (~95 us a solve) and the sums need no
//                     kernels of their own.  A block owns a run of a level's
//                     rows, whose matrices are in its shared memory; every
//                     vector that a step gathers from is kept whole in every
//                     block's shared memory, the owners copying their run into
//                     the other blocks (distributed shared memory, 16 bytes a
//                     store); the lowest levels every block cycles for itself.
//                     A step then reads nothing from L2 (with the vectors in
//                     global memory a step cost 3.2 us: the release to L2, the
//                     L1 that an acquire empties, two dependent round trips).
//                     What bounds it is latency (ncu at 14^3: of the 23 clocks
//                     between a warp's issues 10 at a barrier, 3 on shared memory); it takes what fits in shared
//                     memory (14^3 cells, not 32^3).
// A pressure pass at 14^3 cells: 1.56 -> 1.12 ms.
#pragma once

constexpr int kClBlocks = kClusterBlocks, kClThreads = 1024;
constexpr int kClLevels = 10;
constexpr int kClCoarse = 96;          // rows of the largest coarsest level
constexpr int kClSmem = 206 * 1024;    // dynamic shared memory at most
constexpr int64_t kLocalNnz = 8000;    // entries of k_local_cycle's largest level

template <class V>
struct ClMat {      // CSR rows in shared memory (16-bit columns) at byte offsets, 2^lg lanes a row; what they are loaded from
    int ptr, col, val, lg;
    const int *gptr, *gcol;
    const V* gval;
};
template <class V>
struct ClLevel {
    int n, ch;                  // rows, rows a block owns (a local level: all)
    ClMat<V> A, P, R;
    const V* dinv;
    V inv_theta, c1, c2;
    // byte offsets in shared memory: whole vectors t (the first iterate
    // D^-1 b / theta; own rows: d), x, r; own rows b, D^-1
    int t, x, r, b, d;
};
template <class V>
struct ClArgs {
    int nlev, coarse_n;
    int local;                  // first local level
    int smem, inv;              // bytes in all; the inverse's place
    const double* cinv;
    const V* b;                 // level 0's b and x in global memory
    V* xout;
    ClLevel<V> lev[kClLevels];
};
struct ClCg {                   // k_cluster_cg: the FP64 system
    ClMat<double> A;
    const double* b;
    double *x, *scal;
    double tol;
    int max_iter, own;          // own: place of the FP64 vectors of the owned rows
    bool zero_guess;
};

__device__ __forceinline__ void cl_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ unsigned cl_map(const void* p, int rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void cl_store(double* p, int rank, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(cl_map(p, rank)), "d"(v) : "memory");
}
// The block's run of a vector, [r0, r0 + cnt) of whole (in this block's shared
// memory and written by its threads), into the other blocks; then arrives at
// the cluster barrier.  Only the threads that stored release to the cluster: a
// release by all 1,024 made the barrier 600 clocks instead of 180.  A run
// starts on a 16-byte boundary (ch and the vectors' places are rounded so); the
// words past its end that its last 16 bytes cover belong to no row.
template <class V>
__device__ __forceinline__ void cl_share(V* whole, int r0, int cnt) {
    __syncthreads();
    const int quads = (cnt * (int)sizeof(V) + 15) / 16;
    bool stored = false;
    for (int w = threadIdx.x; w < quads * kClBlocks; w += kClThreads) {
        const int to = w / quads, q = w - to * quads;
        if (to == (int)blockIdx.x) continue;
        char* const at = reinterpret_cast<char*>(whole + r0) + 16 * q;
        const int4 v = *reinterpret_cast<const int4*>(at);
        asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(cl_map(at, to)), "r"(v.x), "r"(v.y),
                     "r"(v.z), "r"(v.w)
                     : "memory");
        stored = true;
    }
    if (stored) asm volatile("fence.acq_rel.cluster;" ::: "memory");
    __syncwarp();
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}

template <class V>
__device__ __forceinline__ int cl_first(const ClLevel<V>& L) { return min(L.n, (int)blockIdx.x * L.ch); }
template <class V>
__device__ __forceinline__ int cl_count(const ClLevel<V>& L) { return min(L.n, ((int)blockIdx.x + 1) * L.ch) - cl_first(L); }
template <class V>
__device__ __forceinline__ V* cl_at(char* sm, int off) { return reinterpret_cast<V*>(sm + off); }

// What stays in shared memory: the levels' matrices and D^-1 (of the owned
// rows of a shared level, of all rows of a local one) and the inverse.
template <class V>
__device__ void cl_load_rows(char* sm, const ClMat<V>& m, int r0, int rows) {
    int* const ptr = cl_at<int>(sm, m.ptr);
    unsigned short* const col = cl_at<unsigned short>(sm, m.col);
    V* const val = cl_at<V>(sm, m.val);
    const int k0 = __ldg(m.gptr + r0), nnz = __ldg(m.gptr + r0 + rows) - k0;
    for (int i = threadIdx.x; i <= rows; i += kClThreads) ptr[i] = __ldg(m.gptr + r0 + i) - k0;
#pragma unroll 4
    for (int k = threadIdx.x; k < nnz; k += kClThreads) {
        col[k] = (unsigned short)__ldg(m.gcol + k0 + k);
        val[k] = __ldg(m.gval + k0 + k);
    }
}
template <class V>
__device__ void cl_load(const ClArgs<V>& a, char* sm) {
    for (int l = 0; l + 1 < a.nlev; ++l) {
        const ClLevel<V>& L = a.lev[l];
        const bool local = l >= a.local;
        const int r0 = local ? 0 : cl_first(L), cnt = local ? L.n : cl_count(L);
        for (int i = threadIdx.x; i < cnt; i += kClThreads) cl_at<V>(sm, L.d)[i] = __ldg(L.dinv + r0 + i);
        cl_load_rows(sm, L.A, r0, cnt);
        cl_load_rows(sm, L.P, r0, cnt);
        const ClLevel<V>& C = a.lev[l + 1];   // R's rows
        cl_load_rows(sm, L.R, local ? 0 : cl_first(C), local ? C.n : cl_count(C));
    }
    for (int i = threadIdx.x; i < a.coarse_n * a.coarse_n; i += kClThreads) cl_at<double>(sm, a.inv)[i] = __ldg(a.cinv + i);
}

// f(row, (M x)_row) for a matrix's rows, by a row's first lane
template <class V, class X, class F>
__device__ __forceinline__ void cl_rows(char* sm, const ClMat<V>& M, int rows, const X& x, const F& f) {
    const int lg = M.lg, vs = 1 << lg, sub = threadIdx.x & (vs - 1), groups = kClThreads >> lg;
    const int mine = threadIdx.x >> lg, warp0 = (threadIdx.x & ~31) >> lg;   // the warp's first row: uniform trip count
    const int* const ptr = cl_at<int>(sm, M.ptr);
    const unsigned short* const col = cl_at<unsigned short>(sm, M.col);
    const V* const val = cl_at<V>(sm, M.val);
    for (int b = warp0; b < rows; b += groups) {
        const int row = b + (mine - warp0);
        V s = V(0);
        if (row < rows) {
            const int e = ptr[row + 1];
#pragma unroll 4
            for (int k = ptr[row] + sub; k < e; k += vs) s += val[k] * x(col[k]);
        }
        for (int o = vs >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (sub == 0 && row < rows) f(row, s);
    }
}

// The local levels' cycle, by a block for itself: from the whole b of the
// first local level to its whole x; begins and ends with a block barrier.
template <class V>
__device__ void cl_local(const ClArgs<V>& a, char* sm) {
    const int nl = a.nlev;
    __syncthreads();
    for (int l = a.local; l + 1 < nl; ++l) {
        const ClLevel<V>& L = a.lev[l];
        V *const t = cl_at<V>(sm, L.t), *const x = cl_at<V>(sm, L.x), *const r = cl_at<V>(sm, L.r);
        V *const b = cl_at<V>(sm, L.b), *const d = cl_at<V>(sm, L.d), *const cb = cl_at<V>(sm, a.lev[l + 1].b);
        for (int i = threadIdx.x; i < L.n; i += kClThreads) t[i] = d[i] * b[i] * L.inv_theta;
        __syncthreads();
        cl_rows(sm, L.A, L.n, [&](int j) { return t[j]; }, [&](int i, V s) {
            const V d0 = t[i];
            x[i] = d0 + L.c1 * d0 + L.c2 * (d[i] * (b[i] - s));
        });
        __syncthreads();
        cl_rows(sm, L.A, L.n, [&](int j) { return x[j]; }, [&](int i, V s) { r[i] = b[i] - s; });
        __syncthreads();
        cl_rows(sm, L.R, a.lev[l + 1].n, [&](int j) { return r[j]; }, [&](int i, V s) { cb[i] = s; });
        __syncthreads();
    }
    {   // coarsest level: the explicit FP64 inverse, 4 lanes a row
        const ClLevel<V>& L = a.lev[nl - 1];
        const int m = a.coarse_n, sub = threadIdx.x & 3, i = threadIdx.x >> 2;   // kClCoarse rows fit the block
        if ((threadIdx.x & ~31) < 4 * m) {   // whole warps
            const double* const inv = cl_at<double>(sm, a.inv) + (size_t)min(i, m - 1) * m;
            const V* const b = cl_at<V>(sm, L.b);
            double s = 0.0;
            for (int k = sub; k < m; k += 4) s += inv[k] * (double)b[k];
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            if (i < m && sub == 0) cl_at<V>(sm, L.x)[i] = (V)s;
        }
        __syncthreads();
    }
    for (int l = nl - 2; l >= a.local; --l) {
        const ClLevel<V>& L = a.lev[l];
        V *const t = cl_at<V>(sm, L.t), *const x = cl_at<V>(sm, L.x), *const r = cl_at<V>(sm, L.r);
        V *const b = cl_at<V>(sm, L.b), *const d = cl_at<V>(sm, L.d), *const cx = cl_at<V>(sm, a.lev[l + 1].x);
        cl_rows(sm, L.P, L.n, [&](int j) { return cx[j]; }, [&](int i, V s) { x[i] += s; });
        __syncthreads();
        cl_rows(sm, L.A, L.n, [&](int j) { return x[j]; }, [&](int i, V s) {
            const V dv = d[i] * (b[i] - s) * L.inv_theta;
            t[i] = dv;
            r[i] = x[i] + dv;
        });
        __syncthreads();
        cl_rows(sm, L.A, L.n, [&](int j) { return r[j]; },
                  [&](int i, V s) { x[i] = r[i] + L.c1 * t[i] + L.c2 * (d[i] * (b[i] - s)); });
        __syncthreads();
    }
}

// One V-cycle of the cluster's levels and the local ones below: level 0's t
// whole in every block and its b in the owner's.  last(local row, z) gets the
// result of the block's rows; nothing is synchronised after it.
template <class V, class Last>
__device__ void cl_vcycle(const ClArgs<V>& a, char* sm, const Last& last) {
    for (int l = 0; l < a.local; ++l) {
        const ClLevel<V>& L = a.lev[l];
        const ClLevel<V>& C = a.lev[l + 1];
        V *const t = cl_at<V>(sm, L.t), *const x = cl_at<V>(sm, L.x), *const r = cl_at<V>(sm, L.r);
        V *const b = cl_at<V>(sm, L.b), *const d = cl_at<V>(sm, L.d);
        const int r0 = cl_first(L), cnt = cl_count(L);
        cl_rows(sm, L.A, cnt, [&](int j) { return t[j]; }, [&](int i, V s) {
            const V d0 = t[r0 + i];
            x[r0 + i] = d0 + L.c1 * d0 + L.c2 * (d[i] * (b[i] - s));
        });
        cl_share(x, r0, cnt);
        cl_wait();
        cl_rows(sm, L.A, cnt, [&](int j) { return x[j]; }, [&](int i, V s) { r[r0 + i] = b[i] - s; });
        cl_share(r, r0, cnt);
        cl_wait();
        const int q0 = cl_first(C), qn = cl_count(C);
        const bool bottom = l + 1 == a.local;
        V *const ct = cl_at<V>(sm, C.t), *const cb = cl_at<V>(sm, C.b), *const cd = cl_at<V>(sm, C.d);
        cl_rows(sm, L.R, qn, [&](int j) { return r[j]; }, [&](int i, V s) {
            if (bottom) {
                cb[q0 + i] = s;   // a local level's b is whole
            } else {
                cb[i] = s;
                ct[q0 + i] = cd[i] * s * C.inv_theta;
            }
        });
        cl_share(bottom ? cb : ct, q0, qn);
        cl_wait();
    }
    cl_local(a, sm);
    for (int l = a.local - 1; l >= 0; --l) {
        const ClLevel<V>& L = a.lev[l];
        const ClLevel<V>& C = a.lev[l + 1];
        V *const t = cl_at<V>(sm, L.t), *const x = cl_at<V>(sm, L.x), *const r = cl_at<V>(sm, L.r);
        V *const b = cl_at<V>(sm, L.b), *const d = cl_at<V>(sm, L.d), *const cx = cl_at<V>(sm, C.x);
        const int r0 = cl_first(L), cnt = cl_count(L);
        if (l + 1 < a.local) {
            cl_share(cx, cl_first(C), cl_count(C));
            cl_wait();
        }
        cl_rows(sm, L.P, cnt, [&](int j) { return cx[j]; }, [&](int i, V s) { x[r0 + i] += s; });
        cl_share(x, r0, cnt);
        cl_wait();
        cl_rows(sm, L.A, cnt, [&](int j) { return x[j]; }, [&](int i, V s) {
            const V dv = d[i] * (b[i] - s) * L.inv_theta;
            t[r0 + i] = dv;
            r[r0 + i] = x[r0 + i] + dv;
        });
        cl_share(r, r0, cnt);
        cl_wait();
        cl_rows(sm, L.A, cnt, [&](int j) { return r[j]; }, [&](int i, V s) {
            const V z = r[r0 + i] + L.c1 * t[r0 + i] + L.c2 * (d[i] * (b[i] - s));
            if (l == 0) last(i, z);
            else x[r0 + i] = z;
        });
    }
}

template <class V>
__global__ void __launch_bounds__(kClThreads, 1) k_local_cycle(const __grid_constant__ ClArgs<V> a) {
    extern __shared__ double sm_cl[];
    char* const sm = reinterpret_cast<char*>(sm_cl);
    const ClLevel<V>& L = a.lev[0];
    cl_load(a, sm);   // what the setup wrote was there before the previous kernel
    pdl_enter();
    for (int i = threadIdx.x; i < L.n; i += kClThreads) cl_at<V>(sm, L.b)[i] = a.b[i];
    cl_local(a, sm);
    for (int i = threadIdx.x; i < L.n; i += kClThreads) a.xout[i] = cl_at<V>(sm, L.x)[i];
}

// Sums over the cluster of v (and w, with kTwo) of the first `threads` threads
// of every block: four warps a sum add them (a shuffle tree in every warp would
// be five FP64 instructions each, 64 clocks apiece on a warp's scheduler) and
// leave four partial sums a block in part[2][4 kClBlocks] of every block; after
// the next cluster barrier (that of a release by all threads, or cl_share's)
// cl_get adds them.  All threads call both; red: 2 kClThreads doubles.
template <bool kTwo>
__device__ __forceinline__ void cl_put(double v, double w, double* part, double* red, int threads) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x < threads) {
        red[threadIdx.x] = v;
        if (kTwo) red[kClThreads + threadIdx.x] = w;
    }
    __syncthreads();
    if (wid < (kTwo ? 8 : 4)) {
        const int which = wid >> 2, t0 = threadIdx.x & 127;
        double s = 0.0;
        for (int t = t0; t < threads; t += 128) s += red[which * kClThreads + t];
        s = __shfl_sync(0xffffffffu, warp_sum(s), 0);
        if (lane < kClBlocks) cl_store(part + (which * kClBlocks + blockIdx.x) * 4 + (wid & 3), lane, s);
        asm volatile("fence.acq_rel.cluster;" ::: "memory");
    }
}
// f(v, w) on the sums by one thread, which leaves what follows from them in
// shared memory for all (an FP64 division by all 1,024 threads takes some 5,000 clocks).
template <bool kTwo, class F>
__device__ __forceinline__ void cl_get(const double* part, const F& f) {
    static_assert(4 * kClBlocks == 32, "a partial sum a lane");
    if (threadIdx.x < 32) {
        const double v = warp_sum(part[threadIdx.x]);
        const double w = kTwo ? warp_sum(part[32 + threadIdx.x]) : 0.0;
        if (threadIdx.x == 0) f(v, w);
    }
    __syncthreads();
}

template <class V>
__global__ void __launch_bounds__(kClThreads, 1) k_cluster_cg(const __grid_constant__ ClArgs<V> a,
                                                              const __grid_constant__ ClCg g) {
    extern __shared__ double sm_cl[];
    __shared__ double red[2 * kClThreads], part[4][8 * kClBlocks];
    __shared__ struct { double b2, r2, stop, rz, pq, alpha, beta; int go, it, status; } sc;
    char* const sm = reinterpret_cast<char*>(sm_cl);
    const ClLevel<V>& L = a.lev[0];
    const int ch = L.ch, r0 = cl_first(L), cnt = cl_count(L);
    double *const r = cl_at<double>(sm, g.own), *const p = r + ch, *const q = p + ch, *const x = q + ch;   // own rows
    V *const t = cl_at<V>(sm, L.t), *const zx = cl_at<V>(sm, L.x), *const vb = cl_at<V>(sm, L.b);
    V* const vd = cl_at<V>(sm, L.d);
    const bool cycle = a.local > 0;   // else level 0 is the coarsest: every block has the whole b
    cl_arrive();
    cl_load(a, sm);
    cl_load_rows(sm, g.A, r0, cnt);
    // r = b - A x, 8 lanes a row: a row's products in the order of every other
    // FP64 residual of the library (a converged one is all cancellation)
    auto residual = [&](double& bb, double& rr) {
        ClMat<double> A8 = g.A;
        A8.lg = 3;
        cl_rows(sm, A8, cnt, [&](int j) { return g.x[j]; }, [&](int i, double s) {
            const double bi = g.b[r0 + i], ri = bi - s;
            r[i] = ri;
            bb += bi * bi;
            rr += ri * ri;
        });
    };
    double bb = 0.0, rr = 0.0;
    if (g.zero_guess) {
        for (int i = threadIdx.x; i < cnt; i += kClThreads) {
            const double bi = g.b[r0 + i];
            r[i] = bi;
            bb += bi * bi;
        }
        rr = bb;
    } else {
        __syncthreads();   // the matrix
        residual(bb, rr);
    }
    __syncthreads();
    cl_wait();
    // the residual in the V-cycle's type, and its first iterate (one level: b)
    auto to_cycle = [&](int i, double ri) {
        const V v = (V)ri;
        if (cycle) {
            vb[i] = v;
            t[r0 + i] = vd[i] * v * L.inv_theta;
        } else {
            vb[r0 + i] = v;
        }
    };
    V* const shared = cycle ? t : vb;
    for (int i = threadIdx.x; i < cnt; i += kClThreads) {
        to_cycle(i, r[i]);
        p[i] = 0.0;
        q[i] = 0.0;
        x[i] = g.zero_guess ? 0.0 : g.x[r0 + i];
    }
    cl_put<true>(bb, rr, part[0], red, kClThreads);
    cl_share(shared, r0, cnt);
    cl_wait();
    cl_get<true>(part[0], [&](double b2, double r2) {
        const double bn = sqrt(b2), bnorm = bn > 0.0 ? bn : 1.0;
        sc.b2 = b2;
        sc.r2 = r2;
        sc.stop = (g.tol * bnorm) * (g.tol * bnorm);
        sc.go = isfinite(bn) && isfinite(r2) && sqrt(r2) > g.tol * bnorm && g.max_iter > 0;
        sc.it = sc.status = 0;
    });
    while (sc.go) {
        double zr = 0.0, zq = 0.0, pq = 0.0, rr = 0.0;
        cl_vcycle(a, sm, [&](int i, V z) { zx[r0 + i] = z; });
        __syncthreads();
        if (threadIdx.x < cnt) {   // a thread a row (ch <= kClThreads)
            const double z = (double)zx[r0 + threadIdx.x];
            zr = z * r[threadIdx.x];
            zq = z * q[threadIdx.x];
        }
        cl_put<true>(zr, zq, part[1], red, cnt);
        cl_share(zx, r0, cnt);
        cl_wait();
        cl_get<true>(part[1], [&](double rz, double zqs) {
            // Polak-Ribiere: beta = z.(r_k - r_{k-1}) / (z_{k-1}.r_{k-1}) = -alpha_{k-1} z.q_{k-1} / rz_prev
            sc.beta = sc.it == 0 ? 0.0 : -sc.alpha * zqs / sc.rz;
            sc.rz = rz;
        });
        const double beta = sc.beta;
        cl_rows(sm, g.A, cnt, [&](int j) { return (double)zx[j]; }, [&](int i, double w) {
            const double qi = w + beta * q[i], pi = (double)zx[r0 + i] + beta * p[i];
            q[i] = qi;
            p[i] = pi;
            pq += pi * qi;
        });
        cl_put<false>(pq, 0.0, part[2], red, cnt);
        cl_arrive();
        cl_wait();
        cl_get<false>(part[2], [&](double s, double) {
            sc.pq = s;
            sc.alpha = sc.rz / s;
        });
        const double alpha = sc.alpha;
        for (int i = threadIdx.x; i < cnt; i += kClThreads) {
            x[i] += alpha * p[i];
            const double ri = r[i] - alpha * q[i];
            r[i] = ri;
            to_cycle(i, ri);
            rr += ri * ri;
        }
        cl_put<false>(rr, 0.0, part[3], red, cnt);
        cl_share(shared, r0, cnt);
        cl_wait();
        cl_get<false>(part[3], [&](double s, double) {
            ++sc.it;
            if (!isfinite(s) || !isfinite(sc.pq)) { sc.status = 1; sc.go = 0; }
            else if (!(sc.pq > 0.0)) { sc.status = 2; sc.go = 0; }
            else if (!(s > sc.stop) || sc.it >= g.max_iter) sc.go = 0;
        });
    }
    for (int i = threadIdx.x; i < cnt; i += kClThreads) g.x[r0 + i] = x[i];
    cl_arrive();
    cl_wait();
    // true FP64 residual of the returned solution
    bb = rr = 0.0;
    residual(bb, rr);
    cl_put<false>(rr, 0.0, part[0], red, kClThreads);
    cl_arrive();
    cl_wait();
    cl_get<false>(part[0], [&](double s, double) {
        if (blockIdx.x != 0) return;
        g.scal[11] = sc.b2;
        g.scal[12] = sc.r2;
        g.scal[13] = sc.it;
        g.scal[14] = sc.status;
        g.scal[16] = s;
    });
}

// --------------------------------------------------------------- host side
// Levels l0.. of h with those from `local` on cycled by every block for itself;
// false when they do not fit.  For k_cluster_cg g is the FP64 system (its
// pattern level l0's), whose place and that of its four vectors are set.
template <class V>
bool cl_layout(const Amg<V>& h, int l0, int local, ClArgs<V>& a, ClCg* g) {
    a.nlev = (int)h.lev.size() - l0;
    a.local = local;
    a.coarse_n = h.coarse_n;
    a.cinv = h.cinv.p;
    a.b = h.lev[l0].b.p;
    a.xout = h.lev[l0].x.p;
    int64_t off = 0;
    bool fits = true;
    auto take = [&](int64_t bytes) {
        const int64_t o = off;
        off += (bytes + 15) & ~(int64_t)15;
        fits &= off <= kClSmem;
        return fits ? (int)o : 0;
    };
    // rows of a matrix that a block holds: places and lanes a row (about four
    // entries a lane, more lanes while the block's threads outnumber its rows)
    auto place = [&](auto& m, int rows, int64_t nnz, int size) {
        m.lg = 0;
        while (m.lg < 5 && ((int64_t)rows << m.lg) < nnz &&
               ((rows << (m.lg + 1)) <= kClThreads || ((int64_t)4 * rows << m.lg) < nnz))
            ++m.lg;
        m.ptr = take(4ll * (rows + 1));
        m.col = take(2ll * nnz);
        m.val = take(size * nnz);
    };
    auto mat = [&](const DCsr<V>& M, bool in) {
        ClMat<V> m;
        m.gptr = M.ptr.p;
        m.gcol = M.col.p;
        m.gval = M.val.p;
        fits &= M.m <= 65536 && (in || M.run > 0);   // 16-bit columns; a shared level's runs are known
        place(m, in ? M.n : std::min(M.n, cluster_run(M.n)), in ? M.nnz : M.run, (int)sizeof(V));
        return m;
    };
    a.inv = take(8ll * a.coarse_n * a.coarse_n);
    for (int l = 0; l < a.nlev && fits; ++l) {
        const AmgLevel<V>& L = h.lev[l0 + l];
        ClLevel<V>& q = a.lev[l];
        const bool in = l >= local, last = l + 1 == a.nlev;
        q.n = L.A.n;
        q.ch = cluster_run(q.n);
        const int mine = in ? q.n : q.ch;
        q.x = take((q.n + 4) * (int64_t)sizeof(V));
        q.b = take((mine + 4) * (int64_t)sizeof(V));
        q.t = q.r = q.d = q.b;
        if (last) continue;
        q.t = take((q.n + 4) * (int64_t)sizeof(V));
        q.r = take((q.n + 4) * (int64_t)sizeof(V));
        q.d = take(mine * (int64_t)sizeof(V));
        q.dinv = L.dinv.p;
        const ChebCoef cc = cheb2(L.lam_max);
        q.inv_theta = (V)cc.inv_theta;
        q.c1 = (V)cc.c1;
        q.c2 = (V)cc.c2;
        q.A = mat(L.A, in);
        q.P = mat(L.P, in);
        q.R = mat(L.R, in);   // rows: the next level's
    }
    if (g && fits) {
        const DCsr<V>& A = h.lev[l0].A;
        fits &= A.run > 0;
        place(g->A, std::min(A.n, cluster_run(A.n)), A.run, (int)sizeof(double));
        g->A.lg = 0;   // a thread a row: shuffles in FP64 cost more than the products
        g->own = take(4ll * a.lev[0].ch * 8);
    }
    a.smem = (int)off;
    return fits;
}
// shared: the cluster shares level l0 (and as many below as do not fit as
// local ones); else all levels are local
template <class V>
bool cl_args(const Amg<V>& h, int l0, bool shared, ClArgs<V>& a, ClCg* g) {
    const int nl = (int)h.lev.size() - l0;
    if (nl < 1 || nl > kClLevels || h.coarse_n > kClCoarse) return false;
    if (!shared) return cl_layout(h, l0, 0, a, g);
    for (int local = 1; local < nl; ++local)
        if (cl_layout(h, l0, local, a, g)) return true;
    return false;
}

template <class K, class... A>
void launch_cluster(K* kern, cudaStream_t s, int blocks, int smem, bool pdl, const A&... args) {
    SEMO_CUDA(cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kClSmem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(kClThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    int n = 0;
    if (blocks > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = (unsigned)blocks;
        at[n].val.clusterDim.y = at[n].val.clusterDim.z = 1;
        ++n;
    }
    if (pdl) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    SEMO_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
    SEMO_CHECK_LAUNCH();
}
