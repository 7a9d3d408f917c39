// krylov_bodies.cuh -- per-tile bodies of the Krylov kernels.
//
// Each body works on one canonical tile `tc.tile` of a system with
// `tc.ntiles` tiles.  The single-system kernels (kernels_krylov.cu) pass the
// grid (tile = block, ntiles = grid size); the batched kernels
// (kernels_batch.cu) pass a (system, local tile) entry of their tile map, so a
// system's arithmetic -- row sums, reduction trees, scalar decisions -- is the
// same whether it is solved alone or inside a batch.
#pragma once
#include <cooperative_groups.h>

#include "dev_common.cuh"
#include "kernels.hpp"

namespace xcal {

template <class T>
__device__ __forceinline__ T row_dot(const CSRView& A, const T* __restrict__ nz, const T* __restrict__ x, int i) {
    // xmul! row (src/Multithread/spmvm.jl:47-53): sequential from 0.0
    T acc = T(0);
    const int rb = row_base(A, i), rl = A.len[i];
    for (int k = 0; k < rl; ++k) {
        int e = rb + SELL_C * k;
        acc = acc + ld_stream(nz + e) * x[ld_stream(A.colval + e)];
    }
    return acc;
}

// the same sum with the first 8 slots' loads issued together (wide tile
// kernels: two rows per thread and registers to spare)
template <class T>
__device__ __forceinline__ T row_dot8(const CSRView& A, const T* __restrict__ nz, const T* __restrict__ x, int i) {
    const int rb = row_base(A, i), rl = A.len[i];
    T v[8], xv[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (k < rl) {
            v[k] = ld_stream(nz + rb + SELL_C * k);
            xv[k] = x[ld_stream(A.colval + rb + SELL_C * k)];
        }
    T acc = T(0);
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (k < rl) acc = acc + v[k] * xv[k];
    for (int k = 8; k < rl; ++k) {
        const int e = rb + SELL_C * k;
        acc = acc + ld_stream(nz + e) * x[ld_stream(A.colval + e)];
    }
    return acc;
}
template <int NT, class T>
__device__ __forceinline__ T row_sum(const CSRView& A, const T* __restrict__ nz, const T* __restrict__ x, int i) {
    return NT > RED_THREADS ? row_dot8(A, nz, x, i) : row_dot(A, nz, x, i);
}

// The tile kernels run in two block sizes.  NT = RED_THREADS: thread t takes
// the tile's rows t + 256 k one after the other.  NT = WIDE_NT (launches of at
// most WIDE_TILES tiles, which leave the chip short of threads): two rows per
// thread, the rows' products through shared memory, threads 0..255 adding them
// in k order -- the same partials, bit for bit.  Measured on B200: residual of
// 27,025 rows 43 -> 12 us; CG SpMV, update and <r, z> of 116,440 rows together
// 58 -> 34 us per DILU-CG iteration; 16 batched cases' steps around the solves
// (95 tiles) 1.4 -> 0.9 ms per batch iteration.
constexpr int WIDE_NT = 1024;
constexpr int WIDE_TILES = 296;  // two per SM
__host__ __device__ constexpr int tile_min_blocks(int nt) { return nt > RED_THREADS ? 1 : 8; }

// f(i) for the rows i < n of the tile
template <class F>
__device__ __forceinline__ void tile_rows(const TileCtx& tc, int n, F&& f) {
    for (int l = threadIdx.x; l < RED_TILE; l += blockDim.x) {
        const int i = tc.tile * RED_TILE + l;
        if (i < n) f(i);
    }
}

template <int NT, int NV>
struct TileSmem {
    double pr[NT > RED_THREADS ? NV : 1][NT > RED_THREADS ? RED_TILE : 1];
    double sm[8];
};
// the tile's canonical partials of the NV products f(i, v) gives for each row,
// in tot of thread 0
template <int NT, int NV, class F>
__device__ __forceinline__ void tile_reduce(const TileCtx& tc, int n, TileSmem<NT, NV>& sh, double (&tot)[NV], F&& f) {
    double acc[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) acc[q] = 0.0;
    if constexpr (NT == RED_THREADS) {
        for (int k = 0; k < RED_ITEMS; ++k) {
            const int i = tile_row(tc, k);
            if (i < n) {
                double v[NV];
                f(i, v);
#pragma unroll
                for (int q = 0; q < NV; ++q) acc[q] = acc[q] + v[q];
            }
        }
    } else {
        // rows past n add 0.0, which leaves every partial sum as it is (they
        // start at +0.0 and are never -0.0)
#pragma unroll
        for (int j = 0; j < RED_TILE / NT; ++j) {
            const int l = j * NT + threadIdx.x, i = tc.tile * RED_TILE + l;
            double v[NV];
#pragma unroll
            for (int q = 0; q < NV; ++q) v[q] = 0.0;
            if (i < n) f(i, v);
#pragma unroll
            for (int q = 0; q < NV; ++q) sh.pr[q][l] = v[q];
        }
        __syncthreads();
        if (threadIdx.x < RED_THREADS)
#pragma unroll
            for (int k = 0; k < RED_ITEMS; ++k)
#pragma unroll
                for (int q = 0; q < NV; ++q) acc[q] = acc[q] + sh.pr[q][k * RED_THREADS + threadIdx.x];
    }
#pragma unroll
    for (int q = 0; q < NV; ++q) tot[q] = block_tree(acc[q], sh.sm);
}

// CG stopping decisions after gamma_next = <r,z> (Krylov.jl cg!)
__device__ __forceinline__ void cg_finalize(KScalars* S, double gamma_next) {
    double rNorm = sqrt(gamma_next);
    S->rNorm = rNorm;
    bool mach = (rNorm + 1.0 <= 1.0);
    bool solved = (rNorm <= S->eps) || mach;
    if (!solved) {
        double beta = gamma_next / S->gamma;
        S->pNorm2 = gamma_next + (beta * beta) * S->pNorm2;
        S->gamma = gamma_next;
        S->beta = beta;
    }
    S->iter = S->iter + 1;
    bool tired = S->iter >= S->itmax;
    if (solved) {
        S->done = 1;
        S->status = KS_SOLVED;
    } else if (tired) {
        S->done = 1;
        S->status = KS_TIRED;
    }
}

// Stopping tolerance at the start of a solve.  Plain mode: Krylov.jl's
// atol + rtol*||r0||.  Mixed mode (inner solve of a defect-correction
// step): the outer target atol + rtol*||r0|| is fixed by the first defect of
// the solve; an inner solve stops at the looser of that target and
// inner_rtol times its own initial norm, and a defect already below the
// target ends the outer loop.
__device__ __forceinline__ void start_eps(KScalars* S, double rNorm) {
    if (!S->mixed) {
        S->eps = S->atol + S->rtol * rNorm;
        return;
    }
    if (S->outer == 0) S->eps_outer = S->atol + S->rtol * rNorm;
    S->eps = fmax(S->eps_outer, S->inner_rtol * rNorm);
    S->outer_conv = rNorm <= S->eps_outer ? 1 : 0;
}

// CG direction buffers alternate: iteration k uses p_k = P[k & 1].  cg_start
// stores p_0 = z in P[0]; for k >= 1 the SpMV forms p_k = z + beta*p_{k-1}
// on the fly (Krylov.jl kaxpby!(n, 1, z, beta, p) -- the same expression for
// every reader, so gathered neighbours see bit-identical values) and the
// thread owning a row stores it.  The separate p-update pass disappears.
template <class T>
__device__ __forceinline__ T cg_dir(const T* __restrict__ z, const T* __restrict__ pold, T beta, int j) {
    return z[j] + beta * pold[j];
}

// q_i = sum_k nz[i,k] * d[col(i,k)] in slot order, d = p (first iteration) or
// z + beta p_old gathered on the fly: the first 8 slots' loads are issued
// together, the products are then added in slot order (wide forms only; the
// narrow forms keep the plain loop, which needs fewer registers).
template <class T, bool FIRST>
__device__ __forceinline__ T cg_row_q(const CSRView& A, const T* __restrict__ nz, const T* z, const T* pold,
                                      const T* pk, T b, int i) {
    const int rb = row_base(A, i), ln = A.len[i];
    T qi = T(0);
    int c[8];
    T v[8];
#pragma unroll
    for (int t = 0; t < 8; ++t)
        if (t < ln) {
            c[t] = ld_stream(A.colval + rb + SELL_C * t);
            v[t] = ld_stream(nz + rb + SELL_C * t);
        }
#pragma unroll
    for (int t = 0; t < 8; ++t)
        if (t < ln) qi = qi + v[t] * (FIRST ? pk[c[t]] : cg_dir(z, pold, b, c[t]));
    for (int t = 8; t < ln; ++t) {
        const int s = rb + SELL_C * t;
        const int cc = ld_stream(A.colval + s);
        qi = qi + ld_stream(nz + s) * (FIRST ? pk[cc] : cg_dir(z, pold, b, cc));
    }
    return qi;
}

template <class T, int NT>
__device__ __forceinline__ void spmv_body(const TileCtx& tc, CSRView A, const T* __restrict__ nz,
                                          const T* __restrict__ x, T* y, const KScalars* S) {
    if (S && S->done) return;
    tile_rows(tc, A.n, [&](int i) { y[i] = row_sum<NT>(A, nz, x, i); });
}

template <class T>
__device__ __forceinline__ void jacobi_apply_body(const TileCtx& tc, int n, const T* __restrict__ P, const T* __restrict__ r, T* z, const KScalars* S) {
    if (S && S->done) return;
    tile_rows(tc, n, [&](int i) { z[i] = P[i] * r[i]; });
}

template <class T>
__device__ __forceinline__ void copy_body(const TileCtx& tc, int n, const T* __restrict__ a, T* b, const KScalars* S) {
    if (S && S->done) return;
    tile_rows(tc, n, [&](int i) { b[i] = a[i]; });
}

// the start of a cg! solve from gamma = <r0, z0> (Krylov.jl cg!): norms,
// the stopping tolerance (start_eps), zero right-hand side, immediate stop
__device__ __forceinline__ void cg_start_scalars(KScalars* S, double gamma) {
    S->gamma = gamma;
    double rNorm = sqrt(gamma);
    S->rNorm = rNorm;
    S->rNorm0 = rNorm;
    S->iter = 0;
    S->done = 0;
    S->status = KS_RUNNING;
    S->outer_conv = 0;
    S->loops = 0;
    if (gamma == 0.0) {
        S->done = 1;
        S->status = KS_ZERO_RHS;
        S->outer_conv = 1;
        return;
    }
    S->pNorm2 = gamma;
    start_eps(S, rNorm);
    if (rNorm <= S->eps) {
        S->done = 1;
        S->status = KS_SOLVED;
    } else if (S->iter >= S->itmax) {
        S->done = 1;
        S->status = KS_TIRED;
    }
}

template <class T, int NT>
__device__ __forceinline__ void cg_start_body(const TileCtx& tc, int n, const T* __restrict__ r, const T* __restrict__ z, T* p, KScalars* S,
                           double* part, double* ring) {
    __shared__ TileSmem<NT, 1> sh;
    // the resident CG's exchange buffers start unset (cg_resident_body)
    if (ring)
        for (int k = threadIdx.x; k < 4 * tc.ntiles; k += blockDim.x)
            ring[((size_t)(k / tc.ntiles) * tc.ntiles + tc.tile) * tc.ntiles + k % tc.ntiles] =
                __longlong_as_double(-1LL);
    double tot[1];
    tile_reduce<NT, 1>(tc, n, sh, tot, [&](int i, double* v) {
        T zi = z[i];
        p[i] = zi;
        v[0] = (double)r[i] * (double)zi;
    });
    if (threadIdx.x == 0) part[tc.tile] = tot[0];
    if (!last_block(&S->counter, tc.ntiles)) return;
    double gamma = reduce_partials(part, tc.ntiles, sh.sm);
    if (threadIdx.x == 0) cg_start_scalars(S, gamma);
}

template <class T, int NT>
__device__ __forceinline__ void cg_spmv_body(const TileCtx& tc, CSRView A, const T* __restrict__ nz,
                                                         const T* __restrict__ z, T* P0, T* P1, T* q, KScalars* S,
                                                         double* part) {
    if (S->done) return;
    __shared__ TileSmem<NT, 1> sh;
    const int it = S->iter;
    const T beta = (T)S->beta;
    T* pk = (it & 1) ? P1 : P0;
    const T* pold = (it & 1) ? P0 : P1;
    double tot[1];
    tile_reduce<NT, 1>(tc, A.n, sh, tot, [&](int i, double* v) {
        T qi = T(0), pi;
        if constexpr (NT > RED_THREADS) {
            if (it == 0) {
                qi = cg_row_q<T, true>(A, nz, z, pold, pk, beta, i);
                pi = pk[i];
            } else {
                qi = cg_row_q<T, false>(A, nz, z, pold, pk, beta, i);
                pi = cg_dir(z, pold, beta, i);
                pk[i] = pi;
            }
        } else {
            const int rb = row_base(A, i), e1 = rb + SELL_C * A.len[i];
            if (it == 0) {
                for (int e = rb; e < e1; e += SELL_C) qi = qi + ld_stream(nz + e) * pk[ld_stream(A.colval + e)];
                pi = pk[i];
            } else {
                for (int e = rb; e < e1; e += SELL_C)
                    qi = qi + ld_stream(nz + e) * cg_dir(z, pold, beta, ld_stream(A.colval + e));
                pi = cg_dir(z, pold, beta, i);
                pk[i] = pi;
            }
        }
        q[i] = qi;
        v[0] = (double)pi * (double)qi;
    });
    if (threadIdx.x == 0) part[tc.tile] = tot[0];
    if (!last_block(&S->counter, tc.ntiles)) return;
    double pAp = reduce_partials(part, tc.ntiles, sh.sm);
    if (threadIdx.x == 0) {
        const double epsT = sizeof(T) == 8 ? 2.220446049250313e-16 : 1.1920928955078125e-07;  // eps(T)
        double lim = epsT * S->pNorm2;
        if (pAp <= lim && fabs(pAp) <= lim) {
            S->done = 1;
            S->status = KS_ZERO_CURV;
            return;
        }
        S->alpha = S->gamma / pAp;
    }
}

template <class T, int NT>
__device__ __forceinline__ void cg_update_body(const TileCtx& tc, int n, T* x, const T* __restrict__ P0, const T* __restrict__ P1, T* r,
                            const T* __restrict__ q, T* z, const T* __restrict__ P, int jacobi_fused, KScalars* S,
                            double* part) {
    if (S->done) return;
    __shared__ TileSmem<NT, 1> sh;
    double* sm = sh.sm;
    const T* p = (S->iter & 1) ? P1 : P0;
    const T alpha = (T)S->alpha;
    double acc = 0.0;
    if constexpr (sizeof(T) == 4 && NT == RED_THREADS) {
        // FP32: 4-byte elements leave too few bytes in flight per thread when
        // each row waits for its loads; issue all rows' loads first (same
        // arithmetic, same order of the sums).  Measured 18.4 -> 14.4 us on
        // 2M rows.
        if (jacobi_fused) {
            T xv[RED_ITEMS], pv[RED_ITEMS], rv[RED_ITEMS], qv[RED_ITEMS], Pv[RED_ITEMS];
#pragma unroll
            for (int k = 0; k < RED_ITEMS; ++k) {
                int i = tile_row(tc, k);
                if (i < n) {
                    xv[k] = ld_stream(x + i);
                    pv[k] = p[i];
                    rv[k] = r[i];
                    qv[k] = ld_stream(q + i);
                    Pv[k] = ld_stream(P + i);
                }
            }
#pragma unroll
            for (int k = 0; k < RED_ITEMS; ++k) {
                int i = tile_row(tc, k);
                if (i < n) {
                    __stcs(x + i, xv[k] + alpha * pv[k]);
                    T ri = rv[k] + (-alpha) * qv[k];
                    r[i] = ri;
                    T zi = Pv[k] * ri;
                    z[i] = zi;
                    acc = acc + (double)ri * (double)zi;
                }
            }
            double tot = block_tree(acc, sm);
            if (threadIdx.x == 0) part[tc.tile] = tot;
            if (!last_block(&S->counter, tc.ntiles)) return;
            double g = reduce_partials(part, tc.ntiles, sm);
            if (threadIdx.x == 0) cg_finalize(S, g);
            return;
        }
    }
    // x, q and P are not read again before the next update: evict-first keeps
    // L2 for z and p, which the next SpMV gathers
    auto row = [&](int i) {
        __stcs(x + i, ld_stream(x + i) + alpha * p[i]);
        T ri = r[i] + (-alpha) * ld_stream(q + i);
        r[i] = ri;
        return ri;
    };
    if (!jacobi_fused) {
        tile_rows(tc, n, [&](int i) { row(i); });
        return;
    }
    double tot[1];
    tile_reduce<NT, 1>(tc, n, sh, tot, [&](int i, double* v) {
        T ri = row(i);
        T zi = ld_stream(P + i) * ri;
        z[i] = zi;
        v[0] = (double)ri * (double)zi;
    });
    if (threadIdx.x == 0) part[tc.tile] = tot[0];
    if (!last_block(&S->counter, tc.ntiles)) return;
    double g = reduce_partials(part, tc.ntiles, sm);
    if (threadIdx.x == 0) cg_finalize(S, g);
}

template <class T, int NT>
__device__ __forceinline__ void cg_rz_body(const TileCtx& tc, int n, const T* __restrict__ r, const T* __restrict__ z, KScalars* S, double* part) {
    if (S->done) return;
    __shared__ TileSmem<NT, 1> sh;
    double tot[1];
    tile_reduce<NT, 1>(tc, n, sh, tot, [&](int i, double* v) { v[0] = (double)r[i] * (double)z[i]; });
    if (threadIdx.x == 0) part[tc.tile] = tot[0];
    if (!last_block(&S->counter, tc.ntiles)) return;
    double g = reduce_partials(part, tc.ntiles, sh.sm);
    if (threadIdx.x == 0) cg_finalize(S, g);
}

// BiCGSTAB's scalar decisions (Krylov.jl bicgstab!), taken by one thread once
// a reduction is complete.  The start, from ||r||^2 and <c, r>:
__device__ __forceinline__ void bicg_start_scalars(KScalars* S, double rr, double cr) {
    double rNorm = sqrt(rr);
    S->rNorm = rNorm;
    S->rNorm0 = rNorm;
    S->iter = 0;
    S->done = 0;
    S->status = KS_RUNNING;
    S->outer_conv = 0;
    S->loops = 0;
    if (rNorm == 0.0) {
        S->done = 1;
        S->status = KS_ZERO_RHS;
        S->outer_conv = 1;
        return;
    }
    start_eps(S, rNorm);
    S->next_rho = cr;
    if (cr == 0.0) {
        S->done = 1;
        S->status = KS_BREAKDOWN;
        return;
    }
    if (rNorm <= S->eps) {
        S->done = 1;
        S->status = KS_SOLVED;
    } else if (S->iter >= S->itmax) {
        S->done = 1;
        S->status = KS_TIRED;
    }
}
// alpha = rho / <c, v> (the iteration counter advances)
__device__ __forceinline__ void bicg_alpha_scalars(KScalars* S, double cv) {
    S->iter = S->iter + 1;
    S->rho = S->next_rho;
    S->cv = cv;
    S->alpha = S->rho / cv;
}
// beta and the stopping tests, from <c, r> and ||r||^2 of the new residual
__device__ __forceinline__ void bicg_xr_scalars(KScalars* S, double omega, double cr, double rr) {
    S->next_rho = cr;
    S->beta = (cr / S->rho) * (S->alpha / omega);
    double rNorm = sqrt(rr);
    S->rNorm = rNorm;
    bool mach = (rNorm + 1.0 <= 1.0);
    bool solved = (rNorm <= S->eps) || mach;
    bool tired = S->iter >= S->itmax;
    bool breakdown = (S->alpha == 0.0) || isnan(S->alpha);
    if (solved) {
        S->done = 1;
        S->status = KS_SOLVED;
    } else if (tired) {
        S->done = 1;
        S->status = KS_TIRED;
    } else if (breakdown) {
        S->done = 1;
        S->status = KS_BREAKDOWN;
    }
}
// the scaled residual (Solve_1_api.jl:441-464) from ||b - A x||^2 and ||b||^2
__device__ __forceinline__ void residual_scalars(KScalars* S, double sR, double sb, double* out) {
    double normb = sqrt(sb);
    double denom = normb > jl_eps(normb) ? normb : 1.0;
    double res = sqrt(sR) / denom;
    S->resid = res;
    S->normb = normb;
    if (out) *out = res;
}

template <class T, int NT>
__device__ __forceinline__ void bicg_start_body(const TileCtx& tc, int n, const T* __restrict__ c, const T* __restrict__ r, T* p, KScalars* S,
                             double* part0, double* part1) {
    __shared__ TileSmem<NT, 2> sh;
    double tot[2];
    tile_reduce<NT, 2>(tc, n, sh, tot, [&](int i, double* v) {
        T ri = r[i];
        p[i] = ri;
        v[0] = (double)ri * (double)ri;
        v[1] = (double)c[i] * (double)ri;
    });
    if (threadIdx.x == 0) {
        part0[tc.tile] = tot[0];
        part1[tc.tile] = tot[1];
    }
    if (!last_block(&S->counter, tc.ntiles)) return;
    double rr = reduce_partials(part0, tc.ntiles, sh.sm);
    double cr = reduce_partials(part1, tc.ntiles, sh.sm);
    if (threadIdx.x == 0) bicg_start_scalars(S, rr, cr);
}

template <class T, int NT>
__device__ __forceinline__ void bicg_alpha_body(const TileCtx& tc, int n, const T* __restrict__ c, const T* __restrict__ v, KScalars* S, double* part) {
    if (S->done) return;
    __shared__ TileSmem<NT, 1> sh;
    double tot[1];
    tile_reduce<NT, 1>(tc, n, sh, tot, [&](int i, double* o) { o[0] = (double)c[i] * (double)v[i]; });
    if (threadIdx.x == 0) part[tc.tile] = tot[0];
    if (!last_block(&S->counter, tc.ntiles)) return;
    double cv = reduce_partials(part, tc.ntiles, sh.sm);
    if (threadIdx.x == 0) bicg_alpha_scalars(S, cv);
}

template <class T>
__device__ __forceinline__ void bicg_s_body(const TileCtx& tc, int n, const T* __restrict__ r, const T* __restrict__ v, const T* __restrict__ p, T* s,
                         T* x, const KScalars* S) {
    if (S->done) return;
    const T alpha = (T)S->alpha;
    tile_rows(tc, n, [&](int i) {
        s[i] = r[i] + (-alpha) * v[i];
        x[i] = x[i] + alpha * p[i];
    });
}

template <class T, int NT>
__device__ __forceinline__ void bicg_omega_body(const TileCtx& tc, int n, const T* __restrict__ t, const T* __restrict__ s, KScalars* S, double* part0,
                             double* part1) {
    if (S->done) return;
    __shared__ TileSmem<NT, 2> sh;
    double tot[2];
    tile_reduce<NT, 2>(tc, n, sh, tot, [&](int i, double* v) {
        double ti = (double)t[i];
        v[0] = ti * (double)s[i];
        v[1] = ti * ti;
    });
    if (threadIdx.x == 0) {
        part0[tc.tile] = tot[0];
        part1[tc.tile] = tot[1];
    }
    if (!last_block(&S->counter, tc.ntiles)) return;
    double ts = reduce_partials(part0, tc.ntiles, sh.sm);
    double tt = reduce_partials(part1, tc.ntiles, sh.sm);
    if (threadIdx.x == 0) S->omega = ts / tt;
}

template <class T, int NT>
__device__ __forceinline__ void bicg_xr_body(const TileCtx& tc, int n, T* x, const T* __restrict__ s, const T* __restrict__ t, T* r,
                          const T* __restrict__ c, KScalars* S, double* part0, double* part1) {
    if (S->done) return;
    __shared__ TileSmem<NT, 2> sh;
    const double omega = S->omega;
    const T om = (T)omega;
    double tot[2];
    tile_reduce<NT, 2>(tc, n, sh, tot, [&](int i, double* v) {
        T si = s[i];
        x[i] = x[i] + om * si;
        T ri = si + (-om) * t[i];
        r[i] = ri;
        v[0] = (double)c[i] * (double)ri;
        v[1] = (double)ri * (double)ri;
    });
    if (threadIdx.x == 0) {
        part0[tc.tile] = tot[0];
        part1[tc.tile] = tot[1];
    }
    if (!last_block(&S->counter, tc.ntiles)) return;
    double cr = reduce_partials(part0, tc.ntiles, sh.sm);
    double rr = reduce_partials(part1, tc.ntiles, sh.sm);
    if (threadIdx.x == 0) bicg_xr_scalars(S, omega, cr, rr);
}

template <class T>
__device__ __forceinline__ void bicg_p_body(const TileCtx& tc, int n, const T* __restrict__ r, const T* __restrict__ v, T* p, const KScalars* S) {
    if (S->done) return;
    const T beta = (T)S->beta, omega = (T)S->omega;
    tile_rows(tc, n, [&](int i) { p[i] = r[i] + beta * (p[i] + (-omega) * v[i]); });
}

// residual (src/Solve/Solve_1_api.jl:441-464): ||b - A x|| / max(||b||, 1 if tiny)
template <int NT>
__device__ __forceinline__ void residual_body(const TileCtx& tc, const CSRView& A, const double* __restrict__ nz,
                                              const double* __restrict__ x, const double* __restrict__ b, KScalars* S,
                                              double* part0, double* part1, double* out) {
    __shared__ TileSmem<NT, 2> sh;
    double tot[2];
    tile_reduce<NT, 2>(tc, A.n, sh, tot, [&](int i, double* v) {
        double fx = row_sum<NT>(A, nz, x, i);
        double bi = b[i];
        double d = bi - fx;
        v[0] = d * d;
        v[1] = bi * bi;
    });
    if (threadIdx.x == 0) {
        part0[tc.tile] = tot[0];
        part1[tc.tile] = tot[1];
    }
    if (!last_block(&S->counter2, tc.ntiles)) return;
    double sR = reduce_partials(part0, tc.ntiles, sh.sm);
    double sb = reduce_partials(part1, tc.ntiles, sh.sm);
    if (threadIdx.x == 0) residual_scalars(S, sR, sb, out);
}

// A DILU application of a small system as one
// block: every level of the forward sweep, then of the backward sweep, with a
// block barrier between levels (rows of a level are independent).  It reads
// the level-ordered triangles (position k of level order: cnt[k] slots at
// slice[k/32] + k%32 + 32 j, coalesced across a warp) and, in the forward
// sweep, dinv = T(1)/D[col] per slot, so a row's loads do not wait on one
// another and no division sits on the sweep's critical path; ys is y
// itself or, when y fits, a shared-memory copy written back at the end.
// Per row the arithmetic is forward_substitution! / backward_substitution!
// (preconditioners_1_DILU.jl:84-114) in the row's own entry order:
//   forward  y_i = b_i - sum_j (a_ij y_j) (1/D_j)      (j < i)
//   backward x_i = (x_i - sum_j a_ij x_j) / D_i        (j > i)
constexpr int DILU_BLOCK_THREADS = 1024;

// One level of a sweep over level positions k0..k1.  FP32: each thread
// takes the rows k and k + blockDim.x together (all their slot loads issued
// before either row's sum), so a level wider than the block costs one
// dependent load chain per pair of rows, not per row; FP64 keeps one row at a
// time (two rows' registers spill at 1024 threads).  LOWER: forward
// substitution (y_i = b_i - sum (a_ij y_j) (1/D_j)); else backward (x_i =
// (x_i - sum a_ij x_j) / D_i).  The first U slots of a row sit in registers,
// the rest are read in a loop; each row's sum runs in its own entry order.
// (start, stride): the thread's first position and the stride between its
// positions -- the block (threadIdx.x, blockDim.x) for one-block sweeps, the
// grid for sweeps spread over every block (k_dilu_grid).
template <class T, bool LOWER>
__device__ __forceinline__ void dilu_level_s(const LevelView<T>& L, int k0, int k1, const T* __restrict__ D,
                                             const T* __restrict__ b, T* ys, int start, int stride) {
    constexpr int R = sizeof(T) == 4 ? 2 : 1;  // rows per thread per step
    constexpr int U = sizeof(T) == 4 ? 6 : 8;
    for (int k = k0 + start; k < k1; k += R * stride) {
        int kk[R];
#pragma unroll
        for (int r = 0; r < R; ++r) kk[r] = k + r * stride;
        int i[R], c[R], base[R];
        T rhs[R];
        int cj[R][U];
        T vj[R][U], dj[R][U];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            c[r] = 0;
            i[r] = 0;
            base[r] = 0;
            rhs[r] = T(0);
            if (kk[r] < k1) {
                i[r] = L.rows[kk[r]];
                c[r] = L.cnt[kk[r]];
                base[r] = L.slice[kk[r] / SELL_C] + (kk[r] % SELL_C);
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (kk[r] < k1) rhs[r] = LOWER ? b[i[r]] : D[i[r]];
#pragma unroll
            for (int j = 0; j < U; ++j)
                if (j < c[r]) {
                    const int e = base[r] + SELL_C * j;
                    cj[r][j] = ld_stream(L.col + e);
                    vj[r][j] = ld_stream(L.val + e);
                    if (LOWER) dj[r][j] = ld_stream(L.dinv + e);
                }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (kk[r] >= k1) continue;
            T sum = T(0);
#pragma unroll
            for (int j = 0; j < U; ++j)
                if (j < c[r]) sum = LOWER ? sum + (vj[r][j] * ys[cj[r][j]]) * dj[r][j] : sum + vj[r][j] * ys[cj[r][j]];
            for (int j = U; j < c[r]; ++j) {
                const int e = base[r] + SELL_C * j;
                sum = LOWER ? sum + (ld_stream(L.val + e) * ys[ld_stream(L.col + e)]) * ld_stream(L.dinv + e)
                            : sum + ld_stream(L.val + e) * ys[ld_stream(L.col + e)];
            }
            ys[i[r]] = LOWER ? rhs[r] - sum : (ys[i[r]] - sum) / rhs[r];
        }
    }
}

template <class T, bool LOWER>
__device__ __forceinline__ void dilu_level(const LevelView<T>& L, int k0, int k1, const T* __restrict__ D,
                                           const T* __restrict__ b, T* ys) {
    dilu_level_s<T, LOWER>(L, k0, k1, D, b, ys, (int)threadIdx.x, (int)blockDim.x);
}

template <class T>
__device__ __forceinline__ void dilu_level_sweep(int n, const LevelView<T>& lo, const LevelView<T>& up,
                                                 const T* __restrict__ D, const T* __restrict__ b, T* y, T* ys) {
    for (int l = 0; l < lo.nlev; ++l) {
        dilu_level<T, true>(lo, lo.off[l], lo.off[l + 1], D, b, ys);
        __syncthreads();
    }
    for (int l = 0; l < up.nlev; ++l) {
        dilu_level<T, false>(up, up.off[l], up.off[l + 1], D, b, ys);
        __syncthreads();
    }
    if (ys != y)
        for (int i = threadIdx.x; i < n; i += blockDim.x) y[i] = ys[i];
}

// ---- DILU sweeps as a dataflow over the level order ----
// A level barrier costs a launch or a grid barrier per level (about 4 us
// each, 11-40 levels per application) although a row needs only its own few
// neighbours.  Here every row waits for exactly the values it reads, and the
// value is its own flag: the result array starts as a bit pattern that no
// row ever stores (all ones, a NaN; a row whose result is NaN stores the
// canonical one), so one relaxed load both polls and fetches, with no fence
// and no flag array.  Rows are dealt out in level order, over co-resident
// blocks (cooperative launch) or by tickets, and a warp takes its rows in
// ascending position; a row's dependencies have smaller positions, so the
// first unfinished row always runs and nothing can wait in a circle.  Waits
// are bounded: after FLOW_SPIN_LIMIT polls *err is set and every block leaves.
// Each row's arithmetic is that of the level kernels, in the row's entry
// order, so the results are theirs bit for bit.  What bounds it: the chain of
// dependent L2 round trips, one per level (about 1.05 us), then DRAM.
// Measured on B200 per application, this against the fastest level form
// (FP64, 2 x 13..20 levels): 6,400 rows 27 / 43 us, 27,025 rows 37 / 88 us,
// 62,403 rows 45 / 123 us, 116,440 rows 48 / 119 us; FP32 262,144 rows
// 61 / 131 us, 884,736 rows 117 / 155 us.  At 2.1M rows the level order's
// scattered vector accesses cost more than its barriers (283 / 252 us), so
// the autotuner times both.
constexpr int FLOW_U = 6;  // slots per row held in registers (a hexahedral row has at most 6 in one triangle)
constexpr int FLOW_SPIN_LIMIT = 1 << 21;

__device__ __forceinline__ double ld_flow(const double* p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ float ld_flow(const float* p) {
    float v;
    asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ double ld_flow_acquire(const double* p) {
    double v;
    asm volatile("ld.acquire.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool flow_unset(double v) { return __double_as_longlong(v) == -1LL; }
__device__ __forceinline__ bool flow_unset(float v) { return __float_as_int(v) == -1; }
__device__ __forceinline__ void st_flow(double* p, double v) {
    if (isnan(v)) v = __longlong_as_double(0x7ff8000000000000LL);
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ void st_flow(float* p, float v) {
    if (isnan(v)) v = __int_as_float(0x7fc00000);
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}
template <class T>
__device__ __forceinline__ T flow_unset_value();
template <>
__device__ __forceinline__ double flow_unset_value<double>() { return __longlong_as_double(-1LL); }
template <>
__device__ __forceinline__ float flow_unset_value<float>() { return __int_as_float(-1); }

// whether a warp that has polled `spins` times stops waiting (the same answer
// in every lane): past the limit, or as another warp gave up
__device__ __forceinline__ bool flow_give_up(int spins, int spin_limit, int* err) {
    if (spins < spin_limit && (spins & 1023) != 1023) return false;
    if (!__any_sync(0xffffffffu, spins >= spin_limit || *(volatile int*)err)) return false;
    *(volatile int*)err = 1;
    return true;
}

// Polls the values ys[col] of one row's c slots (the first FLOW_U's columns
// in cj, values landing in yv) until all are set, then runs `finish` --
// inside the loop, so that a row another lane of the warp waits for is
// stored without the warp having to leave the loop together.  Every lane of
// the warp calls it (c < 0: no row).  false: gave up.
template <class T, class F>
__device__ __forceinline__ bool flow_wait(const T* ys, const int* __restrict__ col, int base, int c,
                                          const int (&cj)[FLOW_U], T (&yv)[FLOW_U], int* err, F&& finish,
                                          int spin_limit = FLOW_SPIN_LIMIT) {
    bool fin = c < 0;
#pragma unroll
    for (int j = 0; j < FLOW_U; ++j)
        if (j < c) yv[j] = ld_flow(ys + cj[j]);
    for (int spins = 0;; ++spins) {
        if (!fin) {
            bool ready = true;
#pragma unroll
            for (int j = 0; j < FLOW_U; ++j)
                if (j < c && flow_unset(yv[j])) ready = false;
            for (int j = FLOW_U; ready && j < c; ++j)
                ready = !flow_unset(ld_flow(ys + ld_stream(col + base + SELL_C * j)));
            if (ready) {
                finish();
                fin = true;
            }
        }
        if (__all_sync(0xffffffffu, fin)) return true;
        if (flow_give_up(spins, spin_limit, err)) return false;
        if (!fin) {
#pragma unroll
            for (int j = 0; j < FLOW_U; ++j)
                if (j < c && flow_unset(yv[j])) yv[j] = ld_flow(ys + cj[j]);
        }
    }
}

// a block's next chunk of work, drawn from a counter that only grows: chunks
// are handed out in order to blocks that run, so waiting on an earlier chunk
// always ends.  Called by every thread of the block; ok: whether the thread's
// last chunk went well.  Where one warp gave up the whole block gets no more
// work: a warp that left alone could be the one that draws, and the others
// would go on with its last ticket for good
constexpr int FLOW_NO_CHUNK = 0x7fffffff;
__device__ __forceinline__ int flow_ticket(unsigned int* ticket, int* sh, bool ok) {
    if (__syncthreads_or(!ok)) return FLOW_NO_CHUNK;
    if (threadIdx.x == 0) *sh = (int)atomicAdd(ticket, 1u);
    __syncthreads();
    return *sh;
}

// forward_substitution! (preconditioners_1_DILU.jl:84-98) of the warp's
// positions k0 .. k0 + 31 of the lower level order into y (unset before);
// marks out's rows unset for the backward rows
template <class T>
__device__ __forceinline__ bool flow_lower_rows(int n, const LevelView<T>& lo, const T* __restrict__ b, T* y, T* out,
                                                int k0, int* err, int spin_limit = FLOW_SPIN_LIMIT) {
    const int k = k0 + (threadIdx.x & 31);
    int i = 0, c = -1, base = 0;
    int cj[FLOW_U];
    T vj[FLOW_U], dj[FLOW_U], yv[FLOW_U];
    T rhs = T(0);
    if (k < n) {
        i = lo.rows[k];
        c = lo.cnt[k];
        base = lo.slice[k / SELL_C] + (k % SELL_C);
#pragma unroll
        for (int j = 0; j < FLOW_U; ++j)
            if (j < c) {
                const int e = base + SELL_C * j;
                cj[j] = ld_stream(lo.col + e);
                vj[j] = ld_stream(lo.val + e);
                dj[j] = ld_stream(lo.dinv + e);
            }
        rhs = b[i];
        out[i] = flow_unset_value<T>();
    }
    return flow_wait((const T*)y, lo.col, base, c, cj, yv, err, [&] {
        T sum = T(0);
#pragma unroll
        for (int j = 0; j < FLOW_U; ++j)
            if (j < c) sum = sum + (vj[j] * yv[j]) * dj[j];
        for (int j = FLOW_U; j < c; ++j) {
            const int e = base + SELL_C * j;
            sum = sum + (ld_stream(lo.val + e) * ld_flow(y + ld_stream(lo.col + e))) * ld_stream(lo.dinv + e);
        }
        st_flow(y + i, rhs - sum);
    }, spin_limit);
}

// backward_substitution! (preconditioners_1_DILU.jl:100-114) of the warp's
// positions of the upper level order into out (unset before, its forward
// values in y, which are marked unset again)
template <class T>
__device__ __forceinline__ bool flow_upper_rows(int n, const LevelView<T>& up, const T* __restrict__ D, T* y, T* out,
                                                int k0, int* err, int spin_limit = FLOW_SPIN_LIMIT) {
    const int k = k0 + (threadIdx.x & 31);
    int i = 0, c = -1, base = 0;
    int cj[FLOW_U];
    T vj[FLOW_U], yv[FLOW_U];
    T yi = T(0), Di = T(0);
    if (k < n) {
        i = up.rows[k];
        c = up.cnt[k];
        base = up.slice[k / SELL_C] + (k % SELL_C);
#pragma unroll
        for (int j = 0; j < FLOW_U; ++j)
            if (j < c) {
                const int e = base + SELL_C * j;
                cj[j] = ld_stream(up.col + e);
                vj[j] = ld_stream(up.val + e);
            }
        yi = ld_flow(y + i);
        Di = D[i];
        y[i] = flow_unset_value<T>();
    }
    return flow_wait((const T*)out, up.col, base, c, cj, yv, err, [&] {
        T sum = T(0);
#pragma unroll
        for (int j = 0; j < FLOW_U; ++j)
            if (j < c) sum = sum + vj[j] * yv[j];
        for (int j = FLOW_U; j < c; ++j) {
            const int e = base + SELL_C * j;
            sum = sum + ld_stream(up.val + e) * ld_flow((const T*)out + ld_stream(up.col + e));
        }
        st_flow(out + i, (yi - sum) / Di);
    }, spin_limit);
}

// update_dilu_diagonal! row i (preconditioners_1_DILU.jl:43-82)
__device__ __forceinline__ void dilu_D_row(const CSRView& A, const double* __restrict__ nz, double* D, int i) {
    int ds = A.diag[i];
    double d = nz[ds];
    for (int e = row_base(A, i); e < ds; e += SELL_C) {
        int j = A.colval[e];
        d = d - (nz[A.trans[e]] * nz[e]) / D[j];
    }
    D[i] = d;
}

// ---- persistent CG (Jacobi or no preconditioner) ----
// Grid-wide barrier among the nblocks co-resident blocks of one system.
// `count` only grows during a launch (zeroed before it): barrier number nb
// completes when it reaches (nb + 1) * nblocks, so there is no reset and no
// second atomic.  Thread 0 alone arrives, with a release reduction (the
// block's writes, ordered before it by __syncthreads, become visible with
// it), and polls with acquire loads; __syncthreads orders the rest of the
// block after it.  (Measured alone on B200: 1.6 us per barrier among 148
// blocks, against 2.0 us with full fences around a relaxed atomic.)  A
// single-block system needs no more than the __syncthreads.  Bounded: a
// block that polls more than BAR_SPIN_LIMIT times, or sees *err set by
// another block, returns false (and sets *err), so a failure ends every
// block within one bounded wait.
constexpr long BAR_SPIN_LIMIT = 1L << 22;
__device__ __forceinline__ void red_release_add(unsigned int* p, unsigned int v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool grid_barrier(unsigned int* count, int nblocks, unsigned int& nb, int* err,
                                             int* sh_err, long spin_limit = BAR_SPIN_LIMIT) {
    __syncthreads();
    if (nblocks == 1) return true;
    if (threadIdx.x == 0) {
        const unsigned int target = (nb + 1u) * (unsigned int)nblocks;
        red_release_add(count, 1u);
        long spins = 0;
        int e = 0;
        while ((int)(ld_acquire(count) - target) < 0) {
            if (++spins > spin_limit) {
                e = 1;
                *(volatile int*)err = 1;
                break;
            }
            if ((spins & 255) == 0 && *(volatile int*)err) {
                e = 1;
                break;
            }
            __nanosleep(32);
        }
        *sh_err = e;
    }
    ++nb;
    __syncthreads();
    return *sh_err == 0;
}

// Bulk prefetch of [p, p + bytes) into L2 (no data reaches the SM; p and
// bytes 16-byte multiples)
__device__ __forceinline__ void l2_prefetch(const void* p, unsigned bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// __launch_bounds__ minimum blocks per SM of each form: 64 registers for the
// wide forms, 32 for the narrow one (8 blocks of 256 threads per SM)
constexpr int persist_min_blocks(int nt) { return nt == 1024 ? 1 : nt == 512 ? 2 : 8; }

// The whole CG loop of Krylov.jl cg! (Jacobi-fused update) for one system,
// run by its ntiles blocks (block with tile t owns canonical tile t); per
// iteration
//   phase 1: p_k = z + beta p_{k-1} (gathered), q = A p_k for the tile's rows,
//            q kept in shared memory, p_k stored; tile partial of <p_k, q>;
//   barrier; every block reduces the partials (same tree) -> alpha, zero-
//            curvature test (identical decisions in every block);
//   phase 2: x += alpha p_k, r -= alpha q, z = P r; tile partial of <r, z>;
//   barrier; every block reduces -> cg! stopping tests, beta.
// The arithmetic is that of k_cg_spmv + k_cg_update; q never goes to HBM and
// the two kernel boundaries per iteration disappear.  The block of tile 0
// writes the scalar state back.  Runs at most max_iters iterations.  The
// barriers count only this system's blocks, so in a batched launch every
// system runs (and finishes) on its own.
//
// NT threads per block.  NT = RED_THREADS (narrow): thread t owns the tile's
// rows t + 256 k, k < 8, and accumulates its partial as it goes -- few
// registers, so 7-8 blocks fit an SM and a 2M-row system is co-resident.
// NT = 512 / 1024 (wide, for systems of at most 2 / 1 tiles per SM): thread
// t covers rows (t mod 256) + 256 k for NT/256 times fewer k, writes each
// row's product to shared memory, and threads 0..255 then add the products
// of "their" rows in k order -- the same partials, bit for bit, with a 4-8x
// shorter dependent-load chain per thread.
//
// Narrow form only: while a block waits at a barrier, the data its next
// phase streams is already being pulled into L2 -- x, r and P of its rows
// before the first barrier, and (pf_kb > 0, for matrices that fit L2) up to
// pf_kb KB of its matrix slots before the second.  Measured on B200 at 96^3
// / 128^3 (FP64): the vectors 5% / 1.7% faster; the matrix another 5% at
// 96^3 but 15% slower at 128^3 (it evicts the gathered vectors), hence the
// size condition.
// The canonical final tree over the tile partials of a system whose blocks
// form one thread-block cluster: thread t < T reads block t's partial from
// its shared memory (the values reduce_partials reads from global memory).
__device__ __forceinline__ double reduce_cluster(double* mine, int T, double* smem8) {
    double s = 0.0;
    if (threadIdx.x < RED_THREADS)
        for (int i = threadIdx.x; i < T; i += RED_THREADS)
            s = s + *cooperative_groups::this_cluster().map_shared_rank(mine, i);
    return block_tree(s, smem8);
}

// CL (cluster form, wide blocks only): the system's tiles are the blocks of
// one thread-block cluster (blocks past its tile count have no rows); the
// barriers are hardware cluster barriers (release / acquire at cluster
// scope) and the partials travel through distributed shared memory -- no
// global spin, no atomics, no cooperative launch (clusters are scheduled
// whole), and each cluster runs on its own.  Every block takes the same
// decisions, so all reach the same barriers; a last barrier keeps every
// block's shared memory alive until its peers have read it.
template <class T, int NT, bool CL = false>
__device__ __forceinline__ void cg_persist_body(const TileCtx& tc, const CSRView& A, const T* __restrict__ nz,
                                                const T* __restrict__ Pj, int jacobi, T* x, T* r, T* z, T* P0,
                                                T* P1, KScalars* S, double* part, double* part2, unsigned int* bar,
                                                int* err, int max_iters, int pf_kb) {
    constexpr bool WIDE = NT > RED_THREADS;
    static_assert(!CL || WIDE, "the cluster form uses wide blocks");
    __shared__ double cl_part[2];  // cluster form: this block's two tile partials
    constexpr int IPT = RED_ITEMS / (NT / RED_THREADS);  // rows per thread
    __shared__ T q_s[RED_TILE];
    __shared__ double pr_s[WIDE ? RED_TILE : 1];
    __shared__ double sm[8];
    __shared__ double sh_d[4];
    __shared__ int sh_i[3];
    __shared__ int sh_err;
    const int n = A.n;
    const int v = threadIdx.x & (RED_THREADS - 1), k0 = (threadIdx.x / RED_THREADS) * IPT;
    int iter = S->iter, done = S->done, status = S->status;
    const int itmax = S->itmax;
    double gamma = S->gamma, beta = S->beta, pNorm2 = S->pNorm2, alpha = S->alpha, rNorm = S->rNorm;
    const double eps = S->eps;
    const double epsT = sizeof(T) == 8 ? 2.220446049250313e-16 : 1.1920928955078125e-07;  // eps(T)
    int ran = 0;
    unsigned int nb = 0;
    bool ok = true;
    while (!done && ran < max_iters) {
        // phase 1: q = A p_k (k_cg_spmv)
        T* pk = (iter & 1) ? P1 : P0;
        const T* pold = (iter & 1) ? P0 : P1;
        const T b = (T)beta;
        double acc = 0.0;
        if constexpr (!WIDE) {
            for (int k = 0; k < RED_ITEMS; ++k) {
                int i = tile_row(tc, k);
                if (i < n) {
                    T qi = T(0), pi;
                    const int rb = row_base(A, i), e1 = rb + SELL_C * A.len[i];
                    if (iter == 0) {
                        for (int e = rb; e < e1; e += SELL_C)
                            qi = qi + ld_stream(nz + e) * pk[ld_stream(A.colval + e)];
                        pi = pk[i];
                    } else {
                        for (int e = rb; e < e1; e += SELL_C)
                            qi = qi + ld_stream(nz + e) * cg_dir(z, pold, b, ld_stream(A.colval + e));
                        pi = cg_dir(z, pold, b, i);
                        pk[i] = pi;
                    }
                    q_s[k * RED_THREADS + threadIdx.x] = qi;
                    acc = acc + (double)pi * (double)qi;
                }
            }
        } else {
            // rows past n contribute 0.0 to the k-ordered sums below: the
            // narrow form skips them, and x + 0.0 == x for every partial
            // sum that starts at +0.0 (it can never be -0.0)
#pragma unroll
            for (int j = 0; j < IPT; ++j) {
                const int k = k0 + j, i = tc.tile * RED_TILE + k * RED_THREADS + v;
                double prod = 0.0;
                if (i < n) {
                    T qi, pi;
                    if (iter == 0) {
                        qi = cg_row_q<T, true>(A, nz, z, pold, pk, b, i);
                        pi = pk[i];
                    } else {
                        qi = cg_row_q<T, false>(A, nz, z, pold, pk, b, i);
                        pi = cg_dir(z, pold, b, i);
                        pk[i] = pi;
                    }
                    q_s[k * RED_THREADS + v] = qi;
                    prod = (double)pi * (double)qi;
                }
                pr_s[k * RED_THREADS + v] = prod;
            }
            __syncthreads();
            if (threadIdx.x < RED_THREADS)
#pragma unroll
                for (int k = 0; k < RED_ITEMS; ++k) acc = acc + pr_s[k * RED_THREADS + v];
        }
        double tot = block_tree(acc, sm);
        if (threadIdx.x == 0) {
            if constexpr (CL)
                cl_part[0] = tot;
            else
                part[tc.tile] = tot;
        }
        if (!WIDE && threadIdx.x < 3 && (threadIdx.x < 2 || jacobi)) {
            const long r0 = (long)tc.tile * RED_TILE;
            const long nr = min((long)RED_TILE, (long)n - r0);
            const unsigned bytes = (unsigned)((nr * (long)sizeof(T)) & ~15L);
            const T* base = threadIdx.x == 0 ? x : threadIdx.x == 1 ? r : Pj;
            if (bytes) l2_prefetch(base + r0, bytes);
        }
        if constexpr (CL)
            cooperative_groups::this_cluster().sync();
        else if (!(ok = grid_barrier(bar, tc.ntiles, nb, err, &sh_err)))
            break;
        double pAp = CL ? reduce_cluster(&cl_part[0], tc.ntiles, sm) : reduce_partials(part, tc.ntiles, sm);
        if (threadIdx.x == 0) {
            double lim = epsT * pNorm2;
            sh_i[0] = (pAp <= lim && fabs(pAp) <= lim) ? 1 : 0;
            sh_d[0] = gamma / pAp;
        }
        __syncthreads();
        if (sh_i[0]) {
            done = 1;
            status = KS_ZERO_CURV;
            break;
        }
        alpha = sh_d[0];
        // phase 2: x, r, z and <r, z> (k_cg_update, Jacobi fused)
        const T a = (T)alpha;
        double acc2 = 0.0;
        if constexpr (!WIDE) {
            for (int k = 0; k < RED_ITEMS; ++k) {
                int i = tile_row(tc, k);
                if (i < n) {
                    __stcs(x + i, ld_stream(x + i) + a * pk[i]);
                    T ri = r[i] + (-a) * q_s[k * RED_THREADS + threadIdx.x];
                    r[i] = ri;
                    T zi = jacobi ? ld_stream(Pj + i) * ri : ri;
                    if (jacobi) z[i] = zi;
                    acc2 = acc2 + (double)ri * (double)zi;
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < IPT; ++j) {
                const int k = k0 + j, i = tc.tile * RED_TILE + k * RED_THREADS + v;
                double prod = 0.0;
                if (i < n) {
                    __stcs(x + i, ld_stream(x + i) + a * pk[i]);
                    T ri = r[i] + (-a) * q_s[k * RED_THREADS + v];
                    r[i] = ri;
                    T zi = jacobi ? ld_stream(Pj + i) * ri : ri;
                    if (jacobi) z[i] = zi;
                    prod = (double)ri * (double)zi;
                }
                pr_s[k * RED_THREADS + v] = prod;
            }
            __syncthreads();
            if (threadIdx.x < RED_THREADS)
#pragma unroll
                for (int k = 0; k < RED_ITEMS; ++k) acc2 = acc2 + pr_s[k * RED_THREADS + v];
        }
        double tot2 = block_tree(acc2, sm);
        if (threadIdx.x == 0) {
            if constexpr (CL)
                cl_part[1] = tot2;
            else
                part2[tc.tile] = tot2;
        }
        if (!WIDE && pf_kb > 0 && threadIdx.x < 32) {
            // the tile's slots are contiguous: slices s0 .. s1 (16 KB pieces;
            // lanes 0..15 the values, 16..31 the columns)
            const int s0 = tc.tile * (RED_TILE / SELL_C);
            const int s1 = min(s0 + RED_TILE / SELL_C, (n + SELL_C - 1) / SELL_C);
            const long e0 = A.slice[s0], e1 = A.slice[s1];
            const bool vals = threadIdx.x < 16;
            const char* p0 = vals ? (const char*)(nz + e0) : (const char*)(A.colval + e0);
            const long span = (e1 - e0) * (vals ? (long)sizeof(T) : 4L);
            const long lim = min(span, (long)pf_kb * (vals ? 1024L : 512L));
            for (long o = (threadIdx.x & 15) * 16384L; o < lim; o += 16 * 16384L) {
                const unsigned bytes = (unsigned)(min(16384L, lim - o) & ~15L);
                if (bytes) l2_prefetch(p0 + o, bytes);
            }
        }
        if constexpr (CL)
            cooperative_groups::this_cluster().sync();
        else if (!(ok = grid_barrier(bar, tc.ntiles, nb, err, &sh_err)))
            break;
        double g = CL ? reduce_cluster(&cl_part[1], tc.ntiles, sm) : reduce_partials(part2, tc.ntiles, sm);
        if (threadIdx.x == 0) {  // cg_finalize on the block's copy of the state
            double rn = sqrt(g);
            bool mach = (rn + 1.0 <= 1.0);
            bool solved = (rn <= eps) || mach;
            double bt = beta, pn = pNorm2, gm = gamma;
            if (!solved) {
                bt = g / gamma;
                pn = g + (bt * bt) * pNorm2;
                gm = g;
            }
            int it1 = iter + 1;
            int dn = 0, stt = status;
            if (solved) {
                dn = 1;
                stt = KS_SOLVED;
            } else if (it1 >= itmax) {
                dn = 1;
                stt = KS_TIRED;
            }
            sh_d[0] = rn;
            sh_d[1] = bt;
            sh_d[2] = pn;
            sh_d[3] = gm;
            sh_i[0] = it1;
            sh_i[1] = dn;
            sh_i[2] = stt;
        }
        __syncthreads();
        rNorm = sh_d[0];
        beta = sh_d[1];
        pNorm2 = sh_d[2];
        gamma = sh_d[3];
        iter = sh_i[0];
        done = sh_i[1];
        status = sh_i[2];
        ++ran;
    }
    if constexpr (CL) cooperative_groups::this_cluster().sync();
    if (ok && tc.tile == 0 && threadIdx.x == 0) {
        S->iter = iter;
        S->done = done;
        S->status = status;
        S->gamma = gamma;
        S->beta = beta;
        S->pNorm2 = pNorm2;
        S->alpha = alpha;
        S->rNorm = rNorm;
    }
}

// The same CG loop with one block per SM, each block owning the canonical
// tiles t = blockIdx.x, blockIdx.x + G, ... (G blocks): per tile and phase it
// runs the wide form's rows (NT / 256 row groups per tile, the rows'
// products in k order by threads 0..255) and writes the tile's partial, so
// the partials -- and every value -- are those of one block per tile, bit
// for bit.  Only G blocks meet at each grid barrier (148 instead of one per
// 2048-row tile), and each thread issues a row's slot loads together.  q of
// all the block's tiles stays in shared memory (dynamic, tpb tiles).
template <class T, int NT>
__device__ __forceinline__ void cg_persist_mt_body(const CSRView& A, const T* __restrict__ nz,
                                                   const T* __restrict__ Pj, int jacobi, T* x, T* r, T* z, T* P0,
                                                   T* P1, KScalars* S, double* part, double* part2,
                                                   unsigned int* bar, int* err, int max_iters, T* q_s) {
    static_assert(NT > RED_THREADS, "one block covers a tile's rows in NT / 256 groups");
    constexpr int IPT = RED_ITEMS / (NT / RED_THREADS);  // rows per thread and tile
    __shared__ double pr_s[RED_TILE];
    __shared__ double sm[8];
    __shared__ double sh_d[4];
    __shared__ int sh_i[3];
    __shared__ int sh_err;
    const int n = A.n;
    const int ntiles = (n + RED_TILE - 1) / RED_TILE;
    const int G = gridDim.x;
    const int v = threadIdx.x & (RED_THREADS - 1), k0 = (threadIdx.x / RED_THREADS) * IPT;
    int iter = S->iter, done = S->done, status = S->status;
    const int itmax = S->itmax;
    double gamma = S->gamma, beta = S->beta, pNorm2 = S->pNorm2, alpha = S->alpha, rNorm = S->rNorm;
    const double eps = S->eps;
    const double epsT = sizeof(T) == 8 ? 2.220446049250313e-16 : 1.1920928955078125e-07;  // eps(T)
    int ran = 0;
    unsigned int nb = 0;
    bool ok = true;
    while (!done && ran < max_iters) {
        T* pk = (iter & 1) ? P1 : P0;
        const T* pold = (iter & 1) ? P0 : P1;
        const T b = (T)beta;
        // phase 1, tile by tile: q = A p_k into q_s, the tile's <p_k, q>
        for (int t = blockIdx.x, j = 0; t < ntiles; t += G, ++j) {
#pragma unroll
            for (int u = 0; u < IPT; ++u) {
                const int k = k0 + u, i = t * RED_TILE + k * RED_THREADS + v;
                double prod = 0.0;
                if (i < n) {
                    T qi, pi;
                    if (iter == 0) {
                        qi = cg_row_q<T, true>(A, nz, z, pold, pk, b, i);
                        pi = pk[i];
                    } else {
                        qi = cg_row_q<T, false>(A, nz, z, pold, pk, b, i);
                        pi = cg_dir(z, pold, b, i);
                        pk[i] = pi;
                    }
                    q_s[j * RED_TILE + k * RED_THREADS + v] = qi;
                    prod = (double)pi * (double)qi;
                }
                pr_s[k * RED_THREADS + v] = prod;
            }
            __syncthreads();
            double acc = 0.0;
            if (threadIdx.x < RED_THREADS)
#pragma unroll
                for (int k = 0; k < RED_ITEMS; ++k) acc = acc + pr_s[k * RED_THREADS + v];
            const double tot = block_tree(acc, sm);  // its barriers also free pr_s for the next tile
            if (threadIdx.x == 0) part[t] = tot;
        }
        if (!(ok = grid_barrier(bar, G, nb, err, &sh_err))) break;
        const double pAp = reduce_partials(part, ntiles, sm);
        if (threadIdx.x == 0) {
            const double lim = epsT * pNorm2;
            sh_i[0] = (pAp <= lim && fabs(pAp) <= lim) ? 1 : 0;
            sh_d[0] = gamma / pAp;
        }
        __syncthreads();
        if (sh_i[0]) {
            done = 1;
            status = KS_ZERO_CURV;
            break;
        }
        alpha = sh_d[0];
        // phase 2, tile by tile: x, r, z and the tile's <r, z>
        const T a = (T)alpha;
        for (int t = blockIdx.x, j = 0; t < ntiles; t += G, ++j) {
#pragma unroll
            for (int u = 0; u < IPT; ++u) {
                const int k = k0 + u, i = t * RED_TILE + k * RED_THREADS + v;
                double prod = 0.0;
                if (i < n) {
                    __stcs(x + i, ld_stream(x + i) + a * pk[i]);
                    T ri = r[i] + (-a) * q_s[j * RED_TILE + k * RED_THREADS + v];
                    r[i] = ri;
                    T zi = jacobi ? ld_stream(Pj + i) * ri : ri;
                    if (jacobi) z[i] = zi;
                    prod = (double)ri * (double)zi;
                }
                pr_s[k * RED_THREADS + v] = prod;
            }
            __syncthreads();
            double acc2 = 0.0;
            if (threadIdx.x < RED_THREADS)
#pragma unroll
                for (int k = 0; k < RED_ITEMS; ++k) acc2 = acc2 + pr_s[k * RED_THREADS + v];
            const double tot2 = block_tree(acc2, sm);
            if (threadIdx.x == 0) part2[t] = tot2;
        }
        if (!(ok = grid_barrier(bar, G, nb, err, &sh_err))) break;
        const double g = reduce_partials(part2, ntiles, sm);
        if (threadIdx.x == 0) {  // cg_finalize on the block's copy of the state
            const double rn = sqrt(g);
            const bool solved = (rn <= eps) || (rn + 1.0 <= 1.0);
            double bt = beta, pn = pNorm2, gm = gamma;
            if (!solved) {
                bt = g / gamma;
                pn = g + (bt * bt) * pNorm2;
                gm = g;
            }
            const int it1 = iter + 1;
            int dn = 0, stt = status;
            if (solved) {
                dn = 1;
                stt = KS_SOLVED;
            } else if (it1 >= itmax) {
                dn = 1;
                stt = KS_TIRED;
            }
            sh_d[0] = rn;
            sh_d[1] = bt;
            sh_d[2] = pn;
            sh_d[3] = gm;
            sh_i[0] = it1;
            sh_i[1] = dn;
            sh_i[2] = stt;
        }
        __syncthreads();
        rNorm = sh_d[0];
        beta = sh_d[1];
        pNorm2 = sh_d[2];
        gamma = sh_d[3];
        iter = sh_i[0];
        done = sh_i[1];
        status = sh_i[2];
        ++ran;
    }
    if (ok && blockIdx.x == 0 && threadIdx.x == 0) {
        S->iter = iter;
        S->done = done;
        S->status = status;
        S->gamma = gamma;
        S->beta = beta;
        S->pNorm2 = pNorm2;
        S->alpha = alpha;
        S->rNorm = rNorm;
    }
}

// ---- persistent CG with the matrix resident in shared memory ----
// For systems of at most one canonical tile per SM.  The block of tile t
// keeps the tile's slots (values, and columns as 16-bit local indices) in
// shared memory for the whole solve, z of its rows and halo beside them, and x,
// r, p, q of its rows in registers (1024 threads, two rows each), so an
// iteration touches L2 only for the values other tiles own: the tile's halo,
// one entry per slot whose column lies outside it (and in a cluster not even
// for those).  Per iteration
//   each thread forms p_k = z + beta p_{k-1} for its rows and its halo
//   entries once (not once per slot), into shared memory;
//   q = A p_k from shared memory; <p_k, q>;
//   x += alpha p_k, r -= alpha q, z = P r; z published; <r, z>.
// (A halo entry's p_{k-1} is what this thread formed for it in the last
// iteration, so p is never published.)  The two reductions are also the
// iteration's only synchronisation: a block writes its tile partial into its
// column of every block's row of a buffer whose entries start unset
// (flow_unset), and polls its own row -- one store-to-load latency where the
// barrier forms paid an arrival, a poll and a second read, and no line that
// every block polls (one shared row measured 1.5-3 us more per reduction at
// 14-64 tiles).  Each reduction alternates between two buffers.  A block
// leaves its row unset as it reads it; an entry is written again two
// iterations later, by a block that has acquired this one's <r, z> in between,
// whose release covers the reset and z.  <p, q> needs no release: its block has
// written nothing since but its own rows' resets, and whoever overwrites the z
// it read depends on the partial those reads went into.  Arithmetic and
// reduction trees are cg_persist_body's, so the results are the same bit for
// bit.  Waits are bounded as in grid_barrier.
//
// What bounds it: shared-memory bandwidth of the slots (2048 rows x 7 slots x
// 18 bytes and their bank conflicts, 1.2 us FP32, 2.4 us FP64) and the two
// exchanges (1.2-1.5 us each in a cluster, 2.5-3.5 us through L2).  Measured
// on B200, us per iteration over whole solves, loading the matrix included,
// this against the forms without it in shared memory: FP64 1,073 rows 3.5 / 8.3,
// 7,500 rows 6.6 / 11.7, 27,025 rows 7.0 / 12.1, 129,150 rows 9.2 / 15.1; FP32 3.1 /
// 7.4, 4.7 / 9.3, 5.0 / 9.3, 7.5 / 11.5.
constexpr int RES_THREADS = 1024;
constexpr int RES_ROWS = RED_TILE / RES_THREADS;  // rows per thread
constexpr int RES_HALO_PT = 4;                    // halo entries per thread
constexpr int RES_HALO_MAX = RES_HALO_PT * RES_THREADS;
constexpr int RES_SMEM_MAX = 226 * 1024;
template <class T>
__host__ __device__ constexpr size_t res_smem_bytes(int slots, int halo) {
    // products (double per row), z of rows and halo, directions of both, values, local columns
    return RED_TILE * sizeof(double) + 2 * (((size_t)(RED_TILE + halo) * sizeof(T) + 15) / 16 * 16) +
           ((size_t)slots * sizeof(T) + 15) / 16 * 16 + (size_t)slots * sizeof(unsigned short);
}

struct ResState {
    double gamma, beta, pNorm2, alpha, rNorm;
    int iter, done, status, stop;
};

// the tile's sum of the products in pr (cg_persist_body's order: thread v <
// 256 adds rows v + 256 k in k order, then block_tree), in every lane of warp
// 0; called by the whole block after the products are visible
__device__ __forceinline__ double res_tile_sum(const double* pr, double* sm8) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < RED_THREADS) {
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < RED_ITEMS; ++k) acc = acc + pr[k * RED_THREADS + threadIdx.x];
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) acc = acc + __shfl_xor_sync(0xffffffffu, acc, off);
        if (lane == 0) sm8[warp] = acc;
        asm volatile("bar.sync 1, 256;" ::: "memory");
    }
    if (warp != 0) return 0.0;
    return ((sm8[0] + sm8[4]) + (sm8[2] + sm8[6])) + ((sm8[1] + sm8[5]) + (sm8[3] + sm8[7]));
}

// reduce_partials over the ntiles <= 256 tiles, by warp 0 of every block: tot
// is this block's partial, written into its column of every block's row of
// buf; the block polls its own row and leaves it unset again (release: with
// everything the block wrote before).  false: gave up.
__device__ __forceinline__ bool res_exchange(double tot, const TileCtx& tc, double* buf, bool release, int* err,
                                             double& sum, int spin_limit) {
    const int T = tc.ntiles, lane = threadIdx.x & 31;
    if (T == 1) {
        sum = 0.0 + tot;
        return true;
    }
    if (release) __threadfence();
    for (int t = lane; t < T; t += 32) st_flow(buf + (size_t)t * T + tc.tile, tot);
    double* row = buf + (size_t)tc.tile * T;
    // every entry in flight at once; acquire loads only where data was
    // released (they cost 0.1-1 us more per exchange)
    double w[8];
    bool ok = true;
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = 32 * j + lane < T ? flow_unset_value<double>() : 0.0;
    for (int spins = 0;; ++spins) {
        bool all = true;
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (flow_unset(w[j])) w[j] = release ? ld_flow_acquire(row + 32 * j + lane) : ld_flow(row + 32 * j + lane);
#pragma unroll
        for (int j = 0; j < 8; ++j) all = all && !flow_unset(w[j]);
        if (__all_sync(0xffffffffu, all)) break;
        if (flow_give_up(spins, spin_limit, err)) {
            ok = false;
            break;
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if (32 * j + lane < T) {
            row[32 * j + lane] = flow_unset_value<double>();
            w[j] = 0.0 + w[j];
        }
    if (!ok) return false;
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1)
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (32 * j < T) w[j] = w[j] + __shfl_xor_sync(0xffffffffu, w[j], off);
    sum = ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
    return true;
}

// the same among the blocks of one cluster (ntiles <= 16): the partial goes
// into every block's shared memory (mine[0 .. ntiles) of each), a hardware
// cluster barrier makes it and the blocks' z visible.  Called by every thread;
// the sum is valid in warp 0.
__device__ __forceinline__ double res_exchange_cl(double tot, const TileCtx& tc, double* mine) {
    if (tc.ntiles == 1) return 0.0 + tot;
    if (threadIdx.x < tc.ntiles)
        *cooperative_groups::this_cluster().map_shared_rank(mine + tc.tile, threadIdx.x) = tot;
    cooperative_groups::this_cluster().sync();
    double w = 0.0;
    if (threadIdx.x < 32) {
        w = threadIdx.x < tc.ntiles ? 0.0 + mine[threadIdx.x] : 0.0;
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) w = w + __shfl_xor_sync(0xffffffffu, w, off);
    }
    return w + 0.0;  // block_tree's other seven warps hold zeros
}

// CL: the system's tiles are the blocks of one thread-block cluster; z and the
// partials travel through distributed shared memory, with no trip to L2 in an
// iteration.  The owner of a row writes its z into the halo entries that read
// it (27,025 rows, long solves: 6.6 us per iteration; 7.7 us when the entries
// were read from their owners at the start of the next iteration).  The same through L2,
// with a tag beside each z, measured slower than a coalesced z array behind
// the <r, z> exchange's release (62,403 rows: 19.4 against 18.5 ms per pass).
template <class T, bool CL>
__device__ __forceinline__ void cg_resident_body(const TileCtx& tc, const CSRView& A, const T* __restrict__ nz,
                                                 const T* __restrict__ Pj, int jacobi, T* x, const T* r, T* z, const T* pg,
                                                 KScalars* S, double* ring, int* err, int max_iters, int slots,
                                                 int halo, unsigned char* smem,
                                                 int spin_limit = FLOW_SPIN_LIMIT) {
    __shared__ double sm8[8];
    __shared__ ResState st;
    double* pr = reinterpret_cast<double*>(smem);
    T* z_s = reinterpret_cast<T*>(smem + RED_TILE * sizeof(double));
    T* dir = reinterpret_cast<T*>((unsigned char*)z_s + ((size_t)(RED_TILE + halo) * sizeof(T) + 15) / 16 * 16);
    __shared__ double cl_part[2][16];
    T* val = reinterpret_cast<T*>((unsigned char*)dir + ((size_t)(RED_TILE + halo) * sizeof(T) + 15) / 16 * 16);
    unsigned short* idx =
        reinterpret_cast<unsigned short*>((unsigned char*)val + ((size_t)slots * sizeof(T) + 15) / 16 * 16);
    const int n = A.n, row0 = tc.tile * RED_TILE, e0 = A.slice[row0 / SELL_C];
    if (threadIdx.x == 0) {
        st = ResState{S->gamma, S->beta, S->pNorm2, S->alpha, S->rNorm, S->iter, S->done, S->status, 0};
    }
    __syncthreads();
    if (st.done) return;  // the same in every block
    const int itmax = S->itmax;
    const double eps = S->eps;
    const double epsT = sizeof(T) == 8 ? 2.220446049250313e-16 : 1.1920928955078125e-07;  // eps(T)
    const int h0 = tc.ntiles > 1 ? A.hoff[tc.tile] : 0, nh = tc.ntiles > 1 ? A.hoff[tc.tile + 1] - h0 : 0;
    // the tile's slots and this thread's rows; the halo entries' first
    // directions, p_0, straight into dir, their columns into pr (as ints)
    int* hcol = reinterpret_cast<int*>(pr);
    int lb[RES_ROWS], ln[RES_ROWS];
    T xi[RES_ROWS], ri[RES_ROWS], Pi[RES_ROWS], pi[RES_ROWS], qi[RES_ROWS];
#pragma unroll
    for (int j = 0; j < RES_ROWS; ++j) {
        const int i = row0 + j * RES_THREADS + threadIdx.x;
        lb[j] = ln[j] = 0;
        xi[j] = ri[j] = pi[j] = qi[j] = T(0);
        Pi[j] = T(1);
        if (i < n) {
            const int b = row_base(A, i);
            lb[j] = b - e0;
            ln[j] = A.len[i];
            int h = A.rowh[i];
            for (int t = 0; t < ln[j]; ++t) {
                const int c = ld_stream(A.colval + b + SELL_C * t);
                int li = c - row0;
                if (li < 0 || li >= RED_TILE) {
                    hcol[h] = c;
                    li = RED_TILE + h++;
                    dir[li] = __ldcg(pg + c);
                }
                idx[lb[j] + SELL_C * t] = (unsigned short)li;
                val[lb[j] + SELL_C * t] = ld_stream(nz + b + SELL_C * t);
            }
            xi[j] = x[i];
            ri[j] = r[i];
            pi[j] = pg[i];
            if (jacobi) Pi[j] = Pj[i];
        }
    }
    __syncthreads();
    // this thread's halo entries.  CL: where each one's z goes (the row whose z
    // it takes, the rank and entry it is written to); else the column it reads
    int hto[RES_HALO_PT], hrow[RES_HALO_PT];
#pragma unroll
    for (int u = 0; u < RES_HALO_PT; ++u) {
        const int h = u * RES_THREADS + threadIdx.x;
        hto[u] = -1;
        hrow[u] = 0;
        if (h < nh) {
            if constexpr (CL) {
                const int g = A.hdst[h0 + h];
                int k = 0;
                while (g >= A.hoff[k + 1]) ++k;
                hto[u] = k << 16 | (g - A.hoff[k]);
                hrow[u] = A.hrow[h0 + h];
            } else {
                hto[u] = hcol[h];
            }
        }
    }
    __syncthreads();
    // every block of the cluster runs before any touches another's shared memory
    if (CL && tc.ntiles > 1) cooperative_groups::this_cluster().sync();
    // p_k of the halo and of this thread's rows (kaxpby!, cg_dir); the first
    // directions are in place
    for (int ran = 0; ran < max_iters; ++ran) {
        if (ran > 0) {
            const T b = (T)st.beta;
            T hz[RES_HALO_PT];
#pragma unroll
            for (int u = 0; u < RES_HALO_PT; ++u)
                if (hto[u] >= 0) hz[u] = CL ? z_s[RED_TILE + u * RES_THREADS + threadIdx.x] : __ldcg(z + hto[u]);
#pragma unroll
            for (int j = 0; j < RES_ROWS; ++j) pi[j] = z_s[j * RES_THREADS + threadIdx.x] + b * pi[j];
#pragma unroll
            for (int u = 0; u < RES_HALO_PT; ++u)
                if (hto[u] >= 0) {
                    const int l = RED_TILE + u * RES_THREADS + threadIdx.x;
                    dir[l] = hz[u] + b * dir[l];
                }
        }
#pragma unroll
        for (int j = 0; j < RES_ROWS; ++j) dir[j * RES_THREADS + threadIdx.x] = pi[j];
        __syncthreads();
#pragma unroll
        for (int j = 0; j < RES_ROWS; ++j) {
            T q = T(0);
            for (int t = 0; t < ln[j]; ++t) q = q + val[lb[j] + SELL_C * t] * dir[idx[lb[j] + SELL_C * t]];
            qi[j] = q;
            pr[j * RES_THREADS + threadIdx.x] = ln[j] ? (double)pi[j] * (double)q : 0.0;
        }
        __syncthreads();
        double tot = res_tile_sum(pr, sm8);
        double pAp = 0.0;
        if constexpr (CL) pAp = res_exchange_cl(tot, tc, cl_part[0]);
        if (threadIdx.x < 32) {
            const bool ok = CL || res_exchange(tot, tc, ring + (size_t)(ran & 1) * tc.ntiles * tc.ntiles, false, err, pAp,
                                             spin_limit);
            if (threadIdx.x == 0) {
                const double lim = epsT * st.pNorm2;
                if (!ok) {
                    st.stop = 2;
                } else if (pAp <= lim && fabs(pAp) <= lim) {
                    st.stop = 1;
                    st.done = 1;
                    st.status = KS_ZERO_CURV;
                } else {
                    st.alpha = st.gamma / pAp;
                }
            }
        }
        __syncthreads();
        if (st.stop) break;
        const T a = (T)st.alpha;
#pragma unroll
        for (int j = 0; j < RES_ROWS; ++j) {
            const int i = row0 + j * RES_THREADS + threadIdx.x;
            xi[j] = xi[j] + a * pi[j];
            ri[j] = ri[j] + (-a) * qi[j];
            const T zi = jacobi ? Pi[j] * ri[j] : ri[j];
            z_s[j * RES_THREADS + threadIdx.x] = zi;
            if (!CL && tc.ntiles > 1 && i < n) z[i] = zi;
            pr[j * RES_THREADS + threadIdx.x] = ln[j] ? (double)ri[j] * (double)zi : 0.0;
        }
        __syncthreads();
        if constexpr (CL) {
#pragma unroll
            for (int u = 0; u < RES_HALO_PT; ++u)
                if (hto[u] >= 0)
                    *cooperative_groups::this_cluster().map_shared_rank(z_s + RED_TILE + (hto[u] & 0xffff),
                                                                        hto[u] >> 16) = z_s[hrow[u]];
        }
        tot = res_tile_sum(pr, sm8);
        double g = 0.0;
        if constexpr (CL) g = res_exchange_cl(tot, tc, cl_part[1]);
        if (threadIdx.x < 32) {
            const bool ok =
                CL || res_exchange(tot, tc, ring + (size_t)(2 + (ran & 1)) * tc.ntiles * tc.ntiles, true, err, g,
                                   spin_limit);
            if (threadIdx.x == 0) {  // cg_finalize on the block's copy of the state
                const double rn = sqrt(g);
                const bool solved = (rn <= eps) || (rn + 1.0 <= 1.0);
                st.rNorm = rn;
                if (!solved) {
                    const double bt = g / st.gamma;
                    st.beta = bt;
                    st.pNorm2 = g + (bt * bt) * st.pNorm2;
                    st.gamma = g;
                }
                st.iter = st.iter + 1;
                if (solved) {
                    st.done = 1;
                    st.status = KS_SOLVED;
                } else if (st.iter >= itmax) {
                    st.done = 1;
                    st.status = KS_TIRED;
                }
                if (st.done) st.stop = 1;
                if (!ok) st.stop = 2;
            }
        }
        __syncthreads();
        if (st.stop) break;
    }
    if (st.stop == 2) return;
#pragma unroll
    for (int j = 0; j < RES_ROWS; ++j) {
        const int i = row0 + j * RES_THREADS + threadIdx.x;
        if (i < n) x[i] = xi[j];
    }
    if (tc.tile == 0 && threadIdx.x == 0) {
        S->iter = st.iter;
        S->done = st.done;
        S->status = st.status;
        S->gamma = st.gamma;
        S->beta = st.beta;
        S->pNorm2 = st.pNorm2;
        S->alpha = st.alpha;
        S->rNorm = st.rNorm;
    }
}

}  // namespace xcal
