// bicg_fused.cu -- BiCGSTAB of up to three systems that share their matrix's
// off-diagonal entries: the three momentum components (their matrices differ
// in the diagonal alone), or one transported scalar.
//
// A momentum solve to a tenth of its residual takes one or two BiCGSTAB
// iterations (Krylov.jl bicgstab!, Solve_1_api.jl:268-307), so its cost is
// latency: about 25 launches, three dependent DILU applications and several
// host round trips per component, one component after the other.  Here
//   * the components run side by side: a row's slots are read once for all
//     three, and their DILU dataflows (krylov_bodies.cuh) overlap;
//   * an iteration is five launches: A p with M^-1 (k_bf_flow), alpha,
//     A s with M^-1 (s = r - alpha v formed for every gathered column, the
//     owner storing s and x += alpha p), omega, x / r with the stopping tests;
//     p is updated at the start of the next iteration, so a solve that ends
//     after one never does;
//   * the tile reductions use 1024 threads per canonical tile (two rows per
//     thread, the products added by threads 0..255 in the canonical order)
//     where the tile kernels walk eight rows per thread one after the other;
//   * x + x0 and the FP64 residual are launched with the first iterations, so
//     a solve that ends there costs one host synchronisation.
// Arithmetic per component: that of k_init_resid, k_spmv, the DILU or Jacobi
// application and the k_bicg_* kernels, in the same order, with the same
// canonical reduction trees -- bit for bit the results of solving the
// components one by one.  Mixed precision (T = float): the FP32 inner solve
// of the FP64 defect correction, as Case::solve_mixed does it.
//
// What bounds it: the three DILU dataflows (27-61 us each) and the launches
// between them.  Measured on B200, momentum solve per SIMPLE iteration (one
// BiCGSTAB iteration per component, DILU), this against the components one by
// one: 1,073 cells FP64 0.25 / 0.55 ms, 27,025 cells 0.40 / 0.80 ms, 262,144
// cells mixed 0.67 / 1.19 ms, 2.1M cells mixed 2.24 / 3.50 ms.  Captured (graph
// mode; mixed: an outer WHILE over the defect-correction steps), LES at 884,736
// cells, a step: 7.6 -> 6.3 ms.
#include <algorithm>
#include <cstring>

#include "case.hpp"
#include "krylov_bodies.cuh"

namespace xcal {

constexpr int BF_NT = 1024;                     // threads per tile
constexpr int BF_IPT = RED_TILE / BF_NT;        // rows per thread
constexpr int BF_MAX = 3;

// one solve's systems as the kernels read them (component d of d < NC)
template <class T, int NC>
struct BfView {
    CSRView A;
    const T* nz;          // matrix values (NC > 1: the diagonal slots are not read)
    const T* dg[NC];      // diagonals of the components (NC > 1; else nz's own)
    const double* nz64;   // the FP64 matrix: nz, dg themselves for T = double
    const double* dg64[NC];
    const double* b[NC];
    double* field[NC];
    const T* P;           // Jacobi inverse diagonal or DILU D
    LevelView<T> lo, up;
    const T* c[NC];       // shadow vector (b; mixed: the FP32 defect)
    T *x[NC], *r[NC], *p[NC], *v[NC], *s[NC], *t[NC], *q[NC], *y[NC];
    double* dx[NC];
    KScalars* S;          // [NC]
    double *part0, *part1;  // [NC] x tiles
    double* res[NC];
    unsigned int* bar;
    int* err;
    int active;  // components that take part (bit d); a host-known subset of all
};

// values the solve reads, from the assembled FP64 system: the level copies of
// the DILU triangles and 1/D per lower slot, the sweeps' scratch unset, and for
// T = float the FP32 copies of the matrix, diagonals and preconditioner
struct BfRefresh {
    long nnz;
    int n, pre;
    const double* nz;
    const double* P;
    float *nz32, *P32;
    const double* dg64[BF_MAX];
    float* dg32[BF_MAX];
    long nlo, nup;
    const int *lsrc, *lcol, *usrc;
    double *lval, *ldinv, *uval;
    float *lval32, *ldinv32, *uval32;
    void* y[BF_MAX];
    unsigned int* bar;
    int nc, fp32;
};
__global__ void k_bf_refresh(BfRefresh R) {
    const long g = blockIdx.x * (long)blockDim.x + threadIdx.x, G = (long)gridDim.x * blockDim.x;
    if (g == 0) R.bar[0] = 0u;
    if (R.fp32) {
        for (long e = g; e < R.nnz; e += G) R.nz32[e] = (float)ld_stream(R.nz + e);
        for (long i = g; i < R.n; i += G) {
            if (R.pre != XCAL_PRECOND_NONE) R.P32[i] = (float)R.P[i];
            for (int d = 0; d < R.nc; ++d)
                if (R.dg32[d]) R.dg32[d][i] = (float)R.dg64[d][i];
        }
    }
    if (R.pre != XCAL_PRECOND_DILU) return;
    for (long e = g; e < R.nlo; e += G) {
        const double a = R.nz[ld_stream(R.lsrc + e)], D = R.P[ld_stream(R.lcol + e)];
        if (R.fp32) {
            R.lval32[e] = (float)a;
            R.ldinv32[e] = 1.0f / (float)D;
        } else {
            R.lval[e] = a;
            R.ldinv[e] = 1.0 / D;
        }
    }
    for (long e = g; e < R.nup; e += G) {
        const double a = R.nz[ld_stream(R.usrc + e)];
        if (R.fp32)
            R.uval32[e] = (float)a;
        else
            R.uval[e] = a;
    }
    for (long i = g; i < R.n; i += G)
        for (int d = 0; d < R.nc; ++d) {
            if (R.fp32)
                ((float*)R.y[d])[i] = flow_unset_value<float>();
            else
                ((double*)R.y[d])[i] = flow_unset_value<double>();
        }
}

// whether component d takes part, and the components that do (or, running: whose
// solve goes on) as a bit mask; the same in every block: no kernel that reads
// them changes them
template <class T, int NC>
__device__ __forceinline__ bool bf_active(const BfView<T, NC>& V, int d) {
    return (V.active >> d & 1) && !V.S[d].off;
}
template <class T, int NC>
__device__ __forceinline__ int bf_mask(const BfView<T, NC>& V, bool running) {
    int m = 0;
#pragma unroll
    for (int d = 0; d < NC; ++d)
        if (bf_active(V, d) && !(running && V.S[d].done)) m |= 1 << d;
    return m;
}

// flow_wait over the components of one row: waits until the values of every
// column are set in every running component, then finish()
template <class T, int NC, class F>
__device__ __forceinline__ bool bf_wait(T* const (&ys)[NC], int run, const int* __restrict__ col, int base, int c,
                                        const int (&cj)[FLOW_U], T (&yv)[NC][FLOW_U], int* err, F&& finish,
                                        int spin_limit = FLOW_SPIN_LIMIT) {
    bool fin = c < 0;
#pragma unroll
    for (int d = 0; d < NC; ++d)
        if (run >> d & 1)
#pragma unroll
            for (int j = 0; j < FLOW_U; ++j)
                if (j < c) yv[d][j] = ld_flow((const T*)ys[d] + cj[j]);
    for (int spins = 0;; ++spins) {
        if (!fin) {
            bool ready = true;
#pragma unroll
            for (int d = 0; d < NC; ++d)
                if (run >> d & 1) {
#pragma unroll
                    for (int j = 0; j < FLOW_U; ++j)
                        if (j < c && flow_unset(yv[d][j])) ready = false;
                    for (int j = FLOW_U; ready && j < c; ++j)
                        ready = !flow_unset(ld_flow((const T*)ys[d] + ld_stream(col + base + SELL_C * j)));
                }
            if (ready) {
                finish();
                fin = true;
            }
        }
        if (__all_sync(0xffffffffu, fin)) return true;
        if (flow_give_up(spins, spin_limit, err)) return false;
        if (!fin) {
#pragma unroll
            for (int d = 0; d < NC; ++d)
                if (run >> d & 1)
#pragma unroll
                    for (int j = 0; j < FLOW_U; ++j)
                        if (j < c && flow_unset(yv[d][j])) yv[d][j] = ld_flow((const T*)ys[d] + cj[j]);
        }
    }
}

// q = (what M is applied to) row by row, then out = M^-1 q.
//   MODE 0: q = b - A field (FP64; mixed: rounded, and the shadow vector c),
//           x = 0, dx = field;  out = r
//   MODE 1: q = A p;  out = v
//   MODE 2: q = A s with s = r - alpha v, s stored, x += alpha p;  out = t
// PRE = DILU: a cooperative launch (the rows, a grid barrier, the forward rows
// and the backward rows as a dataflow); else an ordinary one.
template <class T, int NC, int PRE, int MODE>
__global__ void __launch_bounds__(FLOW_THREADS) k_bf_flow(const __grid_constant__ BfView<T, NC> V) {
    __shared__ int sh_err;
    const int run = bf_mask(V, MODE != 0);
    if (!run) return;
    const int n = V.A.n;
    const int start = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    T* const(&out)[NC] = MODE == 0 ? V.r : MODE == 1 ? V.v : V.t;
    T alpha[NC];
    if (MODE == 2)
#pragma unroll
        for (int d = 0; d < NC; ++d) alpha[d] = (T)V.S[d].alpha;
    for (int i = start; i < n; i += stride) {
        const int rb = row_base(V.A, i), ln = V.A.len[i], ds = V.A.diag[i];
        if constexpr (MODE == 0) {
            double acc[NC], dg[NC];
#pragma unroll
            for (int d = 0; d < NC; ++d) {
                acc[d] = 0.0;
                dg[d] = NC > 1 ? V.dg64[d][i] : 0.0;
            }
#pragma unroll 4
            for (int k = 0; k < ln; ++k) {
                const int e = rb + SELL_C * k, j = V.A.colval[e];
                const double a = V.nz64[e];
#pragma unroll
                for (int d = 0; d < NC; ++d)
                    acc[d] = acc[d] + (NC > 1 && e == ds ? dg[d] : a) * V.field[d][j];
            }
#pragma unroll
            for (int d = 0; d < NC; ++d)
                if (run >> d & 1) {
                    const T q = (T)(V.b[d][i] - acc[d]);
                    V.q[d][i] = q;
                    V.x[d][i] = T(0);
                    V.dx[d][i] = V.field[d][i];
                    if (sizeof(T) == 4) const_cast<T*>(V.c[d])[i] = q;
                    if (PRE == XCAL_PRECOND_DILU)
                        out[d][i] = flow_unset_value<T>();
                    else
                        out[d][i] = PRE == XCAL_PRECOND_JACOBI ? V.P[i] * q : q;
                }
        } else {
            T acc[NC], dg[NC];
#pragma unroll
            for (int d = 0; d < NC; ++d) {
                acc[d] = T(0);
                dg[d] = NC > 1 ? V.dg[d][i] : T(0);
            }
#pragma unroll 4
            for (int k = 0; k < ln; ++k) {
                const int e = rb + SELL_C * k, j = V.A.colval[e];
                const T a = V.nz[e];
#pragma unroll
                for (int d = 0; d < NC; ++d)
                    if (run >> d & 1) {
                        const T xj = MODE == 1 ? V.p[d][j] : V.r[d][j] + (-alpha[d]) * V.v[d][j];
                        acc[d] = acc[d] + (NC > 1 && e == ds ? dg[d] : a) * xj;
                    }
            }
#pragma unroll
            for (int d = 0; d < NC; ++d)
                if (run >> d & 1) {
                    if (MODE == 2) {
                        V.s[d][i] = V.r[d][i] + (-alpha[d]) * V.v[d][i];
                        V.x[d][i] = V.x[d][i] + alpha[d] * V.p[d][i];
                    }
                    V.q[d][i] = acc[d];
                    if (PRE == XCAL_PRECOND_DILU)
                        out[d][i] = flow_unset_value<T>();
                    else
                        out[d][i] = PRE == XCAL_PRECOND_JACOBI ? V.P[i] * acc[d] : acc[d];
                }
        }
    }
    if constexpr (PRE == XCAL_PRECOND_DILU) {
        unsigned int nb = 0;
        if (!grid_barrier(V.bar, gridDim.x, nb, V.err, &sh_err)) return;
        for (int k0 = start & ~31; k0 < n; k0 += stride) {
            const int k = k0 + (threadIdx.x & 31);
            int i = 0, c = -1, base = 0;
            int cj[FLOW_U];
            T vj[FLOW_U], dj[FLOW_U], yv[NC][FLOW_U], rhs[NC];
            if (k < n) {
                i = V.lo.rows[k];
                c = V.lo.cnt[k];
                base = V.lo.slice[k / SELL_C] + (k % SELL_C);
#pragma unroll
                for (int j = 0; j < FLOW_U; ++j)
                    if (j < c) {
                        const int e = base + SELL_C * j;
                        cj[j] = ld_stream(V.lo.col + e);
                        vj[j] = ld_stream(V.lo.val + e);
                        dj[j] = ld_stream(V.lo.dinv + e);
                    }
#pragma unroll
                for (int d = 0; d < NC; ++d) rhs[d] = run >> d & 1 ? ld_flow((const T*)V.q[d] + i) : T(0);
            }
            if (!bf_wait<T, NC>(V.y, run, V.lo.col, base, c, cj, yv, V.err, [&] {
#pragma unroll
                    for (int d = 0; d < NC; ++d)
                        if (run >> d & 1) {
                            T sum = T(0);
#pragma unroll
                            for (int j = 0; j < FLOW_U; ++j)
                                if (j < c) sum = sum + (vj[j] * yv[d][j]) * dj[j];
                            for (int j = FLOW_U; j < c; ++j) {
                                const int e = base + SELL_C * j;
                                sum = sum + (ld_stream(V.lo.val + e) *
                                             ld_flow((const T*)V.y[d] + ld_stream(V.lo.col + e))) *
                                                ld_stream(V.lo.dinv + e);
                            }
                            st_flow(V.y[d] + i, rhs[d] - sum);
                        }
                }))
                return;
        }
        // a row's forward value may come from another block: polled as well
        for (int k0 = start & ~31; k0 < n; k0 += stride) {
            const int k = k0 + (threadIdx.x & 31);
            int i = 0, c = -1, base = 0;
            int cj[FLOW_U];
            T vj[FLOW_U], yv[NC][FLOW_U];
            T Di = T(0);
            if (k < n) {
                i = V.up.rows[k];
                c = V.up.cnt[k];
                base = V.up.slice[k / SELL_C] + (k % SELL_C);
#pragma unroll
                for (int j = 0; j < FLOW_U; ++j)
                    if (j < c) {
                        const int e = base + SELL_C * j;
                        cj[j] = ld_stream(V.up.col + e);
                        vj[j] = ld_stream(V.up.val + e);
                    }
                Di = V.P[i];
            }
            if (!bf_wait<T, NC>(out, run, V.up.col, base, c, cj, yv, V.err, [&] {
#pragma unroll
                    for (int d = 0; d < NC; ++d)
                        if (run >> d & 1) {
                            T sum = T(0);
#pragma unroll
                            for (int j = 0; j < FLOW_U; ++j)
                                if (j < c) sum = sum + vj[j] * yv[d][j];
                            for (int j = FLOW_U; j < c; ++j) {
                                const int e = base + SELL_C * j;
                                sum = sum + ld_stream(V.up.val + e) *
                                                ld_flow((const T*)out[d] + ld_stream(V.up.col + e));
                            }
                            T yi = ld_flow((const T*)V.y[d] + i);
                            for (int spins = 0; flow_unset(yi) && spins < FLOW_SPIN_LIMIT; ++spins)
                                yi = ld_flow((const T*)V.y[d] + i);
                            if (flow_unset(yi)) *(volatile int*)V.err = 1;
                            V.y[d][i] = flow_unset_value<T>();
                            st_flow(out[d] + i, (yi - sum) / Di);
                        }
                }))
                return;
        }
    }
}

// canonical partials of one tile from the products pr[v][row of tile], by a
// block of BF_NT threads: threads 0..255 add their eight rows in k order,
// then the block tree
__device__ __forceinline__ double bf_tile_sum(const double* pr, double* sm) {
    double acc = 0.0;
    if (threadIdx.x < RED_THREADS)
#pragma unroll
        for (int k = 0; k < RED_ITEMS; ++k) acc = acc + pr[k * RED_THREADS + threadIdx.x];
    return block_tree(acc, sm);
}

// p = r; ||r||, <c, r>; the start tests of bicgstab!
template <class T, int NC>
__global__ void __launch_bounds__(BF_NT) k_bf_start(const __grid_constant__ BfView<T, NC> V) {
    __shared__ double pr[2][RED_TILE];
    __shared__ double sm[8];
    const int d = blockIdx.y, n = V.A.n, nt = gridDim.x;
    if (blockIdx.x == 0 && d == 0 && threadIdx.x == 0) V.bar[0] = 0u;
    if (!bf_active(V, d)) return;
#pragma unroll
    for (int j = 0; j < BF_IPT; ++j) {
        const int l = j * BF_NT + threadIdx.x, i = blockIdx.x * RED_TILE + l;
        double a = 0.0, c = 0.0;
        if (i < n) {
            const T ri = V.r[d][i];
            V.p[d][i] = ri;
            a = (double)ri * (double)ri;
            c = (double)V.c[d][i] * (double)ri;
        }
        pr[0][l] = a;
        pr[1][l] = c;
    }
    __syncthreads();
    const double t0 = bf_tile_sum(pr[0], sm), t1 = bf_tile_sum(pr[1], sm);
    double *p0 = V.part0 + (size_t)d * nt, *p1 = V.part1 + (size_t)d * nt;
    if (threadIdx.x == 0) {
        p0[blockIdx.x] = t0;
        p1[blockIdx.x] = t1;
    }
    if (!last_block(&V.S[d].counter, nt)) return;
    const double rr = reduce_partials(p0, nt, sm), cr = reduce_partials(p1, nt, sm);
    if (threadIdx.x == 0) bicg_start_scalars(V.S + d, rr, cr);
}

// alpha = rho / <c, v>
template <class T, int NC>
__global__ void __launch_bounds__(BF_NT) k_bf_alpha(const __grid_constant__ BfView<T, NC> V) {
    __shared__ double pr[RED_TILE];
    __shared__ double sm[8];
    const int d = blockIdx.y, n = V.A.n, nt = gridDim.x;
    if (blockIdx.x == 0 && d == 0 && threadIdx.x == 0) V.bar[0] = 0u;
    if (!bf_active(V, d) || V.S[d].done) return;
#pragma unroll
    for (int j = 0; j < BF_IPT; ++j) {
        const int l = j * BF_NT + threadIdx.x, i = blockIdx.x * RED_TILE + l;
        pr[l] = i < n ? (double)V.c[d][i] * (double)V.v[d][i] : 0.0;
    }
    __syncthreads();
    const double t0 = bf_tile_sum(pr, sm);
    double* p0 = V.part0 + (size_t)d * nt;
    if (threadIdx.x == 0) p0[blockIdx.x] = t0;
    if (!last_block(&V.S[d].counter, nt)) return;
    const double cv = reduce_partials(p0, nt, sm);
    if (threadIdx.x == 0) bicg_alpha_scalars(V.S + d, cv);
}

// omega = <t, s> / <t, t>
template <class T, int NC>
__global__ void __launch_bounds__(BF_NT) k_bf_omega(const __grid_constant__ BfView<T, NC> V) {
    __shared__ double pr[2][RED_TILE];
    __shared__ double sm[8];
    const int d = blockIdx.y, n = V.A.n, nt = gridDim.x;
    if (!bf_active(V, d) || V.S[d].done) return;
#pragma unroll
    for (int j = 0; j < BF_IPT; ++j) {
        const int l = j * BF_NT + threadIdx.x, i = blockIdx.x * RED_TILE + l;
        const double ti = i < n ? (double)V.t[d][i] : 0.0;
        pr[0][l] = i < n ? ti * (double)V.s[d][i] : 0.0;
        pr[1][l] = i < n ? ti * ti : 0.0;
    }
    __syncthreads();
    const double t0 = bf_tile_sum(pr[0], sm), t1 = bf_tile_sum(pr[1], sm);
    double *p0 = V.part0 + (size_t)d * nt, *p1 = V.part1 + (size_t)d * nt;
    if (threadIdx.x == 0) {
        p0[blockIdx.x] = t0;
        p1[blockIdx.x] = t1;
    }
    if (!last_block(&V.S[d].counter, nt)) return;
    const double ts = reduce_partials(p0, nt, sm), tt = reduce_partials(p1, nt, sm);
    if (threadIdx.x == 0) V.S[d].omega = ts / tt;
}

// x += omega s; r = s - omega t; <c, r>, ||r||; the stopping tests
template <class T, int NC>
__global__ void __launch_bounds__(BF_NT) k_bf_xr(const __grid_constant__ BfView<T, NC> V) {
    __shared__ double pr[2][RED_TILE];
    __shared__ double sm[8];
    const int d = blockIdx.y, n = V.A.n, nt = gridDim.x;
    if (!bf_active(V, d) || V.S[d].done) return;
    const double omega = V.S[d].omega;
    const T om = (T)omega;
#pragma unroll
    for (int j = 0; j < BF_IPT; ++j) {
        const int l = j * BF_NT + threadIdx.x, i = blockIdx.x * RED_TILE + l;
        double a = 0.0, c = 0.0;
        if (i < n) {
            const T si = V.s[d][i];
            V.x[d][i] = V.x[d][i] + om * si;
            const T ri = si + (-om) * V.t[d][i];
            V.r[d][i] = ri;
            a = (double)V.c[d][i] * (double)ri;
            c = (double)ri * (double)ri;
        }
        pr[0][l] = a;
        pr[1][l] = c;
    }
    __syncthreads();
    const double t0 = bf_tile_sum(pr[0], sm), t1 = bf_tile_sum(pr[1], sm);
    double *p0 = V.part0 + (size_t)d * nt, *p1 = V.part1 + (size_t)d * nt;
    if (threadIdx.x == 0) {
        p0[blockIdx.x] = t0;
        p1[blockIdx.x] = t1;
    }
    if (!last_block(&V.S[d].counter, nt)) return;
    const double cr = reduce_partials(p0, nt, sm), rr = reduce_partials(p1, nt, sm);
    if (threadIdx.x == 0) bicg_xr_scalars(V.S + d, omega, cr, rr);
}

// p = r + beta (p - omega v), at the start of every iteration but the first
template <class T, int NC>
__global__ void __launch_bounds__(BF_NT) k_bf_p(const __grid_constant__ BfView<T, NC> V) {
    const int d = blockIdx.y, n = V.A.n;
    if (blockIdx.x == 0 && d == 0 && threadIdx.x == 0) V.bar[0] = 0u;
    if (!bf_active(V, d) || V.S[d].done || V.S[d].iter == 0) return;
    const T beta = (T)V.S[d].beta, omega = (T)V.S[d].omega;
#pragma unroll
    for (int j = 0; j < BF_IPT; ++j) {
        const int i = blockIdx.x * RED_TILE + j * BF_NT + threadIdx.x;
        if (i < n) V.p[d][i] = V.r[d][i] + beta * (V.p[d][i] + (-omega) * V.v[d][i]);
    }
}

// field = x + x0 (mixed: unless the defect was already at its target) and the
// scaled residual of the new field (k_residual); components still running are
// left alone.  Neighbours' new values are formed from x and x0, so the field
// may be written while they are read.
template <class T, int NC>
__global__ void __launch_bounds__(BF_NT) k_bf_finish(const __grid_constant__ BfView<T, NC> V) {
    __shared__ double pr[2][RED_TILE];
    __shared__ double sm[8];
    const int d = blockIdx.y, n = V.A.n, nt = gridDim.x;
    if (!bf_active(V, d) || !V.S[d].done) return;
    const bool apply = sizeof(T) == 8 || !V.S[d].outer_conv;
    const T* x = V.x[d];
    const double* dx = V.dx[d];
    auto val = [&](int j) { return apply ? (sizeof(T) == 8 ? (double)x[j] + dx[j] : dx[j] + (double)x[j]) : dx[j]; };
#pragma unroll
    for (int jj = 0; jj < BF_IPT; ++jj) {
        const int l = jj * BF_NT + threadIdx.x, i = blockIdx.x * RED_TILE + l;
        double a = 0.0, c = 0.0;
        if (i < n) {
            const int rb = row_base(V.A, i), ln = V.A.len[i], ds = V.A.diag[i];
            const double dg = NC > 1 ? V.dg64[d][i] : 0.0;
            double fx = 0.0;
#pragma unroll 4
            for (int k = 0; k < ln; ++k) {
                const int e = rb + SELL_C * k;
                fx = fx + (NC > 1 && e == ds ? dg : V.nz64[e]) * val(V.A.colval[e]);
            }
            V.field[d][i] = val(i);
            const double bi = V.b[d][i], df = bi - fx;
            a = df * df;
            c = bi * bi;
        }
        pr[0][l] = a;
        pr[1][l] = c;
    }
    __syncthreads();
    const double t0 = bf_tile_sum(pr[0], sm), t1 = bf_tile_sum(pr[1], sm);
    double *p0 = V.part0 + (size_t)d * nt, *p1 = V.part1 + (size_t)d * nt;
    if (threadIdx.x == 0) {
        p0[blockIdx.x] = t0;
        p1[blockIdx.x] = t1;
    }
    if (!last_block(&V.S[d].counter2, nt)) return;
    const double sR = reduce_partials(p0, nt, sm), sb = reduce_partials(p1, nt, sm);
    if (threadIdx.x == 0) residual_scalars(V.S + d, sR, sb, V.res[d]);
}

// device-driven control (graph mode)
template <int NC>
__global__ void k_bf_init(KScalars* S, double atol, double rtol, int itmax, int mixed, double inner_rtol) {
    const int d = threadIdx.x;
    if (blockIdx.x != 0 || d >= NC) return;
    KScalars z = {};
    z.atol = atol;
    z.rtol = rtol;
    z.itmax = itmax;
    z.mixed = mixed;
    z.inner_rtol = inner_rtol;
    S[d] = z;
}
// end of an iteration body: goes on while a component runs, at most cap bodies
template <int NC>
__global__ void k_bf_loop_cond(cudaGraphConditionalHandle h, KScalars* S, int cap, int body_kernels,
                               unsigned long long* launches) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    atomicAdd(launches, (unsigned long long)body_kernels);
    bool any = false;
    for (int d = 0; d < NC; ++d) {
        if (S[d].off) continue;
        S[d].loops = S[d].loops + 1;
        if (!S[d].done && S[d].loops >= cap) {
            S[d].done = 1;
            S[d].status = KS_LOOP_CAP;
        }
        any = any || !S[d].done;
    }
    cudaGraphSetConditional(h, any ? 1u : 0u);
}
// one defect-correction step of the components still in it (solve_mixed's
// loop, on the device): its start, and its exit tests
template <int NC>
__global__ void k_bf_outer_prep(KScalars* S, unsigned int* bar) {
    const int d = threadIdx.x;
    if (blockIdx.x != 0 || d >= NC) return;
    if (d == 0) bar[0] = 0u;
    if (S[d].off) return;
    S[d].iter = 0;
    S[d].done = 0;
    S[d].status = KS_RUNNING;
}
template <int NC>
__global__ void k_bf_outer_cond(cudaGraphConditionalHandle h, KScalars* S, int max_outer, int body_kernels,
                                unsigned long long* launches) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    atomicAdd(launches, (unsigned long long)body_kernels);
    bool any = false;
    for (int d = 0; d < NC; ++d) {
        KScalars& K = S[d];
        if (K.off) continue;
        bool stop = K.outer_conv != 0;
        if (!stop) {
            K.total = K.total + K.iter;
            const int st = K.status;
            stop = st == KS_ZERO_CURV || st == KS_BREAKDOWN || st == KS_TIRED || st == KS_LOOP_CAP ||
                   (st == KS_SOLVED && K.eps <= K.eps_outer);
        }
        K.outer = K.outer + 1;
        if (stop || K.outer >= max_outer)
            K.off = 1;
        else
            any = true;
    }
    cudaGraphSetConditional(h, any ? 1u : 0u);
}
template <int NC>
__global__ void k_bf_record(const KScalars* S, int* out, int* hits) {
    const int d = threadIdx.x;
    if (blockIdx.x != 0 || d >= NC) return;
    if (S[d].status == KS_TIRED) atomicAdd(hits, 1);
    out[2 * d] = S[d].mixed ? S[d].total : S[d].iter;
    out[2 * d + 1] = S[d].status;
}

// bf_wait of a warp whose first row needs, in the last component, a value that
// nothing writes; left[lane]: whether the lane left without its row
__global__ void k_bf_wait_check(double* y0, double* y1, double* y2, const int* col, int* err, int spin_limit,
                                int* left) {
    double* ys[BF_MAX] = {y0, y1, y2};
    const int cj[FLOW_U] = {};
    double yv[BF_MAX][FLOW_U];
    const bool ok = bf_wait<double, BF_MAX>(ys, (1 << BF_MAX) - 1, col, 0, threadIdx.x == 0 ? 1 : 0, cj, yv, err,
                                            [] {}, spin_limit);
    left[threadIdx.x] = ok ? 0 : 1;
}
bool check_fused_wait(int spin_limit, int* err) {
    DBuf<double> y;
    DBuf<int> col, left;
    y.alloc(BF_MAX);
    y.zero(0);
    kr_flow_unset(0, y.p + BF_MAX - 1, sizeof(double));
    col.alloc(1);
    col.zero(0);
    left.alloc(32);
    left.zero(0);
    k_bf_wait_check<<<1, 32>>>(y.p, y.p + 1, y.p + 2, col.p, err, spin_limit, left.p);
    XCAL_CHECK_LAUNCH();
    int h[32];
    XCAL_CUDA(cudaMemcpy(h, left.p, sizeof(h), cudaMemcpyDeviceToHost));
    return std::count(h, h + 32, 1) == 32;
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
template <class T, int NC, int PRE, int MODE>
static void bf_flow_pre(cudaStream_t s, const BfView<T, NC>& V) {
    const void* k = (const void*)k_bf_flow<T, NC, PRE, MODE>;
    const int want = (V.A.n + FLOW_THREADS - 1) / FLOW_THREADS;
    if constexpr (PRE != XCAL_PRECOND_DILU) {
        k_bf_flow<T, NC, PRE, MODE><<<want, FLOW_THREADS, 0, s>>>(V);
        XCAL_CHECK_LAUNCH();
    } else {
        const int blocks = std::min(flow_grid(k), want);
        BfView<T, NC> Vv = V;
        void* args[] = {&Vv};
        if (!flow_launch(k, blocks, s, args))
            fail(XCAL_ERR_CUDA, "fused BiCGSTAB: the DILU kernel does not fit the device");
    }
}
template <class T, int NC, int MODE>
static void bf_flow(cudaStream_t s, const BfView<T, NC>& V, int pre) {
    if (pre == XCAL_PRECOND_DILU)
        bf_flow_pre<T, NC, XCAL_PRECOND_DILU, MODE>(s, V);
    else if (pre == XCAL_PRECOND_JACOBI)
        bf_flow_pre<T, NC, XCAL_PRECOND_JACOBI, MODE>(s, V);
    else
        bf_flow_pre<T, NC, XCAL_PRECOND_NONE, MODE>(s, V);
}

template <class T, int NC>
static void bf_start(cudaStream_t s, const BfView<T, NC>& V, int pre) {
    const dim3 grid((V.A.n + RED_TILE - 1) / RED_TILE, NC);
    bf_flow<T, NC, 0>(s, V, pre);
    k_bf_start<T, NC><<<grid, BF_NT, 0, s>>>(V);
    XCAL_CHECK_LAUNCH();
}
// one iteration; first: the solve's first (no p update to do)
template <class T, int NC>
static void bf_iterate(cudaStream_t s, const BfView<T, NC>& V, int pre, bool first) {
    const dim3 grid((V.A.n + RED_TILE - 1) / RED_TILE, NC);
    if (!first) {
        k_bf_p<T, NC><<<grid, BF_NT, 0, s>>>(V);
        XCAL_CHECK_LAUNCH();
    }
    bf_flow<T, NC, 1>(s, V, pre);
    k_bf_alpha<T, NC><<<grid, BF_NT, 0, s>>>(V);
    XCAL_CHECK_LAUNCH();
    bf_flow<T, NC, 2>(s, V, pre);
    k_bf_omega<T, NC><<<grid, BF_NT, 0, s>>>(V);
    XCAL_CHECK_LAUNCH();
    k_bf_xr<T, NC><<<grid, BF_NT, 0, s>>>(V);
    XCAL_CHECK_LAUNCH();
}
template <class T, int NC>
static void bf_finish(cudaStream_t s, const BfView<T, NC>& V) {
    const dim3 grid((V.A.n + RED_TILE - 1) / RED_TILE, NC);
    k_bf_finish<T, NC><<<grid, BF_NT, 0, s>>>(V);
    XCAL_CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// The fused solve covers BiCGSTAB without a smoother at every size (momentum
// solve per SIMPLE iteration, components in turn with the fastest DILU form
// against this, ms: 884,736 cells mixed 2.35 / 1.08, FP64 2.45 / 1.17; 2.1M cells
// mixed 3.50 / 2.24, FP64 3.95 / 2.74).  A chosen DILU form keeps the separate
// kernels, and so does profiling, which times them, but for a captured step
// (captured): nothing is timed in it, and it outlives the profiling.  A batch
// runs its own batched ones.
bool Case::use_fused(const Equation& E, const xcal_solver_setup& SS, bool captured) {
    if (SS.solver != XCAL_SOLVER_BICGSTAB || SS.smoother_loops > 0 || batch_err || dilu_mode != 0) return false;
    if (profiling && !captured) return false;
    if (SS.precond != XCAL_PRECOND_DILU) return true;
    // the sweeps are cooperative launches, under capture inside WHILE bodies
    return E.flow_D && !E.lower_off.empty() && (captured ? kr_coop_capture_ok(true) : coop_ok_here());
}

// Components may be solved side by side when no boundary condition of one
// reads another: Wall and Symmetry project the cell's velocity on the face
// normal, so their faces must have axis-aligned normals (the other
// components then enter as products with an exact zero)
bool Case::components_apart() {
    if (apart < 0) {
        apart = 1;
        for (const xcal_bc& bc : bcU.src) {
            if (bc.type != XCAL_BC_WALL && bc.type != XCAL_BC_SYMMETRY) continue;
            const int f0 = mesh->patch_start[bc.patch], f1 = f0 + mesh->patch_count[bc.patch];
            for (int f = f0; f < f1 && apart; ++f)
                apart = (mesh->nxh[f] != 0.0) + (mesh->nyh[f] != 0.0) + (mesh->nzh[f] != 0.0) <= 1;
        }
    }
    return apart == 1;
}

// work vectors of components 1 and 2, and the three diagonals, allocated at the
// first fused momentum solve (a case in a batch has none), never under capture;
// where they (above 64 MB) would take more than a quarter of the free memory the
// components are solved in turn
void Case::reserve_fused(bool captured) {
    if (bf.ready || bf.refused || capturing || !use_fused(U, cfg.U_solver, captured) || !components_apart()) return;
    const bool mixed = cfg.precision == XCAL_PREC_MIXED;
    const size_t n = U.n, T = (n + RED_TILE - 1) / RED_TILE;
    // one allocation: seven cost a new case's first step 0.1-0.2 ms (1,073 and
    // 27,025 cells: 0.66 -> 0.57 and 2.04 -> 1.90 ms)
    size_t need = 0;
    auto take = [&](size_t b) {
        const size_t at = need;
        need += (b + 255) & ~size_t(255);
        return at;
    };
    const size_t o_diag = take(3 * n * sizeof(double)), o_dx = take(2 * n * sizeof(double));
    const size_t o_part0 = take(3 * T * sizeof(double)), o_part1 = take(3 * T * sizeof(double));
    const size_t o_res = take(3 * sizeof(double)), o_S = take(3 * sizeof(KScalars));
    const size_t o_vec = take(mixed ? 2 * 9 * n * sizeof(float) : 2 * 8 * n * sizeof(double));
    const size_t o_diag32 = take(mixed ? 3 * n * sizeof(float) : 0);
    size_t held = 0;
    if (need > (size_t)64 << 20) {
        size_t free_b = 0, total_b = 0;
        XCAL_CUDA(cudaMemGetInfo(&free_b, &total_b));
        if (need > free_b / 4) {
            bf.refused = true;
            return;
        }
    }
    try {
        AllocScope acc(&held);
        bf.mem.alloc(need);
    } catch (const Error&) {
        cudaGetLastError();
        bf.refused = true;
        return;
    }
    unsigned char* m = bf.mem.p;
    bf.diag = reinterpret_cast<double*>(m + o_diag);
    bf.dx = reinterpret_cast<double*>(m + o_dx);
    bf.part0 = reinterpret_cast<double*>(m + o_part0);
    bf.part1 = reinterpret_cast<double*>(m + o_part1);
    bf.res = reinterpret_cast<double*>(m + o_res);
    bf.S = reinterpret_cast<KScalars*>(m + o_S);
    if (mixed) {
        bf.vec32 = reinterpret_cast<float*>(m + o_vec);
        bf.diag32 = reinterpret_cast<float*>(m + o_diag32);
    } else {
        bf.vec = reinterpret_cast<double*>(m + o_vec);
    }
    XCAL_CUDA(cudaMemsetAsync(bf.S, 0, 3 * sizeof(KScalars), stream));
    bytes += held;
    bf.ready = true;
}

template <class T, int NC>
BfView<T, NC> Case::bf_view(Equation& E, const xcal_solver_setup& SS, const SolveRef* R) {
    constexpr bool F = sizeof(T) == 4;
    const size_t n = E.n;
    BfView<T, NC> V{};
    V.A = E.view();
    V.nz64 = E.nz.p;
    V.bar = ws.bar.p;
    V.err = ws.err.p;
    V.active = (1 << NC) - 1;
    V.S = NC == 1 ? ws.S.p + R[0].kslot : bf.S;
    V.part0 = NC == 1 ? ws.part0.p : bf.part0;
    V.part1 = NC == 1 ? ws.part1.p : bf.part1;
    if (SS.precond == XCAL_PRECOND_DILU) {
        V.lo = level_view<T>(E, 0);
        V.up = level_view<T>(E, 1);
    }
    if constexpr (F) {
        V.nz = E.nz32.p;
        V.P = E.P32.p;
    } else {
        V.nz = E.nz.p;
        V.P = E.P.p;
    }
    for (int d = 0; d < NC; ++d) {
        V.b[d] = R[d].b;
        V.field[d] = R[d].field;
        V.res[d] = capturing ? gres.p + R[d].slot : NC == 1 ? resbuf.p : bf.res + d;
        V.dg64[d] = NC == 1 ? nullptr : bf.diag + d * n;
        V.dx[d] = d == 0 ? ws.dx.p : bf.dx + (d - 1) * n;
        T* w[9];
        if constexpr (F) {
            T* first[9] = {ws.fx.p, ws.fr.p, ws.fp.p, ws.fv.p, ws.fs.p, ws.ft.p, ws.fq.p, ws.fz.p, ws.fd.p};
            for (int k = 0; k < 9; ++k) w[k] = d == 0 ? first[k] : bf.vec32 + ((d - 1) * 9 + k) * n;
            V.dg[d] = NC == 1 ? nullptr : bf.diag32 + d * n;
            V.c[d] = w[8];
        } else {
            T* first[8] = {ws.x.p, ws.r.p, ws.p.p, ws.v.p, ws.s.p, ws.t.p, ws.q.p, ws.z.p};
            for (int k = 0; k < 8; ++k) w[k] = d == 0 ? first[k] : bf.vec + ((d - 1) * 8 + k) * n;
            V.dg[d] = V.dg64[d];
            V.c[d] = R[d].b;
        }
        V.x[d] = w[0];
        V.r[d] = w[1];
        V.p[d] = w[2];
        V.v[d] = w[3];
        V.s[d] = w[4];
        V.t[d] = w[5];
        V.q[d] = w[6];
        V.y[d] = w[7];
    }
    return V;
}

template <class T, int NC>
static void bf_refresh(cudaStream_t s, Equation& E, const BfView<T, NC>& V, int pre) {
    BfRefresh r{};
    r.nnz = E.nnz;
    r.n = E.n;
    r.pre = pre;
    r.nz = E.nz.p;
    r.P = E.P.p;
    r.fp32 = sizeof(T) == 4;
    r.nz32 = E.nz32.p;
    r.P32 = E.P32.p;
    r.bar = V.bar;
    r.nc = NC;
    for (int d = 0; d < NC; ++d) {
        r.dg64[d] = V.dg64[d];
        r.dg32[d] = sizeof(T) == 4 ? (float*)V.dg[d] : nullptr;
        r.y[d] = V.y[d];
    }
    if (pre == XCAL_PRECOND_DILU) {
        r.nlo = E.lsell.nslots;
        r.nup = E.usell.nslots;
        r.lsrc = E.lsell.src.p;
        r.lcol = E.lsell.col.p;
        r.usrc = E.usell.src.p;
        r.lval = E.lsell.val.p;
        r.ldinv = E.lsell.dinv.p;
        r.uval = E.usell.val.p;
        r.lval32 = E.lsell.val32.p;
        r.ldinv32 = E.lsell.dinv32.p;
        r.uval32 = E.usell.val32.p;
    } else if (sizeof(T) == 8) {
        XCAL_CUDA(cudaMemsetAsync(V.bar, 0, sizeof(unsigned int), s));
        return;
    }
    const long work = std::max((long)E.n, sizeof(T) == 4 ? E.nnz : r.nlo);
    k_bf_refresh<<<(int)std::min((work + 255) / 256, 148L * 8), 256, 0, s>>>(r);
    XCAL_CHECK_LAUNCH();
}

// NC solves of one equation: R[d] their fields, right-hand sides and result
// slots; the residuals into res.  The diagonals of NC = 3 are in bf.diag.
template <class T, int NC>
void Case::fused_solve(Equation& E, const xcal_solver_setup& SS, const SolveRef* R, double* res) {
    const int n = E.n, pre = SS.precond;
    const int itmax = SS.itmax == 0 ? 2 * n : SS.itmax;
    const bool mixed = sizeof(T) == 4;
    const double inner_rtol = cfg.inner_rtol > 0 ? cfg.inner_rtol : 1e-3;
    BfView<T, NC> V = bf_view<T, NC>(E, SS, R);
    bf_refresh<T, NC>(stream, E, V, pre);
    if (capturing) {
        k_bf_init<NC><<<1, 32, 0, stream>>>(V.S, SS.atol, SS.rtol, itmax, mixed ? 1 : 0, inner_rtol);
        XCAL_CHECK_LAUNCH();
        auto solve = [&] {
            bf_start(stream, V, pre);
            capture_while([&](cudaGraphConditionalHandle h) {
                const long long k0 = t_launch_count;
                bf_iterate(stream, V, pre, false);
                k_bf_loop_cond<NC><<<1, 32, 0, stream>>>(h, V.S, itmax + 2, (int)(t_launch_count - k0) + 1, dlaunch.p);
                XCAL_CHECK_LAUNCH();
            });
            bf_finish(stream, V);
        };
        if (mixed)
            capture_while([&](cudaGraphConditionalHandle h) {
                const long long k0 = t_launch_count;
                k_bf_outer_prep<NC><<<1, 32, 0, stream>>>(V.S, V.bar);
                XCAL_CHECK_LAUNCH();
                solve();
                // this body's own kernels (the iterations' bodies count themselves)
                const int own = (int)(t_launch_count - k0 - last_body_kernels) + 1;
                k_bf_outer_cond<NC><<<1, 32, 0, stream>>>(h, V.S, 64, own, dlaunch.p);
                XCAL_CHECK_LAUNCH();
            });
        else
            solve();
        k_bf_record<NC><<<1, 32, 0, stream>>>(V.S, giters.p + 2 * R[0].slot, giters.p + 2 * GRES_N);
        XCAL_CHECK_LAUNCH();
        for (int d = 0; d < NC; ++d) res[d] = 0.0;
        return;
    }
    KScalars* hS = NC == 1 ? h_S + R[0].kslot : h_S + 2;
    double* hres = h_res;
    std::memset(hS, 0, NC * sizeof(KScalars));
    for (int d = 0; d < NC; ++d) {
        hS[d].atol = SS.atol;
        hS[d].rtol = SS.rtol;
        hS[d].itmax = itmax;
        hS[d].mixed = mixed ? 1 : 0;
        hS[d].inner_rtol = mixed ? inner_rtol : 0.0;
    }
    int total[NC] = {}, status[NC] = {}, outers[NC] = {};
    for (int outer = 0; V.active && outer < (mixed ? 64 : 1); ++outer) {
        for (int d = 0; d < NC; ++d)
            if (V.active >> d & 1) {
                hS[d].outer = outer;
                hS[d].iter = hS[d].done = 0;
                hS[d].status = KS_RUNNING;
            }
        XCAL_CUDA(cudaMemcpyAsync(V.S, hS, NC * sizeof(KScalars), cudaMemcpyHostToDevice, stream));
        if (outer > 0) XCAL_CUDA(cudaMemsetAsync(V.bar, 0, sizeof(unsigned int), stream));
        bf_start(stream, V, pre);
        long launched = 0;
        for (int chunk = 1;; chunk = std::min(2 * chunk, 8)) {
            if ((launched += chunk) > (long)itmax + 48)
                fail(XCAL_ERR_TIMEOUT, "BiCGSTAB did not report completion within itmax iterations");
            for (int c = 0; c < chunk; ++c) bf_iterate(stream, V, pre, launched == chunk && c == 0);
            bf_finish(stream, V);
            XCAL_CUDA(cudaMemcpyAsync(hS, V.S, NC * sizeof(KScalars), cudaMemcpyDeviceToHost, stream));
            XCAL_CUDA(cudaMemcpyAsync(hres, V.res[0], NC * sizeof(double), cudaMemcpyDeviceToHost, stream));
            if (pre == XCAL_PRECOND_DILU)
                XCAL_CUDA(cudaMemcpyAsync(h_perr, ws.err.p, sizeof(int), cudaMemcpyDeviceToHost, stream));
            sync();
            if (pre == XCAL_PRECOND_DILU) report_wait(*h_perr, "DILU sweep: a wait gave up");
            bool all = true;
            for (int d = 0; d < NC; ++d) all = all && (!(V.active >> d & 1) || hS[d].done);
            if (all) break;
        }
        for (int d = 0; d < NC; ++d) {
            if (!(V.active >> d & 1)) continue;
            outers[d] = outer + 1;
            status[d] = hS[d].status;
            res[d] = hres[d];
            if (!(mixed && hS[d].outer_conv)) total[d] += hS[d].iter;
            const int st = status[d];
            // solve_mixed's exits: the defect was at its target, or the inner
            // solve failed or met that target
            if (!mixed || hS[d].outer_conv || st == KS_ZERO_CURV || st == KS_BREAKDOWN || st == KS_TIRED ||
                (st == KS_SOLVED && hS[d].eps <= hS[d].eps_outer))
                V.active &= ~(1 << d);
        }
    }
    for (int d = 0; d < NC; ++d) {
        const int gk = R[d].gk;
        last_iters[gk] = total[d];
        if (mixed) last_outer[gk] = outers[d];
        note_status(gk, status[d]);
    }
}
template void Case::fused_solve<double, 1>(Equation&, const xcal_solver_setup&, const SolveRef*, double*);
template void Case::fused_solve<double, 3>(Equation&, const xcal_solver_setup&, const SolveRef*, double*);
template void Case::fused_solve<float, 1>(Equation&, const xcal_solver_setup&, const SolveRef*, double*);
template void Case::fused_solve<float, 3>(Equation&, const xcal_solver_setup&, const SolveRef*, double*);

}  // namespace xcal
