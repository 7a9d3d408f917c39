// autotune.cu -- launch-shape autotuner.
//
// Tunes only choices that leave every result bit-identical:
//  * the row mapping and block size of the SpMVs that carry no reduction
//    (the BiCGSTAB SpMV): the canonical tile kernel or 1/2/4 rows per thread
//    in blocks of 128/256/512 threads;
//  * how a DILU application of a system of more than 524,288 rows runs: rows
//    waiting for the values they read (dataflow), one launch per level, or
//    every level in one cooperative launch with a grid barrier between levels
//    (the fused BiCGSTAB, which shares the waits among components, is always
//    a dataflow).
// Each candidate is timed with CUDA events on the case's own matrix at first
// use; choices are cached per size class (value size, log2 rows, entries per
// row), so later cases of the same class reuse them without timing.
#include <cmath>
#include <map>
#include <mutex>
#include <tuple>

#include "case.hpp"
#include "kernels.hpp"

namespace xcal {

namespace {
using TuneKey = std::tuple<int, int, int, int>;  // (kind, value bytes, log2 n, entries per row)
std::mutex g_tune_mu;
std::map<TuneKey, SpmvShape> g_spmv_choice;
std::map<TuneKey, int> g_dilu_choice;

TuneKey key_of(int kind, int tsize, const Equation& E) {
    int l2 = E.n > 0 ? (int)std::floor(std::log2((double)E.n)) : 0;
    int epr = E.n > 0 ? (int)std::lround((double)E.nnz_csr / E.n) : 0;
    return TuneKey(kind, tsize, l2, epr);
}
}  // namespace

// average device time (ms) of f over reps launches, after one warm-up
template <class F>
static float time_ms(cudaStream_t s, cudaEvent_t a, cudaEvent_t b, int reps, F&& f) {
    f();
    XCAL_CUDA(cudaEventRecord(a, s));
    for (int i = 0; i < reps; ++i) f();
    XCAL_CUDA(cudaEventRecord(b, s));
    XCAL_CUDA(cudaEventSynchronize(b));
    float ms = 0;
    XCAL_CUDA(cudaEventElapsedTime(&ms, a, b));
    return ms / reps;
}

template <class T>
static SpmvShape tune_spmv(Case& C, Equation& E, const T* nz, const T* x, T* y) {
    static const SpmvShape cands[] = {{0, 256}, {1, 128}, {1, 256}, {1, 512}, {2, 128},
                                      {2, 256}, {2, 512}, {4, 128}, {4, 256}, {4, 512}};
    const int reps = (int)std::max(3L, std::min(50L, 20000000L / std::max(E.nnz_csr, 1L)));
    CSRView A = E.view();
    SpmvShape best = cands[0];
    float best_ms = 1e30f;
    for (const SpmvShape& c : cands) {
        float ms = time_ms(C.stream, C.ev[6], C.ev[7], reps,
                           [&] { kr_spmv_shaped<T>(C.stream, c, A, nz, x, y, (const KScalars*)nullptr); });
        if (ms < best_ms) {
            best_ms = ms;
            best = c;
        }
    }
    return best;
}

// the fastest DILU form on this system: 2 one launch per level, 3 one
// cooperative launch over every level, 4 dataflow.  Up to 524,288 rows dataflow
// is taken as it is: measured on B200 (us per application, dataflow against
// the best other form) 27,025 rows FP64 37 / 88, 262,144 rows FP32 61 / 131;
// one-block sweeps come within reach only below some 4k rows (1,518 rows FP32
// 20.3 / 18.6), where the fused BiCGSTAB then shares one sweep among three
// components.  Above, both are timed (884,736 rows FP32: 117 / 155; 2.1M rows:
// 233 / 192, FP64 283 / 252).
constexpr int FLOW_UNTIMED_ROWS = 524288;
template <class T>
static int tune_dilu(Case& C, Equation& E, const T* nz, const T* D, const T* b, T* out) {
    const int reps = (int)std::max(3L, std::min(20L, 20000000L / std::max(E.nnz_csr, 1L)));
    const bool sb = E.use_block, sg = E.use_grid, sf = E.use_flow;
    kr_flow_unset(C.stream, C.flow_scratch<T>(out), (size_t)E.n * sizeof(T));
    int best = 4;
    float best_ms = 1e30f;
    for (int form = 2; form <= 4; ++form) {
        E.use_block = false;
        E.use_grid = form == 3;
        E.use_flow = form == 4;
        float ms = time_ms(C.stream, C.ev[6], C.ev[7], reps, [&] { C.dilu_ldiv(E, nz, D, b, out, nullptr); });
        if (ms < best_ms) {
            best_ms = ms;
            best = form;
        }
    }
    E.use_block = sb;
    E.use_grid = sg;
    E.use_flow = sf;
    return best;
}

void Case::autotune() {
    if (tuned || capturing) return;
    tuned = true;
    const bool mixed = cfg.precision == XCAL_PREC_MIXED;
    const int tsz = mixed ? 4 : 8;
    for (int e = 0; e < 2; ++e) {
        Equation& E = e == 0 ? U : P;
        const xcal_solver_setup& SS = e == 0 ? cfg.U_solver : cfg.p_solver;
        if (SS.solver == XCAL_SOLVER_BICGSTAB) {
            TuneKey k = key_of(0, tsz, E);
            std::unique_lock<std::mutex> lk(g_tune_mu);
            auto it = g_spmv_choice.find(k);
            if (it != g_spmv_choice.end()) {
                E.spmv_shape = it->second;
            } else {
                lk.unlock();
                SpmvShape sh = mixed ? tune_spmv<float>(*this, E, E.nz32.p, ws.fp.p, ws.fq.p)
                                     : tune_spmv<double>(*this, E, E.nz.p, ws.p.p, ws.q.p);
                E.spmv_shape = sh;
                lk.lock();
                g_spmv_choice[k] = sh;
            }
        }
        if (dilu_mode == 0 && SS.precond == XCAL_PRECOND_DILU) {
            TuneKey k = key_of(1, tsz, E);
            std::unique_lock<std::mutex> lk(g_tune_mu);
            auto it = g_dilu_choice.find(k);
            int form;
            if (E.n <= FLOW_UNTIMED_ROWS) {  // not in the cache: its class (524,288 rows) also holds sizes to be timed
                form = 4;
            } else if (it != g_dilu_choice.end()) {
                form = it->second;
            } else {
                lk.unlock();
                form = mixed ? tune_dilu<float>(*this, E, E.nz32.p, E.P32.p, ws.fr.p, ws.fz.p)
                             : tune_dilu<double>(*this, E, E.nz.p, E.P.p, ws.r.p, ws.z.p);
                lk.lock();
                g_dilu_choice[k] = form;
            }
            if (E.use_flow != (form == 4)) drop_graphs();  // chunks of earlier solves hold the other form
            E.use_block = form == 1;
            E.use_grid = form == 3;
            E.use_flow = form == 4;
        }
    }
    sync();
}

}  // namespace xcal
