// autotune.cu -- launch-shape autotuner.
//
// Tunes only choices that leave every result bit-identical:
//  * the row mapping and block size of the SpMVs that carry no reduction
//    (the BiCGSTAB SpMV): the canonical tile kernel or 1/2/4 rows per thread
//    in blocks of 128/256/512 threads;
//  * how a DILU application of a system of more than 524,288 rows runs: rows
//    waiting for the values they read (dataflow), one launch per level, or
//    every level in one cooperative launch with a grid barrier between levels
//    (smaller ones take the dataflow or, some FP32 ones, one-block sweeps
//    untimed; the fused BiCGSTAB, which shares the waits among components, is
//    always a dataflow).
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
// cooperative launch over every level, 4 dataflow (884,736 rows FP32, us per
// application, dataflow / the best other form: 117 / 155; 2.1M rows: 233 / 192,
// FP64 283 / 252).  Up to FLOW_UNTIMED_ROWS nothing is timed (untimed_form).
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

// Up to FLOW_UNTIMED_ROWS dataflow is taken as it is: measured on B200 (us per
// application, dataflow / the best other form) 27,025 rows FP64 37 / 88, 262,144
// rows FP32 61 / 131.  But an FP32 system of 512 to 4,095 rows whose solve
// applies DILU by itself (alone: a CG, or a smoothed BiCGSTAB; the fused one
// shares a dataflow among its components) takes one-block sweeps, 1: y in shared
// memory and one launch, not a cooperative one behind a memset.  Whole DILU-CG
// iterations, us, dataflow / one block, FP32: 250 rows 48.4 / 53.8, 512 rows
// 50.1 / 45.4, 1,073 rows 43.3 / 35.8, 1,920 rows 58.1 / 49.9, 3,072 rows 51.3 /
// 49.1, 4,160 rows 53.3 / 54.1, 5,984 rows 49.8 / 54.0; FP64 250 rows 35.4 / 40.4,
// 1,073 rows 36.8 / 38.2, 3,072 rows 47.1 / 54.4.  (Timed alone, back to back, the launch hides: the
// dataflow then looks faster at 1,920 rows too.)
static int untimed_form(int n, bool fp32, bool alone) {
    return fp32 && alone && n >= 512 && n < 4096 ? 1 : 4;
}

// all: also for an equation whose solves are fused now.  Those read neither
// choice, and the trials were most of a short first run's launches (two steps
// of the smoke case: 510 of 589); they are made once profiling, another DILU
// form or a smoother brings the separate kernels back.
void Case::autotune(bool all) {
    if (capturing) return;
    const bool mixed = cfg.precision == XCAL_PREC_MIXED;
    const int tsz = mixed ? 4 : 8;
    bool ran = false;
    for (int e = 0; e < 2; ++e) {
        Equation& E = e == 0 ? U : P;
        const xcal_solver_setup& SS = e == 0 ? cfg.U_solver : cfg.p_solver;
        // p's system also carries k, omega, kl and the wall distance
        const bool own = e == 0 || !(has_k() || has_y());
        if (E.tuned || (own && !all && use_fused(E, SS, false))) continue;
        E.tuned = ran = true;
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
            const bool alone = SS.solver == XCAL_SOLVER_CG || SS.smoother_loops > 0;
            TuneKey k = key_of(1, tsz, E);
            std::unique_lock<std::mutex> lk(g_tune_mu);
            auto it = g_dilu_choice.find(k);
            int form;
            if (E.n <= FLOW_UNTIMED_ROWS) {  // not in the cache: its class (524,288 rows) also holds sizes to be timed
                form = untimed_form(E.n, mixed, alone);
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
    if (ran) sync();
}

}  // namespace xcal
