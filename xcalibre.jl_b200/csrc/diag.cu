// diag.cu -- device checks of the bounded waits the kernels use.
//
// A spin-wait gives up after a bounded number of polls, sets an error flag and
// its block leaves, so a value that never arrives ends in an error status the
// host reads (XCAL_ERR_TIMEOUT) instead of a hung GPU.  The checks make a wait
// run out, with a short poll limit and without any fault, and report that it
// gave up and that the context still runs work:
//   xcal_check_bounded_wait  the grid barrier: one block waits for a second
//                            that is never launched;
//   xcal_check_wait          the wait named by `which`, for a value nothing
//                            writes: the DILU factor's kernel, the batched
//                            sweeps' loop, the fused BiCGSTAB's wait and the
//                            resident CG's exchange;
//   xcal_case_check_wait     that barrier with a case's own flag, which the
//                            case's next solve reports.
#include <algorithm>
#include <cmath>
#include <vector>

#include "case.hpp"
#include "dev_common.cuh"
#include "krylov_bodies.cuh"

namespace xcal {

// one block, waiting for a second arrival that nothing makes
__global__ void k_wait_check(unsigned int* count, int* err, long spin_limit, int* out) {
    __shared__ int sh_err;
    unsigned int nb = 0;
    const bool ok = grid_barrier(count, 2, nb, err, &sh_err, spin_limit);
    if (threadIdx.x == 0) {
        out[0] = ok ? 0 : 1;
        out[1] = *(volatile int*)err;
    }
}

__global__ void k_wait_check_after(int* out) {
    if (threadIdx.x == 0) out[2] = 42;
}

// 600 rows in level order (3 chunks of 256), of which row 0 needs its own
// result: its warp gives up, and the block with it
struct SelfWait {
    static constexpr int n = 600;
    DBuf<int> rows, slice, zero;  // zero: columns, slots and diagonal slots
    DBuf<unsigned char> cnt;
    DBuf<double> vals, res, scratch;  // vals: matrix values and right-hand side, all 0
    DBuf<unsigned int> ticket;
    SelfWait() {
        std::vector<int> r(n), sl((n + SELL_C - 1) / SELL_C + 1, SELL_C);
        std::vector<unsigned char> c(n, 0);
        for (int k = 0; k < n; ++k) r[k] = k;
        sl[0] = 0;
        c[0] = 1;
        rows.upload(r, 0);
        slice.upload(sl, 0);
        cnt.upload(c, 0);
        zero.alloc(n);
        zero.zero(0);
        vals.alloc(n);
        vals.zero(0);
        res.alloc(n);
        kr_flow_unset(0, res.p, n * sizeof(double));
        scratch.alloc(n);
        scratch.zero(0);
        ticket.alloc(1);
        ticket.zero(0);
    }
    // row 0 has no result; its block stored those of its other warps and left
    bool gave_up() const {
        std::vector<double> h(n);
        XCAL_CUDA(cudaMemcpy(h.data(), res.p, n * sizeof(double), cudaMemcpyDeviceToHost));
        bool others = true;
        for (int k = SELL_C; k < n; ++k) others = others && h[k] == 0.0;
        return others && std::isnan(h[0]);
    }
};

static bool check_dilu_factor(int spin_limit, int* err) {
    SelfWait w;
    LevelDView L{};
    L.rows = w.rows.p;
    L.slice = w.slice.p;
    L.cnt = w.cnt.p;
    L.col = L.src = L.tsrc = L.dslot = w.zero.p;
    kr_dilu_D_flow(0, w.n, L, w.vals.p, w.res.p, w.ticket.p, err, spin_limit);
    return w.gave_up();
}

// the ticketed sweep of one system (kbk_dilu_flow's loop)
template <bool LOWER>
__global__ void __launch_bounds__(FLOW_THREADS) k_sweep_check(int n, LevelView<double> tri, const double* b, double* y,
                                                              double* out, unsigned int* ticket, int* err,
                                                              int spin_limit) {
    __shared__ int sh;
    const int chunks = (n + FLOW_THREADS - 1) / FLOW_THREADS;
    for (bool ok = true;;) {
        const int c = flow_ticket(ticket, &sh, ok);
        if (c >= chunks) return;
        const int k0 = c * FLOW_THREADS + (threadIdx.x & ~31);
        ok = LOWER ? flow_lower_rows(n, tri, b, y, out, k0, err, spin_limit)
                   : flow_upper_rows(n, tri, b, y, out, k0, err, spin_limit);
    }
}
template <bool LOWER>
static bool check_sweep(int spin_limit, int* err) {
    SelfWait w;
    std::vector<double> one(w.n, 1.0);
    DBuf<double> D;  // the upper rows' diagonal
    D.upload(one, 0);
    LevelView<double> t{};
    t.rows = w.rows.p;
    t.slice = w.slice.p;
    t.cnt = w.cnt.p;
    t.col = w.zero.p;
    t.val = t.dinv = w.vals.p;
    k_sweep_check<LOWER><<<2, FLOW_THREADS>>>(w.n, t, LOWER ? w.vals.p : D.p, LOWER ? w.res.p : w.scratch.p,
                                              LOWER ? w.scratch.p : w.res.p, w.ticket.p, err, spin_limit);
    XCAL_CHECK_LAUNCH();
    return w.gave_up();
}

// the resident CG's block of tile 0 of two, on the identity of 2,049 rows:
// the other tile's partial never comes
__global__ void __launch_bounds__(RES_THREADS, 1)
    k_resident_check(CSRView A, const double* nz, double* x, const double* r, double* z, const double* p, KScalars* S,
                     double* ring, int* err, int spin_limit) {
    extern __shared__ __align__(16) unsigned char res_smem[];
    cg_resident_body<double, false>(TileCtx{0, 2}, A, nz, (const double*)nullptr, 0, x, r, z, p, S, ring, err, 3,
                                    A.tile_slots, A.tile_halo, res_smem, spin_limit);
}
static bool check_resident(int spin_limit, int* err) {
    constexpr int n = RED_TILE + 1, nsl = (n + SELL_C - 1) / SELL_C;
    std::vector<int> slice(nsl + 1), col(nsl * SELL_C);
    for (int k = 0; k <= nsl; ++k) slice[k] = k * SELL_C;
    for (int k = 0; k < nsl * SELL_C; ++k) col[k] = std::min(k, n - 1);
    std::vector<unsigned char> len(n, 1);
    std::vector<double> one(nsl * SELL_C, 1.0);
    DBuf<int> d_slice, d_col, hoff;
    DBuf<unsigned char> d_len;
    DBuf<unsigned short> rowh;
    DBuf<double> nz, x, r, z, p, ring;
    DBuf<KScalars> S;
    d_slice.upload(slice, 0);
    d_col.upload(col, 0);
    d_len.upload(len, 0);
    hoff.alloc(3);
    hoff.zero(0);
    rowh.alloc(n);
    rowh.zero(0);
    for (DBuf<double>* b : {&nz, &r, &z, &p}) b->upload(one, 0);
    x.alloc(n);
    x.zero(0);
    ring.alloc(4 * 2 * 2);
    kr_flow_unset(0, ring.p, ring.n * sizeof(double));
    KScalars s{};
    s.gamma = s.pNorm2 = s.rNorm = n;
    s.itmax = 3;
    S.upload(&s, 1, 0);
    CSRView A{};
    A.n = n;
    A.slice = d_slice.p;
    A.len = d_len.p;
    A.colval = d_col.p;
    A.tile_slots = RED_TILE;
    A.hoff = hoff.p;
    A.rowh = rowh.p;
    const size_t smem = res_smem_bytes<double>(A.tile_slots, A.tile_halo);
    XCAL_CUDA(cudaFuncSetAttribute(k_resident_check, cudaFuncAttributeMaxDynamicSharedMemorySize, RES_SMEM_MAX));
    k_resident_check<<<1, RES_THREADS, smem>>>(A, nz.p, x.p, r.p, z.p, p.p, S.p, ring.p, err, spin_limit);
    XCAL_CHECK_LAUNCH();
    XCAL_CUDA(cudaMemcpy(&s, S.p, sizeof(s), cudaMemcpyDeviceToHost));
    return s.done == 0 && s.iter == 0;  // it left without a state to report
}

}  // namespace xcal

using namespace xcal;

extern "C" int32_t xcal_check_bounded_wait(xcal_ctx* ctx, int64_t spin_limit, int32_t* gave_up, int32_t* flag_set,
                                           int32_t* ran_after) {
    if (!ctx || spin_limit < 1 || spin_limit > BAR_SPIN_LIMIT) return XCAL_ERR_INVALID;
    try {
        XCAL_CUDA(cudaSetDevice(ctx->device));
        DBuf<unsigned int> count;
        DBuf<int> err, out;
        count.alloc(2);
        err.alloc(1);
        out.alloc(4);
        XCAL_CUDA(cudaMemset(count.p, 0, 2 * sizeof(unsigned int)));
        XCAL_CUDA(cudaMemset(err.p, 0, sizeof(int)));
        XCAL_CUDA(cudaMemset(out.p, 0, 4 * sizeof(int)));
        k_wait_check<<<1, 32>>>(count.p, err.p, (long)spin_limit, out.p);
        XCAL_CHECK_LAUNCH();
        k_wait_check_after<<<1, 32>>>(out.p);
        XCAL_CHECK_LAUNCH();
        XCAL_CUDA(cudaDeviceSynchronize());
        int h[4] = {0, 0, 0, 0};
        XCAL_CUDA(cudaMemcpy(h, out.p, sizeof(h), cudaMemcpyDeviceToHost));
        if (gave_up) *gave_up = h[0];
        if (flag_set) *flag_set = h[1];
        if (ran_after) *ran_after = h[2] == 42 ? 1 : 0;
        return XCAL_OK;
    } catch (const Error& e) {
        ctx->set_error(e.msg);
        return e.code;
    }
}

extern "C" int32_t xcal_check_wait(xcal_ctx* ctx, int32_t which, int64_t spin_limit, int32_t* gave_up,
                                   int32_t* flag_set, int32_t* ran_after) {
    static bool (*const checks[])(int, int*) = {check_dilu_factor, check_sweep<true>, check_sweep<false>,
                                                check_fused_wait, check_resident};
    if (!ctx || which < 0 || which > XCAL_WAIT_RESIDENT_CG || spin_limit < 1 || spin_limit > FLOW_SPIN_LIMIT)
        return XCAL_ERR_INVALID;
    try {
        XCAL_CUDA(cudaSetDevice(ctx->device));
        DBuf<int> err, out;
        err.alloc(1);
        err.zero(0);
        out.alloc(4);
        out.zero(0);
        const bool gave = checks[which]((int)spin_limit, err.p);
        k_wait_check_after<<<1, 32>>>(out.p);
        XCAL_CHECK_LAUNCH();
        int h[4] = {0, 0, 0, 0}, e = 0;
        XCAL_CUDA(cudaMemcpy(h, out.p, sizeof(h), cudaMemcpyDeviceToHost));
        XCAL_CUDA(cudaMemcpy(&e, err.p, sizeof(int), cudaMemcpyDeviceToHost));
        if (gave_up) *gave_up = gave ? 1 : 0;
        if (flag_set) *flag_set = e;
        if (ran_after) *ran_after = h[2] == 42 ? 1 : 0;
        return XCAL_OK;
    } catch (const Error& e) {
        ctx->set_error(e.msg);
        return e.code;
    }
}

extern "C" int32_t xcal_case_check_wait(xcal_case* cs, int64_t spin_limit) {
    if (!cs || spin_limit < 1 || spin_limit > BAR_SPIN_LIMIT) return XCAL_ERR_INVALID;
    Case* c = cs->c.get();
    try {
        XCAL_CUDA(cudaSetDevice(c->ctx->device));
        DBuf<unsigned int> count;
        DBuf<int> out;
        count.alloc(2);
        count.zero(c->stream);
        out.alloc(4);
        k_wait_check<<<1, 32, 0, c->stream>>>(count.p, c->ws.err.p, (long)spin_limit, out.p);
        XCAL_CHECK_LAUNCH();
        c->sync();
        return XCAL_OK;
    } catch (const Error& e) {
        c->ctx->set_error(e.msg);
        return e.code;
    }
}
