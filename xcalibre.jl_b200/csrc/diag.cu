// diag.cu -- device checks of the bounded waits the kernels use.
//
// A spin-wait gives up after a bounded number of polls, sets an error flag and
// its block leaves, so a value that never arrives ends in an error status the
// host reads (XCAL_ERR_TIMEOUT) instead of a hung GPU.  The checks make a wait
// run out, with a short poll limit and without any fault, and report that it
// gave up and that the context still runs work:
//   xcal_check_bounded_wait  the grid barrier: one block waits for a second
//                            that is never launched;
//   xcal_check_wait          the kernel named by `which`, on a system one of
//                            whose rows waits for a value nothing writes;
//   xcal_case_check_wait     that barrier with a case's own flag, which the
//                            case's next solve reports.
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

// The DILU factor of 600 rows in level order (3 chunks of 256), of which row 0
// needs its own D: its warp gives up, and the block with it
static bool check_dilu_factor(int spin_limit, int* err) {
    constexpr int n = 600;
    std::vector<int> rows(n), slice((n + SELL_C - 1) / SELL_C + 1, SELL_C), zero(n, 0);
    std::vector<unsigned char> cnt(n, 0);
    for (int k = 0; k < n; ++k) rows[k] = k;
    slice[0] = 0;
    cnt[0] = 1;
    DBuf<int> d_rows, d_slice, d_zero;  // zero: columns, slots and diagonal slots
    DBuf<unsigned char> d_cnt;
    DBuf<double> nz, D;
    DBuf<unsigned int> ticket;
    d_rows.upload(rows, 0);
    d_slice.upload(slice, 0);
    d_zero.upload(zero, 0);
    d_cnt.upload(cnt, 0);
    nz.alloc(1);
    nz.zero(0);
    D.alloc(n);
    ticket.alloc(1);
    LevelDView L{};
    L.rows = d_rows.p;
    L.slice = d_slice.p;
    L.cnt = d_cnt.p;
    L.col = L.src = L.tsrc = L.dslot = d_zero.p;
    kr_dilu_D_flow(0, n, L, nz.p, D.p, ticket.p, err, spin_limit);
    std::vector<double> h(n);
    XCAL_CUDA(cudaMemcpy(h.data(), D.p, n * sizeof(double), cudaMemcpyDeviceToHost));
    bool others = true;  // the other warps' rows were stored before the block left
    for (int k = SELL_C; k < n; ++k) others = others && h[k] == 0.0;
    return others && std::isnan(h[0]);
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
    if (!ctx || which != XCAL_WAIT_DILU_FACTOR || spin_limit < 1 || spin_limit > FLOW_SPIN_LIMIT)
        return XCAL_ERR_INVALID;
    try {
        XCAL_CUDA(cudaSetDevice(ctx->device));
        DBuf<int> err, out;
        err.alloc(1);
        err.zero(0);
        out.alloc(4);
        out.zero(0);
        const bool gave = check_dilu_factor((int)spin_limit, err.p);
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
