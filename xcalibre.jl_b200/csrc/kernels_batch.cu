// kernels_batch.cu -- batched Krylov kernels: one launch over the tiles of
// every system in a batch (block-diagonal system with per-system offsets).
// Each block looks up its (system, local tile) and runs the same tile body as
// the single-system kernel (krylov_bodies.cuh).
#include <vector>

#include <algorithm>

#include "batch.hpp"
#include "kernels.hpp"
#include "krylov_bodies.cuh"

namespace xcal {

#define XCAL_BSYS                                   \
    const int2 tm = tmap[blockIdx.x];               \
    const BSys<T>& B = sys[tm.x];                   \
    const TileCtx tc{tm.y, B.ntiles};

template <class T, int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbk_spmv(const BSys<T>* __restrict__ sys, const int2* tmap, int in,
                                                        int out) {
    XCAL_BSYS
    spmv_body<T, NT>(tc, B.A, B.nz, B.vec[in], B.vec[out], B.S);
}

template <class T, int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbk_jacobi_apply(const BSys<T>* __restrict__ sys, const int2* tmap, int in, int out, int use_S) {
    XCAL_BSYS
    jacobi_apply_body<T>(tc, B.n, B.P, B.vec[in], B.vec[out], use_S ? B.S : nullptr);
}

template <class T, int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbk_copy(const BSys<T>* __restrict__ sys, const int2* tmap, int in, int out, int use_S) {
    XCAL_BSYS
    copy_body<T>(tc, B.n, B.vec[in], B.vec[out], use_S ? B.S : nullptr);
}

// DILU sweeps of every system as a dataflow (krylov_bodies.cuh): the blocks
// draw (system, chunk of positions) items, listed in chunk order, from a
// ticket, so whatever a chunk waits for was drawn before it by a running
// block.  The systems' sweeps overlap, where one block per system had left
// the small ones waiting for the largest (16 serving cases, FP32: U solves
// 2.50 -> 1.40 ms per batch iteration).
template <class T, bool LOWER>
__global__ void __launch_bounds__(FLOW_THREADS) kbk_dilu_flow(const BSys<T>* __restrict__ sys,
                                                              const int2* __restrict__ items, int n_items,
                                                              unsigned int* ticket, int* err, int in, int out,
                                                              int use_S) {
    __shared__ int sh_item;
    for (bool ok = true;;) {
        const int t = flow_ticket(ticket, &sh_item, ok);
        if (t >= n_items) return;
        const int2 it = items[t];
        const BSys<T>& B = sys[it.x];
        if (use_S && B.S->done) continue;
        const int k0 = it.y * FLOW_THREADS + (threadIdx.x & ~31);
        ok = LOWER ? flow_lower_rows(B.n, B.lo, (const T*)B.vec[in], B.flow_y, B.vec[out], k0, err)
                   : flow_upper_rows(B.n, B.up, B.P, B.flow_y, B.vec[out], k0, err);
    }
}

template <class T, int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbk_cg_start(const BSys<T>* __restrict__ sys, const int2* tmap) {
    XCAL_BSYS
    cg_start_body<T, NT>(tc, B.n, B.vec[KV_R], B.vec[KV_Z], B.vec[KV_P], B.S, B.part0, B.ring);
}

template <class T, int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbk_cg_spmv(const BSys<T>* __restrict__ sys, const int2* tmap) {
    XCAL_BSYS
    cg_spmv_body<T, NT>(tc, B.A, B.nz, B.vec[KV_Z], B.vec[KV_P], B.vec[KV_V], B.vec[KV_Q], B.S, B.part0);
}

template <class T, int NT>
__global__ void __launch_bounds__(NT, NT > RED_THREADS ? 1 : sizeof(T) == 4 ? 4 : 8) kbk_cg_update(const BSys<T>* __restrict__ sys, const int2* tmap, int jacobi_fused) {
    XCAL_BSYS
    cg_update_body<T, NT>(tc, B.n, B.vec[KV_X], B.vec[KV_P], B.vec[KV_V], B.vec[KV_R], B.vec[KV_Q], B.vec[KV_Z], B.P,
                      jacobi_fused, B.S, B.part0);
}

template <class T, int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbk_cg_rz(const BSys<T>* __restrict__ sys, const int2* tmap) {
    XCAL_BSYS
    cg_rz_body<T, NT>(tc, B.n, B.vec[KV_R], B.vec[KV_Z], B.S, B.part0);
}

template <class T, int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbk_bicg_start(const BSys<T>* __restrict__ sys, const int2* tmap) {
    XCAL_BSYS
    bicg_start_body<T, NT>(tc, B.n, B.vec[KV_C], B.vec[KV_R], B.vec[KV_P], B.S, B.part0, B.part1);
}

template <class T, int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbk_bicg_alpha(const BSys<T>* __restrict__ sys, const int2* tmap) {
    XCAL_BSYS
    bicg_alpha_body<T, NT>(tc, B.n, B.vec[KV_C], B.vec[KV_V], B.S, B.part0);
}

template <class T, int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbk_bicg_s(const BSys<T>* __restrict__ sys, const int2* tmap) {
    XCAL_BSYS
    bicg_s_body<T>(tc, B.n, B.vec[KV_R], B.vec[KV_V], B.vec[KV_P], B.vec[KV_S], B.vec[KV_X], B.S);
}

template <class T, int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbk_bicg_omega(const BSys<T>* __restrict__ sys, const int2* tmap) {
    XCAL_BSYS
    bicg_omega_body<T, NT>(tc, B.n, B.vec[KV_T], B.vec[KV_S], B.S, B.part0, B.part1);
}

template <class T, int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbk_bicg_xr(const BSys<T>* __restrict__ sys, const int2* tmap) {
    XCAL_BSYS
    bicg_xr_body<T, NT>(tc, B.n, B.vec[KV_X], B.vec[KV_S], B.vec[KV_T], B.vec[KV_R], B.vec[KV_C], B.S, B.part0,
                    B.part1);
}

template <class T, int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbk_bicg_p(const BSys<T>* __restrict__ sys, const int2* tmap) {
    XCAL_BSYS
    bicg_p_body<T>(tc, B.n, B.vec[KV_R], B.vec[KV_V], B.vec[KV_P], B.S);
}

// every system's whole CG solve in one cooperative launch: the blocks of a
// system synchronise only among themselves (barrier state bars[2 s .. 2 s+1]),
// so systems finish independently
template <class T, int NT>
__global__ void __launch_bounds__(NT, persist_min_blocks(NT))
    kbk_cg_persist(const BSys<T>* __restrict__ sys, const int2* tmap, int jacobi, unsigned int* bars, int* err,
                   int max_iters) {
    XCAL_BSYS
    cg_persist_body<T, NT>(tc, B.A, B.nz, B.P, jacobi, B.vec[KV_X], B.vec[KV_R], B.vec[KV_Z], B.vec[KV_P],
                           B.vec[KV_V], B.S, B.part0, B.part1, bars + 2 * tm.x, err, max_iters, 0);
}

// every system's whole CG solve with its matrix in shared memory, one block
// per tile of the batch
template <class T>
__global__ void __launch_bounds__(RES_THREADS, 1)
    kbk_cg_resident(const BSys<T>* __restrict__ sys, const int2* tmap, int jacobi, int* err, int max_iters, int slots,
                    int halo) {
    extern __shared__ __align__(16) unsigned char res_smem[];
    XCAL_BSYS
    cg_resident_body<T, false>(tc, B.A, B.nz, B.P, jacobi, B.vec[KV_X], B.vec[KV_R], B.vec[KV_Z], B.vec[KV_P], B.S, B.ring,
                        err, max_iters, slots, halo, res_smem);
}

// the same for systems of at most 16 tiles, each the blocks of one cluster
template <class T>
__global__ void __launch_bounds__(RES_THREADS, 1)
    kbk_cg_resident_cl(const BSys<T>* __restrict__ sys, const int* __restrict__ ids, int C, int jacobi, int max_iters,
                       int slots, int halo) {
    extern __shared__ __align__(16) unsigned char res_smem[];
    const BSys<T>& B = sys[ids[blockIdx.x / C]];
    const TileCtx tc{(int)(blockIdx.x % C), B.ntiles};
    if (tc.tile >= tc.ntiles) return;
    cg_resident_body<T, true>(tc, B.A, B.nz, B.P, jacobi, B.vec[KV_X], B.vec[KV_R], B.vec[KV_Z], B.vec[KV_P], B.S,
                              nullptr, nullptr, max_iters, slots, halo, res_smem);
}

// cluster form: system ids[b / C] is the cluster of blocks b (rank b % C)
template <class T>
__global__ void __launch_bounds__(1024, 1) kbk_cg_persist_cl(const BSys<T>* __restrict__ sys,
                                                            const int* __restrict__ ids, int C, int jacobi,
                                                            int max_iters) {
    const BSys<T>& B = sys[ids[blockIdx.x / C]];
    const TileCtx tc{(int)(blockIdx.x % C), B.ntiles};
    cg_persist_body<T, 1024, true>(tc, B.A, B.nz, B.P, jacobi, B.vec[KV_X], B.vec[KV_R], B.vec[KV_Z], B.vec[KV_P],
                                   B.vec[KV_V], B.S, nullptr, nullptr, nullptr, nullptr, max_iters, 0);
}

// ---- per-case steps of a solve, batched (BAux tables) ----
#define XCAL_BAUX                                   \
    const int2 tm = tmap[blockIdx.x];               \
    const BAux& B = aux[tm.x];                      \
    const TileCtx tc{tm.y, B.ntiles};

// r0 = b - A field, x = 0, dx = field (k_init_resid)
template <int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbx_init_resid(const BAux* __restrict__ aux, const int2* tmap) {
    XCAL_BAUX
    tile_rows(tc, B.n, [&](int i) {
        B.r0[i] = B.b[i] - row_sum<NT>(B.A, B.nz, (const double*)B.field, i);
        B.x[i] = 0.0;
        B.dx[i] = B.field[i];
    });
}

// field = x + dx (k_finish)
template <int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbx_finish(const BAux* __restrict__ aux, const int2* tmap) {
    XCAL_BAUX
    tile_rows(tc, B.n, [&](int i) { B.field[i] = B.x[i] + B.dx[i]; });
}

// d32 = (float)(b - A field), x32 = 0 (k_defect)
template <int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbx_defect(const BAux* __restrict__ aux, const int2* tmap) {
    XCAL_BAUX
    tile_rows(tc, B.n, [&](int i) {
        B.d32[i] = (float)(B.b[i] - row_sum<NT>(B.A, B.nz, (const double*)B.field, i));
        B.x32[i] = 0.0f;
    });
}

// field += x32 unless the outer loop found the defect already at its target
// (k_correct; the case then leaves the outer loop uncorrected)
template <int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbx_correct(const BAux* __restrict__ aux, const int2* tmap) {
    XCAL_BAUX
    if (B.S->outer_conv) return;
    tile_rows(tc, B.n, [&](int i) { B.field[i] = B.field[i] + (double)B.x32[i]; });
}

// ||b - A field|| / max(||b||, 1 if tiny) per system (k_residual: the same
// tile trees, the last of the system's blocks finishes)
template <int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbx_residual(const BAux* __restrict__ aux, const int2* tmap) {
    XCAL_BAUX
    residual_body<NT>(tc, B.A, B.nz, (const double*)B.field, B.b, B.S, B.part0, B.part1, B.res_out);
}

// nz32 = (float) nz over the tile's slots (its rows' slices are contiguous),
// P32 = (float) P over its rows
template <int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbx_to_float(const BAux* __restrict__ aux, const int2* tmap) {
    XCAL_BAUX
    const int s0 = tc.tile * (RED_TILE / SELL_C);
    const int s1 = min(s0 + RED_TILE / SELL_C, (B.n + SELL_C - 1) / SELL_C);
    const int e1 = B.A.slice[s1];
#pragma unroll 4
    for (int e = B.A.slice[s0] + threadIdx.x; e < e1; e += NT) B.nz32[e] = (float)ld_stream(B.nz + e);
    if (B.P32) tile_rows(tc, B.n, [&](int i) { B.P32[i] = (float)B.P[i]; });
}

// level copies: slots of level positions in the tile (contiguous slices)
template <class T>
__device__ __forceinline__ void level_refresh_tile(const TileCtx& tc, int n, const int* slice, const int* src,
                                                   const T* nz, T* val, const int* col, const T* D, T* dinv) {
    const int s0 = tc.tile * (RED_TILE / SELL_C);
    const int s1 = min(s0 + RED_TILE / SELL_C, (n + SELL_C - 1) / SELL_C);
    const int e1 = slice[s1];
#pragma unroll 4
    for (int e = slice[s0] + threadIdx.x; e < e1; e += blockDim.x) {
        val[e] = nz[ld_stream(src + e)];
        if (dinv) dinv[e] = T(1) / D[ld_stream(col + e)];
    }
}

template <class T>
__device__ __forceinline__ void flow_unset_tile(const TileCtx& tc, int n, T* y) {
    tile_rows(tc, n, [&](int i) { y[i] = flow_unset_value<T>(); });
}

template <int NT>
__global__ void __launch_bounds__(NT, tile_min_blocks(NT)) kbx_level_refresh(const BAux* __restrict__ aux, const int2* tmap, int fp32) {
    XCAL_BAUX
    if (!B.lsrc) return;
    if (fp32) {
        level_refresh_tile<float>(tc, B.n, B.lslice, B.lsrc, B.nz32, B.lval32, B.lcol, B.P32, B.ldinv32);
        level_refresh_tile<float>(tc, B.n, B.uslice, B.usrc, B.nz32, B.uval32, nullptr, nullptr, nullptr);
        flow_unset_tile(tc, B.n, reinterpret_cast<float*>(B.flow_y));
    } else {
        level_refresh_tile<double>(tc, B.n, B.lslice, B.lsrc, B.nz, B.lval, B.lcol, B.P, B.ldinv);
        level_refresh_tile<double>(tc, B.n, B.uslice, B.usrc, B.nz, B.uval, nullptr, nullptr, nullptr);
        flow_unset_tile(tc, B.n, B.flow_y);
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
// a kernel over the batch's tiles, in the block size for that many (WIDE_TILES)
#define XCAL_XLAUNCH(K, ...)                                                 \
    do {                                                                     \
        if (ntiles_total <= 0) return;                                       \
        if (ntiles_total <= WIDE_TILES)                                      \
            K<WIDE_NT><<<ntiles_total, WIDE_NT, 0, s>>>(__VA_ARGS__);         \
        else                                                                 \
            K<RED_THREADS><<<ntiles_total, RED_THREADS, 0, s>>>(__VA_ARGS__); \
        XCAL_CHECK_LAUNCH();                                                 \
    } while (0)
void kb_init_resid(cudaStream_t s, const BAux* aux, const int2* tmap, int ntiles_total) {
    XCAL_XLAUNCH(kbx_init_resid, aux, tmap);
}
void kb_finish(cudaStream_t s, const BAux* aux, const int2* tmap, int ntiles_total) {
    XCAL_XLAUNCH(kbx_finish, aux, tmap);
}
void kb_defect(cudaStream_t s, const BAux* aux, const int2* tmap, int ntiles_total) {
    XCAL_XLAUNCH(kbx_defect, aux, tmap);
}
void kb_correct(cudaStream_t s, const BAux* aux, const int2* tmap, int ntiles_total) {
    XCAL_XLAUNCH(kbx_correct, aux, tmap);
}
void kb_residual(cudaStream_t s, const BAux* aux, const int2* tmap, int ntiles_total) {
    XCAL_XLAUNCH(kbx_residual, aux, tmap);
}
void kb_to_float(cudaStream_t s, const BAux* aux, const int2* tmap, int ntiles_total) {
    XCAL_XLAUNCH(kbx_to_float, aux, tmap);
}
void kb_level_refresh(cudaStream_t s, const BAux* aux, const int2* tmap, int ntiles_total, int fp32) {
    XCAL_XLAUNCH(kbx_level_refresh, aux, tmap, fp32);
}
#define XCAL_BLAUNCH(K, ...)                                                    \
    do {                                                                        \
        if (ntiles_total <= 0) return;                                          \
        if (ntiles_total <= WIDE_TILES)                                         \
            K<T, WIDE_NT><<<ntiles_total, WIDE_NT, 0, s>>>(__VA_ARGS__);         \
        else                                                                    \
            K<T, RED_THREADS><<<ntiles_total, RED_THREADS, 0, s>>>(__VA_ARGS__); \
        XCAL_CHECK_LAUNCH();                                                    \
    } while (0)

template <class T>
void kb_spmv(cudaStream_t s, const BSys<T>* sys, const int2* tmap, int ntiles_total, int in, int out) {
    XCAL_BLAUNCH(kbk_spmv, sys, tmap, in, out);
}
template <class T>
void kb_jacobi_apply(cudaStream_t s, const BSys<T>* sys, const int2* tmap, int ntiles_total, int in, int out,
                     int use_S) {
    XCAL_BLAUNCH(kbk_jacobi_apply, sys, tmap, in, out, use_S);
}
template <class T>
void kb_copy(cudaStream_t s, const BSys<T>* sys, const int2* tmap, int ntiles_total, int in, int out, int use_S) {
    XCAL_BLAUNCH(kbk_copy, sys, tmap, in, out, use_S);
}
template <class T>
void kb_dilu(cudaStream_t s, const BSys<T>* sys, const int2* items, int n_items, unsigned int* tickets, int* err,
             int in, int out, int use_S) {
    if (n_items <= 0) return;
    XCAL_CUDA(cudaMemsetAsync(tickets, 0, 2 * sizeof(unsigned int), s));
    const int g0 = std::max(1, std::min(flow_grid((const void*)kbk_dilu_flow<T, true>), n_items));
    const int g1 = std::max(1, std::min(flow_grid((const void*)kbk_dilu_flow<T, false>), n_items));
    kbk_dilu_flow<T, true><<<g0, FLOW_THREADS, 0, s>>>(sys, items, n_items, tickets, err, in, out, use_S);
    XCAL_CHECK_LAUNCH();
    kbk_dilu_flow<T, false><<<g1, FLOW_THREADS, 0, s>>>(sys, items, n_items, tickets + 1, err, in, out, use_S);
    XCAL_CHECK_LAUNCH();
}
template <class T>
bool kb_cg_persist(cudaStream_t s, const BSys<T>* sys, const int2* tmap, int ntiles_total, int jacobi,
                   unsigned int* bars, int nbars, int* err, int max_iters, int width) {
    static PersistCaps caps;
    static const void* const kern[3] = {(const void*)kbk_cg_persist<T, 1024>, (const void*)kbk_cg_persist<T, 512>,
                                        (const void*)kbk_cg_persist<T, RED_THREADS>};
    const int w = persist_pick(caps, kern, ntiles_total, width);
    if (w < 0) return false;
    XCAL_CUDA(cudaMemsetAsync(bars, 0, 2 * (size_t)nbars * sizeof(unsigned int), s));
    XCAL_CUDA(cudaMemsetAsync(err, 0, sizeof(int), s));
    void* args[] = {(void*)&sys, (void*)&tmap, &jacobi, &bars, &err, &max_iters};
    return persist_launch(caps, w, kern[w], ntiles_total, s, args);
}
template <class T>
bool kb_cg_resident(cudaStream_t s, const BSys<T>* sys, const int2* tmap, int ntiles_total, int slots, int halo,
                    int jacobi, int* err, int max_iters) {
    const void* k = (const void*)kbk_cg_resident<T>;
    if (slots <= 0 || halo > RES_HALO_MAX) return false;
    const size_t smem = res_smem_bytes<T>(slots, halo);
    if (ntiles_total <= 0 || ntiles_total > resident_sms(k, smem)) return false;
    XCAL_CUDA(cudaMemsetAsync(err, 0, sizeof(int), s));
    void* args[] = {(void*)&sys, (void*)&tmap, &jacobi, &err, &max_iters, &slots, &halo};
    return resident_launch(k, ntiles_total, smem, s, args);
}
template <class T>
int kb_cg_cluster_size(int tiles, int slots, int halo) {
    if (slots <= 0) return persist_cluster_size((const void*)kbk_cg_persist_cl<T>, tiles);
    const size_t smem = res_smem_bytes<T>(slots, halo);
    const void* k = (const void*)kbk_cg_resident_cl<T>;
    return halo <= RES_HALO_MAX && resident_sms(k, smem) > 0 ? persist_cluster_size(k, tiles, smem) : 0;
}
template <class T>
bool kb_cg_persist_cluster(cudaStream_t s, const BSys<T>* sys, const int* ids, int nsys, int max_tiles, int slots,
                           int halo, int jacobi, int max_iters) {
    const int C = kb_cg_cluster_size<T>(max_tiles, slots, halo);
    if (C == 0 || nsys <= 0) return false;
    int Cv = C;
    if (slots > 0) {
        void* args[] = {(void*)&sys, (void*)&ids, &Cv, &jacobi, &max_iters, &slots, &halo};
        persist_cluster_launch((const void*)kbk_cg_resident_cl<T>, C, nsys, s, args, res_smem_bytes<T>(slots, halo));
        return true;
    }
    const void* k = (const void*)kbk_cg_persist_cl<T>;
    void* args[] = {(void*)&sys, (void*)&ids, &Cv, &jacobi, &max_iters};
    persist_cluster_launch(k, C, nsys, s, args);
    return true;
}
template <class T>
void kb_cg_start(cudaStream_t s, const BSys<T>* sys, const int2* tmap, int ntiles_total) {
    XCAL_BLAUNCH(kbk_cg_start, sys, tmap);
}
template <class T>
void kb_cg_spmv(cudaStream_t s, const BSys<T>* sys, const int2* tmap, int ntiles_total) {
    XCAL_BLAUNCH(kbk_cg_spmv, sys, tmap);
}
template <class T>
void kb_cg_update(cudaStream_t s, const BSys<T>* sys, const int2* tmap, int ntiles_total, int jacobi_fused) {
    XCAL_BLAUNCH(kbk_cg_update, sys, tmap, jacobi_fused);
}
template <class T>
void kb_cg_rz(cudaStream_t s, const BSys<T>* sys, const int2* tmap, int ntiles_total) {
    XCAL_BLAUNCH(kbk_cg_rz, sys, tmap);
}
template <class T>
void kb_bicg_start(cudaStream_t s, const BSys<T>* sys, const int2* tmap, int ntiles_total) {
    XCAL_BLAUNCH(kbk_bicg_start, sys, tmap);
}
template <class T>
void kb_bicg_alpha(cudaStream_t s, const BSys<T>* sys, const int2* tmap, int ntiles_total) {
    XCAL_BLAUNCH(kbk_bicg_alpha, sys, tmap);
}
template <class T>
void kb_bicg_s(cudaStream_t s, const BSys<T>* sys, const int2* tmap, int ntiles_total) {
    XCAL_BLAUNCH(kbk_bicg_s, sys, tmap);
}
template <class T>
void kb_bicg_omega(cudaStream_t s, const BSys<T>* sys, const int2* tmap, int ntiles_total) {
    XCAL_BLAUNCH(kbk_bicg_omega, sys, tmap);
}
template <class T>
void kb_bicg_xr(cudaStream_t s, const BSys<T>* sys, const int2* tmap, int ntiles_total) {
    XCAL_BLAUNCH(kbk_bicg_xr, sys, tmap);
}
template <class T>
void kb_bicg_p(cudaStream_t s, const BSys<T>* sys, const int2* tmap, int ntiles_total) {
    XCAL_BLAUNCH(kbk_bicg_p, sys, tmap);
}

#define XCAL_BATCH_INSTANTIATE(T)                                                                                 \
    template void kb_spmv<T>(cudaStream_t, const BSys<T>*, const int2*, int, int, int);                            \
    template void kb_jacobi_apply<T>(cudaStream_t, const BSys<T>*, const int2*, int, int, int, int);               \
    template void kb_copy<T>(cudaStream_t, const BSys<T>*, const int2*, int, int, int, int);                       \
    template void kb_dilu<T>(cudaStream_t, const BSys<T>*, const int2*, int, unsigned int*, int*, int, int, int);  \
    template void kb_cg_start<T>(cudaStream_t, const BSys<T>*, const int2*, int);                                  \
    template bool kb_cg_persist<T>(cudaStream_t, const BSys<T>*, const int2*, int, int, unsigned int*, int, int*,  \
                                   int, int);                                                                     \
    template bool kb_cg_resident<T>(cudaStream_t, const BSys<T>*, const int2*, int, int, int, int, int*, int);     \
    template bool kb_cg_persist_cluster<T>(cudaStream_t, const BSys<T>*, const int*, int, int, int, int, int, int); \
    template int kb_cg_cluster_size<T>(int, int, int);                                                             \
    template void kb_cg_spmv<T>(cudaStream_t, const BSys<T>*, const int2*, int);                                   \
    template void kb_cg_update<T>(cudaStream_t, const BSys<T>*, const int2*, int, int);                            \
    template void kb_cg_rz<T>(cudaStream_t, const BSys<T>*, const int2*, int);                                     \
    template void kb_bicg_start<T>(cudaStream_t, const BSys<T>*, const int2*, int);                                \
    template void kb_bicg_alpha<T>(cudaStream_t, const BSys<T>*, const int2*, int);                                \
    template void kb_bicg_s<T>(cudaStream_t, const BSys<T>*, const int2*, int);                                    \
    template void kb_bicg_omega<T>(cudaStream_t, const BSys<T>*, const int2*, int);                                \
    template void kb_bicg_xr<T>(cudaStream_t, const BSys<T>*, const int2*, int);                                   \
    template void kb_bicg_p<T>(cudaStream_t, const BSys<T>*, const int2*, int);
XCAL_BATCH_INSTANTIATE(double)
XCAL_BATCH_INSTANTIATE(float)

}  // namespace xcal
