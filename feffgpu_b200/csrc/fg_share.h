// fg_share.h -- the shared-matrix form (fg_shared.cuh) as the calls use it: a sub-batch's view of the workspace and the
// launches on it, instantiated in units of their own (fg_share_*.cu).
#pragma once
#include "fg_kernels.cuh"

namespace fg {

// The workspace of the shared and staged forms holds 16-byte words (records, keys, matrices); the one-kernel forms need no
// more than 8-byte alignment, so a call whose workspace does not start on a 16-byte boundary takes those.
inline bool share_aligned(const void *ws) { return (reinterpret_cast<uintptr_t>(ws) & 15) == 0; }

// The workspace as the kernels of one sub-batch see it.
template <typename R> struct Share : ShareIdx {
    unsigned char *rec;          // n records of rec_bytes (WarpPath<R>)
    size_t rec_bytes;
    int *two;                    // two-leg paths of the sub-batch (at most n)
    R *tab;                      // cls_cap rotation tables of tab_len entries
    int tab_len;
    unsigned char *F;            // the matrices: f_bytes
    size_t f_bytes;
    int chunks;                  // chunks of 32 energies
    int mats;                    // matrices kept per class: 1, or 4 with its derivatives (adjoint)
    int force;                   // this form is taken whatever the sharing (small calls)
    int by_path;                 // signals are stored by path (else by position in the sub-batch)
    __device__ __forceinline__ int64_t path(int64_t i) const { return order ? order[i] : i; }
    __device__ __forceinline__ int64_t row(int64_t i) const { return by_path ? path(i) : i; }
};

template <typename R, int EDGE>
Share<R> share_view(const SharePlan &pl, unsigned char *ws, ShareHead *head, const int *status, int L1)
{
    Share<R> s{};
    s.rec = ws + pl.rec; s.rec_bytes = geo_bytes<R>();
    s.key = pl.staged ? nullptr : reinterpret_cast<ShareKey *>(ws + pl.key);
    s.slot_of = reinterpret_cast<int *>(ws + pl.slot);
    s.hash = reinterpret_cast<unsigned *>(ws + pl.hash); s.hmask = pl.hcap - 1;
    s.cls = reinterpret_cast<int *>(ws + pl.cls);
    s.owner = reinterpret_cast<unsigned *>(ws + pl.owner); s.cls_cap = pl.cls_cap;
    s.two = reinterpret_cast<int *>(ws + pl.two);
    s.tab = reinterpret_cast<R *>(ws + pl.tab); s.tab_len = (L1 + 1) * dstride(pl.staged ? Kinds<EDGE>::MM : lamtab(Kinds<EDGE>::MS).MM);
    s.F = ws + pl.F; s.f_bytes = pl.f_bytes;
    s.chunks = pl.chunks; s.mats = pl.mats; s.force = pl.force; s.nsc_max = pl.nsc_max;
    s.head = head; s.status = status;
    return s;
}

// One sub-batch.  Where the shared form is not taken, signals goes on in the staged form, and adjoint sets head->general and
// writes nothing else; coords, ipots and the gradients are whole arrays indexed by path (order picks the sub-batch) or the
// sub-batch's own.
template <typename R, int EDGE> struct ShareLaunch {
    template <typename CT>
    static fg_status signals(const StageView &sv, const Tables<R> &T, const SharePlan &pl, Share<R> &s, const CT *coords,
                             const int64_t *ipots, int *status, C2<R> *out, cudaStream_t st);
    static fg_status fine(const StageView &sv, const Share<R> &s, const PathsDev &pd, int NK, const double *q,
                          const double *S, const int *span, unsigned char *pts, bool first, const C2<R> *sig,
                          unsigned long long *racc, double *reff_save, int *status, cudaStream_t st);
    static fg_status reff(const Share<R> &s, R *out, cudaStream_t st);
    template <typename CT>
    static fg_status adjoint(const StageView &sv, const Tables<R> &T, const SharePlan &pl, Share<R> &s, unsigned char *ws,
                             const CT *coords, const int64_t *ipots, int *status, const C2<R> *gbar,
                             const double *greff_d, const R *greff_r, double *gout_d, R *gout_r, cudaStream_t st);
};

// ------------------------------------------------------------------------------------------------ forward calls
// The one-kernel form of the drop-in call.
template <typename R, int EDGE, typename CT>
fg_status launch_cchi(const StageView &sv, const Tables<R> &T, int64_t B, int nleg, const CT *coords,
                      const int64_t *ipots, C2<R> *cchi, R *reff, int *bad, int warps, cudaStream_t st)
{
    using K = Kinds<EDGE>;
    const size_t wb = warp_bytes<R>(sv.L1, nleg - 1, nleg == 2 ? K::MMSS : K::MMMS, sv.E, false);
    warps = fit_warps(warps, wb, sv.max_smem);
    int blocks = 0;
    auto kern = k_cchi<R, EDGE, CT>;
    if (fg_status rc = grid_for(kern, warps * 32, wb * warps, sv.num_sms, B, blocks)) return rc;
    kern<<<blocks, warps * 32, wb * warps, st>>>(T, coords, ipots, B, nleg, cchi, reff, bad, wb);
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

template <typename R, int EDGE, typename CT>
fg_status cchi_call(const StageView &sv, const Tables<R> &T, int64_t B, int nleg, const CT *coords,
                    const int64_t *ipots, C2<R> *cchi, R *reff, int *bad, int warps, unsigned char *ws, size_t ws_bytes,
                    cudaStream_t st)
{
    const SharePlan pl = ws ? share_plan(B, nleg, sv.E, sv.L1, sizeof(R) == 8, sv.iorder, sv.ilinit) : SharePlan{};
    if constexpr (EDGE <= 3)
        if (pl.sub && ws_bytes >= kCounterBytes + pl.total && share_aligned(ws)) {
            ShareHead *head = reinterpret_cast<ShareHead *>(ws);
            Share<R> s = share_view<R, EDGE>(pl, ws + kCounterBytes, head, nullptr, sv.L1);
            s.stride = s.nleg_uniform = nleg;
            timer_begin(st);
            for (int64_t t0 = 0; t0 < B; t0 += pl.sub) {
                s.n = std::min<int64_t>(pl.sub, B - t0);
                const CT *c = coords + t0 * nleg * 3;
                const int64_t *ip = ipots + t0 * nleg;
                C2<R> *out = cchi + t0 * sv.E;
                if (fg_status rc = ShareLaunch<R, EDGE>::template signals<CT>(sv, T, pl, s, c, ip, bad, out, st)) return rc;
                if (fg_status rc = ShareLaunch<R, EDGE>::reff(s, reff + t0, st)) return rc;
            }
            timer_end(st);
            return FG_OK;
        }
    timer_begin(st);
    if (fg_status rc = launch_cchi<R, EDGE, CT>(sv, T, B, nleg, coords, ipots, cchi, reff, bad, warps, st)) return rc;
    timer_end(st);
    return FG_OK;
}

template <typename R, int EDGE>
fg_status Launch<R, EDGE>::cchi(const StageView &sv, const Tables<R> &T, int64_t B, int nleg, const void *coords,
                                int coords_f64, const int64_t *ipots, void *cchi, void *reff, int *bad, int warps,
                                unsigned char *ws, size_t ws_bytes, cudaStream_t st)
{
    C2<R> *c = static_cast<C2<R> *>(cchi);
    R *rf = static_cast<R *>(reff);
    if (coords_f64)
        return cchi_call<R, EDGE>(sv, T, B, nleg, static_cast<const double *>(coords), ipots, c, rf, bad, warps, ws, ws_bytes, st);
    return cchi_call<R, EDGE>(sv, T, B, nleg, static_cast<const float *>(coords), ipots, c, rf, bad, warps, ws, ws_bytes, st);
}

template <typename R, int EDGE>
fg_status Launch<R, EDGE>::fused(const StageView &sv, const Tables<R> &T, const fg_paths *P, int NK, const double *q,
                                 const double *S, const int *span, double *rows, void *cchi_save, double *reff_save,
                                 unsigned char *ws, const FusedShape &shape, cudaStream_t st,
                                 unsigned long long *words, unsigned char *share_ws, size_t share_bytes)
{
    unsigned long long *counter = reinterpret_cast<unsigned long long *>(ws);
    int *status = reinterpret_cast<int *>(ws + kStatusOffset);
    unsigned long long *racc = words ? words : reinterpret_cast<unsigned long long *>(ws + kCounterBytes);
    if (words) {
        FG_CUDA(cudaMemsetAsync(ws, 0, kCounterBytes, st));
        FG_CUDA(cudaMemsetAsync(words, 0, (size_t)2 * P->nrows * NK * sizeof(unsigned long long), st));
    } else {
        FG_CUDA(cudaMemsetAsync(ws, 0, kCounterBytes + row_sum_bytes(P->nrows, NK), st));
    }
    if (fg_status rc = launch_validate(P, sv.nph1, status, st)) return rc;
    const SharePlan pl = P->n > 0 ? share_plan(P->n, P->nleg_max, sv.E, sv.L1, sizeof(R) == 8, sv.iorder, sv.ilinit, false, NK) : SharePlan{};
    if (pl.sub && share_ws && share_bytes >= pl.total && share_aligned(share_ws)) {
        if constexpr (EDGE <= 3) {
            ShareHead *head = reinterpret_cast<ShareHead *>(ws + kShareHeadOffset);
            Share<R> s = share_view<R, EDGE>(pl, share_ws, head, status, sv.L1);
            s.stride = P->nleg_max;
            s.nlegs = P->nleg;
            s.by_path = cchi_save != nullptr;
            C2<R> *sig = cchi_save ? static_cast<C2<R> *>(cchi_save) : reinterpret_cast<C2<R> *>(share_ws + pl.sig);
            timer_begin(st);
            for (int64_t t0 = 0; t0 < P->n; t0 += pl.sub) {
                s.n = std::min<int64_t>(pl.sub, P->n - t0);
                s.order = P->order + t0;
                if (fg_status rc = ShareLaunch<R, EDGE>::template signals<double>(sv, T, pl, s, P->coords, P->ipots, status,
                                                                                  sig, st))
                    return rc;
                const PathsDev pd{s.n, P->nleg_max, P->nrows, P->coords, P->ipots, P->nleg, P->deg, P->sigma2, s.order, P->row};
                if (fg_status rc = ShareLaunch<R, EDGE>::fine(sv, s, pd, NK, q, S, span, share_ws + pl.pts, t0 == 0, sig, racc,
                                                              reff_save, status, st))
                    return rc;
            }
            timer_end(st);
        }
    } else if (P->n > 0) {
        const PathsDev pd{P->n, P->nleg_max, P->nrows, P->coords, P->ipots, P->nleg, P->deg, P->sigma2, P->order, P->row};
        timer_begin(st);
        if (fg_status rc = launch_fused<R, EDGE>(sv, T, pd, NK, q, S, span, racc, cchi_save, reff_save, counter, status,
                                                 shape, st))
            return rc;
        timer_end(st);
    }
    if (!rows) return FG_OK;
    return launch_row_finish(P->nrows, NK, racc, rows, status, st);
}

}  // namespace fg
