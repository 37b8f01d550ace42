// fg_shared.cuh -- the path signal with shared scattering matrices.
//
// A scattering matrix F~_k (before its Euler phase) depends on the leg before the scatterer, the leg after it, the
// angle between them and the scatterer's potential, and nothing else of the path: the path finder's lists of
// many-leg paths hold the same triplet of atoms again and again (the 189,419-path benchmark list: 790,095 scatterers,
// 49,088 different ones).  Here every different (leg length, next leg length, beta, potential) of a call, compared
// bit for bit, is one class; its matrix is formed once per energy and kept in the workspace, and the paths read it:
//
//   k_share_geom    a warp per path: geometry, Euler phases, termination rotations (the path's record), the keys
//   k_share_insert  a thread per scatterer: classes from a hash table of the keys (exact comparison)
//   k_share_tables  a thread per (class, rotation-table entry): D of every class
//   k_share_f       a warp per (class, 32 energies): the canonical entries of F~; two-leg paths' signals beside them
//   k_share_chain   a warp per (path, 32 energies): chain product, termination, cfac
//   k_share_fine    a warp per path (fused calls): fine grid and exact row sums
//
// Nothing outlives the call: classes are found anew from the call's coordinates.  The arithmetic of every value is
// that of the one-kernel form (k_fused, k_cchi): the results are the same bits.
//
// Measured on B200 (fused forward, 401 energies and k points): 128,844 paths of two to eight legs, 530,707 scatterers
// in 49,006 classes, mixed form 29.1 -> 12.3 ms (k_share_chain 8.2, k_share_f 2.1, k_share_fine 1.9 ms); 31,142 paths
// of up to seven legs, FP64 form 14.3 -> 5.65 ms.  What bounds it: the chain product's 144 complex multiply-adds per
// scatterer and energy and the 160 bytes (FP32) of matrix it reads for them, 4.3 TB/s from L2 and HBM.
#pragma once
#include "fg_kernels.cuh"

namespace fg {

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
    int force;                   // this form is taken whatever the sharing (small calls)
    int by_path;                 // signals are stored by path (else by position in the sub-batch)
    __device__ __forceinline__ int64_t path(int64_t i) const { return order ? order[i] : i; }
    __device__ __forceinline__ int64_t row(int64_t i) const { return by_path ? path(i) : i; }
};

// bytes of one class's matrices over one chunk
template <typename R, int KIND> __host__ __device__ constexpr size_t f_chunk_bytes()
{
    constexpr LamTab L = lamtab(KIND);
    return (size_t)RepTab<KIND, L.N, L.N>().n * sizeof(C2<R>) * 32;
}

// Chunks per pass that the matrices of all classes fit, 0: this form is not taken (too many classes, or too little
// shared between the paths); the same answer in every kernel of a call.
template <typename R, int KIND> __device__ __forceinline__ int share_chunks(const Share<R> &s)
{
    const int64_t U = s.head->classes, S = s.head->scatterers;
    if (U > s.cls_cap || (!s.force && U * kShareMin > S)) return 0;
    const size_t per = (size_t)max(U, (int64_t)1) * f_chunk_bytes<R, KIND>();
    return (int)min((size_t)s.chunks, s.f_bytes / per);
}

// A matrix's canonical entries, two complex FP32 (one FP64) per 16-byte word, words lane-contiguous.
template <typename R, int NE> __device__ __forceinline__ void store_f(unsigned char *at, int lane, const C2<R> (&f)[NE])
{
    if constexpr (sizeof(R) == 4) {
        static_assert(NE % 2 == 0, "pairs of entries");
#pragma unroll
        for (int i = 0; i < NE / 2; ++i)
            reinterpret_cast<float4 *>(at)[i * 32 + lane] = make_float4(f[2 * i].x, f[2 * i].y, f[2 * i + 1].x, f[2 * i + 1].y);
    } else {
#pragma unroll
        for (int i = 0; i < NE; ++i) reinterpret_cast<double2 *>(at)[i * 32 + lane] = make_double2(f[i].x, f[i].y);
    }
}
template <typename R, int NE> __device__ __forceinline__ void load_f(const unsigned char *at, int lane, C2<R> (&f)[NE])
{
    if constexpr (sizeof(R) == 4) {
#pragma unroll
        for (int i = 0; i < NE / 2; ++i) {
            const float4 v = reinterpret_cast<const float4 *>(at)[i * 32 + lane];
            f[2 * i] = C2<R>{v.x, v.y};
            f[2 * i + 1] = C2<R>{v.z, v.w};
        }
    } else {
#pragma unroll
        for (int i = 0; i < NE; ++i) {
            const double2 v = reinterpret_cast<const double2 *>(at)[i * 32 + lane];
            f[i] = C2<R>{v.x, v.y};
        }
    }
}

__device__ __forceinline__ void copy16(void *dst, const void *src, size_t bytes, int lane)
{
    for (size_t i = lane; i < bytes / 16; i += 32) static_cast<uint4 *>(dst)[i] = static_cast<const uint4 *>(src)[i];
}

// Records, keys and the list of two-leg paths (a batch that k_validate refused is left alone).
template <typename R, typename CT>
__global__ void __launch_bounds__(128) k_share_geom(Tables<R> T, Share<R> s, const CT *__restrict__ coords,
                                                    const int64_t *__restrict__ ipots, int *status, int MM_ss, int MM_ms)
{
    if (status && (*(volatile const int *)status & kBadLayout)) return;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    WarpPath<R> &g = *reinterpret_cast<WarpPath<R> *>(smem + (size_t)w * s.rec_bytes);
    for (int64_t i = (int64_t)blockIdx.x * 4 + w; i < s.n; i += (int64_t)gridDim.x * 4) {
        const int64_t p = s.path(i);
        const int nleg = s.legs(p);
        path_setup<R, CT>(g, nullptr, T, coords + p * s.stride * 3, ipots + p * s.stride, nleg, lane, status,
                          nleg == 2 ? MM_ss : MM_ms, false);
        copy16(s.rec + i * s.rec_bytes, &g, s.rec_bytes, lane);
        if (nleg == 2) {
            if (lane == 0) s.two[atomicAdd(&s.head->two, 1)] = (int)i;
        } else if (lane >= 1 && lane < nleg) {
            ShareKey k;
            k.x = (unsigned long long)__double_as_longlong(g.ri[lane]);
            k.y = (unsigned long long)__double_as_longlong(g.ri[lane + 1]);
            k.z = (unsigned long long)__double_as_longlong(g.beta[lane]);
            k.w = (unsigned long long)g.ip[lane];
            s.key[i * s.nsc_max + lane - 1] = k;
        }
        __syncwarp();
    }
}

// D of every class: a thread per (class, table entry), path_setup's recursion.
template <typename R, int KIND> __global__ void __launch_bounds__(128) k_share_tables(Tables<R> T, Share<R> s)
{
    constexpr int MM = lamtab(KIND).MM, NC = ncanon(MM), DS = dstride(MM);
    if (s.refused()) return;
    if (!share_chunks<R, KIND>(s)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) s.head->general = 1;       // the one-kernel form that follows runs
        return;
    }
    const int64_t tasks = (int64_t)s.head->classes * NC;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < tasks; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = i / NC;
        rotation_column<R>(s.tab + c * s.tab_len, T, __longlong_as_double((long long)s.key[s.owner[c]].z), MM, DS,
                           (int)(i % NC));
    }
}

// The matrices of one pass: items (class, chunk of the pass), a warp each, after the items (two-leg path, chunk),
// whose signal is formed here (their lambda sets are others, and they have one matrix that nothing shares).
template <typename R, int EDGE>
__global__ void __launch_bounds__(128) k_share_f(Tables<R> T, Share<R> s, int pass, C2<R> *__restrict__ out,
                                                 size_t wbytes)
{
    using K = Kinds<EDGE>;
    constexpr int KIND = K::MS;
    constexpr LamTab L = lamtab(KIND);
    constexpr RepTab<KIND, L.N, L.N> RT{};
    if (s.refused()) return;
    const int G = share_chunks<R, KIND>(s), g0 = pass * G;
    if (!G || g0 >= s.chunks) return;
    const int ng = min(G, s.chunks - g0), E = T.E;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned char *base = smem + (size_t)w * wbytes;
    const int64_t n_two = (int64_t)s.head->two * ng, items = n_two + (int64_t)s.head->classes * ng;
    for (int64_t it = (int64_t)blockIdx.x * nw + w; it < items; it += (int64_t)gridDim.x * nw) {
        if (it < n_two) {
            const int64_t i = s.two[it / ng];
            const int e = first_chunk(E) + 32 * (g0 + (int)(it % ng)) + lane;
            WarpPath<R> &g = *reinterpret_cast<WarpPath<R> *>(base);
            R *dh = reinterpret_cast<R *>(base + s.rec_bytes);
            copy16(base, s.rec + i * s.rec_bytes, s.rec_bytes, lane);
            __syncwarp();
            for (int r = lane; r < ncanon(K::MMSS); r += 32)
                rotation_column<R>(dh, T, g.beta[1], K::MMSS, dstride(K::MMSS), r);
            __syncwarp();
            if (e >= 0 && e < E) out[s.row(i) * E + e] = path_energy<R, EDGE>(g, dh, T, e, 2);
        } else {
            const int64_t c = (it - n_two) / ng;
            const int e = first_chunk(E) + 32 * (g0 + (int)((it - n_two) % ng)) + lane;
            R *dh = reinterpret_cast<R *>(base);
            copy16(dh, s.tab + c * s.tab_len, (size_t)s.tab_len * sizeof(R), lane);
            const ShareKey key = s.key[s.owner[c]];
            __syncwarp();
            if (e >= 0 && e < E) {
                const C2<R> ck = T.ck[e];
                if (fabs((double)ck.x) + fabs((double)ck.y) > 1e-16) {
                    const int ip = (int)key.w;
                    C2<R> acc[RT.n];
                    accumulate_f<R, KIND, L.N, L.N, sizeof(R) == 4 ? 2 : 1>(
                        acc, dh, T.tl + (size_t)ip * (T.L1 + 1) * E + e, E, T.lmax[ip * E + e] + 1,
                        zfac(cscl(ck, (R)__longlong_as_double((long long)key.y))),
                        zfac(cscl(ck, (R)__longlong_as_double((long long)key.x))));
                    mask_lambda<R, KIND, L.N, L.N>(acc, T.nlam);
                    store_f<R, RT.n>(s.F + (c * G + (it - n_two) % ng) * f_chunk_bytes<R, KIND>(), lane, acc);
                }
            }
        }
        __syncwarp();
    }
}

// The chain product, termination and cfac of one pass: items (path, part of the pass's chunks), a warp each.  split:
// parts per path (small calls split the energies over warps, large ones keep the path's record for all of a pass).
template <typename R, int EDGE>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 3 : 2)
    k_share_chain(Tables<R> T, Share<R> s, int pass, int split, C2<R> *__restrict__ out)
{
    using K = Kinds<EDGE>;
    constexpr int KIND = K::MS;
    constexpr LamTab L = lamtab(KIND);
    constexpr int N = L.N, N0 = L.N0, MM = L.MM;
    constexpr RepTab<KIND, N, N> RT{};
    if (s.refused()) return;
    const int G = share_chunks<R, KIND>(s), g0 = pass * G;
    if (!G || g0 >= s.chunks) return;
    const int ng = min(G, s.chunks - g0), E = T.E;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int cls_sh[4][kMaxLeg];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned char *base = smem + (size_t)w * s.rec_bytes;
    const WarpPath<R> &g = *reinterpret_cast<const WarpPath<R> *>(base);
    for (int64_t it = (int64_t)blockIdx.x * 4 + w; it < s.n * split; it += (int64_t)gridDim.x * 4) {
        const int64_t i = it / split, p = s.path(i), o = (s.by_path ? p : i) * E;
        const int nleg = s.legs(p), nsc = nleg - 1;
        if (nleg == 2) continue;
        copy16(base, s.rec + i * s.rec_bytes, s.rec_bytes, lane);
        if (lane < nsc) cls_sh[w][lane] = s.cls[s.slot_of[i * s.nsc_max + lane]];
        __syncwarp();
        for (int gc = (int)(it % split); gc < ng; gc += split) {
            const int e = first_chunk(E) + 32 * (g0 + gc) + lane;
            if (e < 0 || e >= E) continue;
            const C2<R> ck = T.ck[e];
            if (fabs((double)ck.x) + fabs((double)ck.y) <= 1e-16) {
                out[o + e] = cz<R>();
                continue;
            }
            C2<R> P[N][N0];
            for (int k = 1; k <= nsc; ++k) {
                C2<R> f[RT.n];
                load_f<R, RT.n>(s.F + ((int64_t)cls_sh[w][k - 1] * G + gc) * f_chunk_bytes<R, KIND>(), lane, f);
                C2<R> ph[2 * MM + 1];
                phase_powers<R, MM>(g.phs[k + 1], ph);
#pragma unroll
                for (int b = 0; b < N0; ++b) {
                    C2<R> col[N];
#pragma unroll
                    for (int a = 0; a < N; ++a) {
                        C2<R> v = cz<R>();
                        if (k == 1) {
                            v = RT.sg[a][b] > 0 ? f[RT.rep[a][b]] : cscl(f[RT.rep[a][b]], R(-1));
                        } else if (sizeof(R) == 8 || a < N0 || k < nsc) {   // the termination reads rows < N0 only
#pragma unroll
                            for (int c = 0; c < N; ++c) {
                                const C2<R> fv = f[RT.rep[a][c]];
                                v = RT.sg[a][c] > 0 ? cfma(fv, P[c][b], v) : cfms(fv, P[c][b], v);
                            }
                        }
                        col[a] = cmul(ph[L.m[a] + MM], v);
                    }
#pragma unroll
                    for (int a = 0; a < N; ++a) P[a][b] = col[a];
                }
            }
            const C2<R> ptrac = termination<R, KIND>(g, T, e, nleg, ck, [&](int b, int a) { return P[b][a]; });
            out[o + e] = cmul(ptrac, cfac(g, T, e, nleg, ck));
        }
        __syncwarp();
    }
}

// Fine grid and exact row sums of the fused calls from the paths' signals, as k_fused forms them.
template <typename R, int KIND>
__global__ void __launch_bounds__(128) k_share_fine(Share<R> s, PathsDev P, int E, int NK, const double *__restrict__ q,
                                                    const double *__restrict__ S, const int *__restrict__ span,
                                                    const C2<R> *__restrict__ cchi, unsigned long long *__restrict__ racc,
                                                    double *__restrict__ reff_save, int *status, size_t wbytes)
{
    if (s.refused() || !share_chunks<R, KIND>(s)) return;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double *pha = reinterpret_cast<double *>(smem + (size_t)w * wbytes);
    double *amp = pha + align_up((size_t)E, 2);
    for (int64_t i = (int64_t)blockIdx.x * nw + w; i < s.n; i += (int64_t)gridDim.x * nw) {
        const int64_t p = s.path(i);
        const C2<R> *c = cchi + (s.by_path ? p : i) * E;
        const double rf = reinterpret_cast<const WarpPath<R> *>(s.rec + i * s.rec_bytes)->reff * kBohr;
        path_terms<R>(P, p, E, NK, lane, q, S, span, [&](int e) { return c[e]; }, amp, pha, rf, racc, status);
        if (lane == 0 && reff_save) reff_save[p] = rf;
        __syncwarp();
    }
}

// reff of the drop-in call from the records
template <typename R, int KIND> __global__ void k_share_reff(Share<R> s, R *__restrict__ reff)
{
    if (!share_chunks<R, KIND>(s)) return;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < s.n; p += (int64_t)gridDim.x * blockDim.x)
        reff[p] = (R)(reinterpret_cast<const WarpPath<R> *>(s.rec + p * s.rec_bytes)->reff * kBohr);
}

// ------------------------------------------------------------------------------------------------ launches
template <typename R, int EDGE>
Share<R> share_view(const SharePlan &pl, unsigned char *ws, ShareHead *head, const int *status, int L1)
{
    Share<R> s{};
    s.rec = ws + pl.rec; s.rec_bytes = geo_bytes<R>();
    s.key = reinterpret_cast<ShareKey *>(ws + pl.key);
    s.slot_of = reinterpret_cast<int *>(ws + pl.slot);
    s.hash = reinterpret_cast<unsigned *>(ws + pl.hash); s.hmask = pl.hcap - 1;
    s.cls = reinterpret_cast<int *>(ws + pl.cls);
    s.owner = reinterpret_cast<unsigned *>(ws + pl.owner); s.cls_cap = pl.cls_cap;
    s.two = reinterpret_cast<int *>(ws + pl.two);
    s.tab = reinterpret_cast<R *>(ws + pl.tab); s.tab_len = (L1 + 1) * dstride(lamtab(Kinds<EDGE>::MS).MM);
    s.F = ws + pl.F; s.f_bytes = pl.f_bytes;
    s.chunks = pl.chunks; s.force = pl.force; s.nsc_max = pl.nsc_max;
    s.head = head; s.status = status;
    return s;
}

// The sub-batch's classes and the signals of its paths in out (n, E); where the form is not taken, head->general is set
// and out is left alone.  coords, ipots, nlegs: whole arrays (order picks the sub-batch) or the sub-batch's own.
template <typename R, int EDGE, typename CT>
fg_status share_signals(const StageView &sv, const Tables<R> &T, const SharePlan &pl, Share<R> &s, const CT *coords,
                        const int64_t *ipots, int *status, C2<R> *out, cudaStream_t st)
{
    using K = Kinds<EDGE>;
    constexpr int KIND = K::MS;
    FG_CUDA(cudaMemsetAsync(s.head, 0, sizeof(ShareHead), st));
    FG_CUDA(cudaMemsetAsync(s.hash, 0xff, (size_t)pl.hcap * sizeof(unsigned), st));
    const int blocks = (int)std::min<int64_t>((s.n + 3) / 4, (int64_t)sv.num_sms * 16);
    k_share_geom<R, CT><<<blocks, 128, 4 * s.rec_bytes, st>>>(T, s, coords, ipots, status, K::MMSS, K::MMMS);
    FG_CUDA(cudaGetLastError());
    if (fg_status rc = launch_share_insert(s, st)) return rc;
    const int64_t tasks = std::min<int64_t>(s.n * s.nsc_max, s.cls_cap) * ncanon(K::MMMS);
    k_share_tables<R, KIND><<<(int)std::min<int64_t>((tasks + 127) / 128, (int64_t)sv.num_sms * 16), 128, 0, st>>>(T, s);
    FG_CUDA(cudaGetLastError());
    const size_t wb = std::max(s.rec_bytes + align_up((size_t)(sv.L1 + 1) * dstride(K::MMSS) * sizeof(R), 16),
                               align_up((size_t)s.tab_len * sizeof(R), 16));
    auto kf = k_share_f<R, EDGE>;
    auto kc = k_share_chain<R, EDGE>;
    const int fw = fit_warps(4, wb, sv.max_smem);
    int fb = 0, cb = 0;
    if (fg_status rc = grid_for(kf, 32 * fw, wb * fw, sv.num_sms, s.n * s.nsc_max * pl.chunks, fb)) return rc;
    const int split = pl.split;
    if (fg_status rc = grid_for(kc, 128, 4 * s.rec_bytes, sv.num_sms, s.n * split, cb)) return rc;
    timer_begin(st);
    for (int pass = 0; pass < pl.passes; ++pass) {
        kf<<<fb, 32 * fw, wb * fw, st>>>(T, s, pass, out, wb);
        kc<<<cb, 128, 4 * s.rec_bytes, st>>>(T, s, pass, split, out);
    }
    timer_end(st);
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

// The one-kernel form of the drop-in call; gate as in launch_fused.
template <typename R, int EDGE, typename CT>
fg_status launch_cchi(const StageView &sv, const Tables<R> &T, int64_t B, int nleg, const CT *coords,
                      const int64_t *ipots, C2<R> *cchi, R *reff, int *bad, int warps, const int *gate, cudaStream_t st)
{
    using K = Kinds<EDGE>;
    const size_t wb = warp_bytes<R>(sv.L1, nleg - 1, nleg == 2 ? K::MMSS : K::MMMS, sv.E, false);
    warps = fit_warps(warps, wb, sv.max_smem);
    int blocks = 0;
    auto kern = k_cchi<R, EDGE, CT>;
    if (fg_status rc = grid_for(kern, warps * 32, wb * warps, sv.num_sms, B, blocks)) return rc;
    kern<<<blocks, warps * 32, wb * warps, st>>>(T, coords, ipots, B, nleg, cchi, reff, bad, wb, gate);
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
        if (pl.sub && ws_bytes >= kCounterBytes + pl.total) {
            ShareHead *head = reinterpret_cast<ShareHead *>(ws);
            Share<R> s = share_view<R, EDGE>(pl, ws + kCounterBytes, head, nullptr, sv.L1);
            s.stride = s.nleg_uniform = nleg;
            for (int64_t t0 = 0; t0 < B; t0 += pl.sub) {
                s.n = std::min<int64_t>(pl.sub, B - t0);
                const CT *c = coords + t0 * nleg * 3;
                const int64_t *ip = ipots + t0 * nleg;
                C2<R> *out = cchi + t0 * sv.E;
                if (fg_status rc = share_signals<R, EDGE, CT>(sv, T, pl, s, c, ip, bad, out, st)) return rc;
                k_share_reff<R, Kinds<EDGE>::MS><<<(int)std::min<int64_t>((s.n + 255) / 256, 148 * 4), 256, 0, st>>>(s, reff + t0);
                FG_CUDA(cudaGetLastError());
                if (!pl.force)
                    if (fg_status rc = launch_cchi<R, EDGE, CT>(sv, T, s.n, nleg, c, ip, out, reff + t0, bad, warps,
                                                                &head->general, st))
                        return rc;
            }
            return FG_OK;
        }
    timer_begin(st);
    if (fg_status rc = launch_cchi<R, EDGE, CT>(sv, T, B, nleg, coords, ipots, cchi, reff, bad, warps, nullptr, st)) return rc;
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
    using K = Kinds<EDGE>;
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
    const SharePlan pl = P->n > 0 ? share_plan(P->n, P->nleg_max, sv.E, sv.L1, sizeof(R) == 8, sv.iorder, sv.ilinit) : SharePlan{};
    if (pl.sub && share_ws && share_bytes >= pl.total) {
        if constexpr (EDGE <= 3) {
            ShareHead *head = reinterpret_cast<ShareHead *>(ws + kShareHeadOffset);
            Share<R> s = share_view<R, EDGE>(pl, share_ws, head, status, sv.L1);
            s.stride = P->nleg_max;
            s.nlegs = P->nleg;
            s.by_path = cchi_save != nullptr;
            C2<R> *sig = cchi_save ? static_cast<C2<R> *>(cchi_save) : reinterpret_cast<C2<R> *>(share_ws + pl.sig);
            auto kern = k_share_fine<R, K::MS>;
            const size_t wb = 2 * align_up((size_t)sv.E * sizeof(double), 16);
            const int warps = fit_warps(4, wb, sv.max_smem);
            for (int64_t t0 = 0; t0 < P->n; t0 += pl.sub) {
                s.n = std::min<int64_t>(pl.sub, P->n - t0);
                s.order = P->order + t0;
                if (fg_status rc = share_signals<R, EDGE, double>(sv, T, pl, s, P->coords, P->ipots, status, sig, st))
                    return rc;
                const PathsDev pd{s.n, P->nleg_max, P->nrows, P->coords, P->ipots, P->nleg, P->deg, P->sigma2, s.order, P->row};
                int blocks = 0;
                if (fg_status rc = grid_for(kern, 32 * warps, wb * warps, sv.num_sms, s.n, blocks)) return rc;
                kern<<<blocks, 32 * warps, wb * warps, st>>>(s, pd, sv.E, NK, q, S, span, sig, racc, reff_save, status, wb);
                FG_CUDA(cudaGetLastError());
                if (!pl.force) {
                    if (t0) FG_CUDA(cudaMemsetAsync(counter, 0, sizeof(*counter), st));
                    if (fg_status rc = launch_fused<R, EDGE>(sv, T, pd, NK, q, S, span, racc, cchi_save, reff_save, counter,
                                                             status, shape, &head->general, st))
                        return rc;
                }
            }
        }
    } else if (P->n > 0) {
        const PathsDev pd{P->n, P->nleg_max, P->nrows, P->coords, P->ipots, P->nleg, P->deg, P->sigma2, P->order, P->row};
        timer_begin(st);
        if (fg_status rc = launch_fused<R, EDGE>(sv, T, pd, NK, q, S, span, racc, cchi_save, reff_save, counter, status,
                                                 shape, nullptr, st))
            return rc;
        timer_end(st);
    }
    if (!rows) return FG_OK;
    return launch_row_finish(P->nrows, NK, racc, rows, status, st);
}

}  // namespace fg
