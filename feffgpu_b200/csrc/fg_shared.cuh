// fg_shared.cuh -- the path signal with shared scattering matrices.
//
// A scattering matrix F~_k (before its Euler phase) depends on the leg before the scatterer, the leg after it, the
// angle between them and the scatterer's potential, and nothing else of the path: the path finder's lists of
// many-leg paths hold the same triplet of atoms again and again (the 189,419-path benchmark list: 789,769 scatterers,
// 58,897 different ones).  Here every different (leg length, next leg length, beta, potential) of a call, compared
// bit for bit, is one class; its matrix is formed once per energy and kept in the workspace, and the paths read it:
//
//   k_share_geom    a thread per (path, leg): geometry, Euler phases, termination rotations (the path's record), the keys
//   k_share_insert  a thread per scatterer: classes from a hash table of the keys (exact comparison)
//   k_share_tables  a thread per (class, rotation-table entry): D of every class
//   k_share_f       a warp per (class, 32 energies): F~ in its two flip blocks; two-leg paths' signals beside them
//   k_share_chain   a warp per (path, 32 energies): chain product, termination, cfac
//   k_share_fine    a warp per range of paths (fused calls): fine grid and exact row sums
//
// Nothing outlives the call: classes are found anew from the call's coordinates.  The arithmetic of every value is
// that of the one-kernel form (k_fused, k_cchi): the results are the same bits.
//
// Measured on B200 (fused forward, 401 energies and k points): 128,844 paths of two to eight legs, 530,707 scatterers
// in 48,885 classes, mixed form 29.1 -> 9.4 ms (k_share_chain 5.2, k_share_f 2.5, k_share_fine 1.3 ms); 31,142 paths of up
// to seven legs, FP64 form 14.3 -> 4.5 ms.  What bounds the chain: issue (59 % of cycles) of its 80 complex multiply-adds
// a step and the latency of the 160 bytes (FP32) of matrix from L1 (38 % hits) and L2 (48 %); fetching the next matrix
// into shared memory while one is multiplied measured the same (5.3 ms), pair instructions 2 % slower, 128 MB passes
// instead of 1 GB 10 % slower.
#pragma once
#include "fg_adjoint.cuh"

namespace fg {

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
    const size_t per = (size_t)max(U, (int64_t)1) * s.mats * f_chunk_bytes<R, KIND>();
    return (int)min((size_t)s.chunks, s.f_bytes / per);
}

// A matrix's entries, two complex FP32 (one FP64) per 16-byte word, words lane-contiguous.
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

template <typename R> __device__ __forceinline__ ShareKey share_key(const WarpPath<R> &g, int k)
{
    return ShareKey{(unsigned long long)__double_as_longlong(g.ri[k]), (unsigned long long)__double_as_longlong(g.ri[k + 1]),
                    (unsigned long long)__double_as_longlong(g.beta[k]), (unsigned long long)g.ip[k]};
}

// The keys of path i's scatterers, or its entry in the list of two-leg paths
template <typename R>
__device__ __forceinline__ void share_keys(const Share<R> &s, const WarpPath<R> &g, int64_t i, int nleg, int lane)
{
    if (nleg == 2) {
        if (lane == 0) s.two[atomicAdd(&s.head->two, 1)] = (int)i;
    } else if (lane >= 1 && lane < nleg) {
        s.key[i * s.nsc_max + lane - 1] = share_key(g, lane);
    }
}

// Records, keys and the list of two-leg paths (a batch that k_validate refused is left alone).  A block takes PB paths
// at a time, a thread per (path, leg) where path_setup has a warp per path with a lane per leg: same operations, most of
// the lanes busy (128,844 paths of up to eight legs: 134 us, 292 us with a warp per path).
// KEYS: the keys and the list of two-leg paths alone (the adjoint, whose records are made once the form is taken), in as much
// of a record as they need (664 bytes FP32, so that shared memory does not limit the blocks).
template <typename R, bool KEYS> __host__ __device__ constexpr size_t geom_bytes(size_t rec_bytes)
{
    return KEYS ? (__builtin_offsetof(WarpPath<R>, dterm) + 15) / 16 * 16 : rec_bytes;
}
template <typename R, typename CT, bool KEYS>
__global__ void __launch_bounds__(128) k_share_geom(Tables<R> T, Share<R> s, const CT *__restrict__ coords,
                                                    const int64_t *__restrict__ ipots, int *status, int PB)
{
    if (s.refused()) return;            // not by status: the drop-in call's is the caller's word, whatever it holds
    extern __shared__ __align__(16) unsigned char smem[];
    const size_t rb = geom_bytes<R, KEYS>(s.rec_bytes);
    double *half = reinterpret_cast<double *>(smem + (size_t)PB * rb);               // cos, sin of beta_nleg / 2
    const int tid = threadIdx.x, nl = s.nsc_max + 1;
    auto rec = [&](int l) -> WarpPath<R> & { return *reinterpret_cast<WarpPath<R> *>(smem + (size_t)l * rb); };
    for (int64_t i0 = (int64_t)blockIdx.x * PB; i0 < s.n; i0 += (int64_t)gridDim.x * PB) {
        const int cnt = (int)min((int64_t)PB, s.n - i0);
        for (int t = tid; t < cnt * nl * 3; t += 128) {
            const int l = t / (3 * nl), r = t % (3 * nl);
            const int64_t p = s.path(i0 + l);
            if (r < 3 * s.legs(p)) rec(l).xyz[r / 3][r % 3] = (double)coords[p * s.stride * 3 + r] / kBohr;
        }
        for (int t = tid; t < cnt * (nl + 1); t += 128) {
            const int l = t / (nl + 1), j = t % (nl + 1);
            const int64_t p = s.path(i0 + l);
            const int nleg = s.legs(p);
            if (j > nleg) continue;
            int64_t v = ipots[p * s.stride + (j == nleg ? 0 : j)];
            if (v < 0 || v >= T.nph1) {
                if (status) atomicOr(status, kBadIpot);
                v = v < 0 ? 0 : T.nph1 - 1;
            }
            rec(l).ip[j] = (int)v;
        }
        __syncthreads();
        for (int t = tid; t < cnt * nl; t += 128) {
            const int l = t / nl, j = t % nl + 1, nleg = s.legs(s.path(i0 + l));
            if (j > nleg) continue;
            WarpPath<R> &g = rec(l);
            auto rat = [&](int i, double *o) {
                const int a = (i == 0 || i == nleg) ? 0 : i;
                o[0] = g.xyz[a][0]; o[1] = g.xyz[a][1]; o[2] = g.xyz[a][2];
            };
            const LegGeom lg = leg_geometry<double>(rat, j, nleg);
            g.ri[j] = lg.ri; g.beta[j] = lg.beta; g.alpha[j] = lg.alpha; g.gamma[j] = lg.gamma;
            if (!KEYS && j == nleg) {
                half[2 * l] = cos(0.5 * lg.beta);
                half[2 * l + 1] = sin(0.5 * lg.beta);
            }
        }
        __syncthreads();
        for (int t = tid; t < cnt * nl; t += 128) {
            const int l = t / nl, j = t % nl + 1, nleg = s.legs(s.path(i0 + l));
            if (j > nleg) continue;
            WarpPath<R> &g = rec(l);
            if constexpr (!KEYS) {
                const double eta = g.alpha[j == 1 ? nleg : j - 1] + g.gamma[j];
                double sn, cs;
                sincos(eta, &sn, &cs);
                g.phs[j] = C2<R>{(R)cs, (R)(-sn)};
                if (j == 1) {
                    double r = 0.0;
                    for (int q = 1; q <= nleg; ++q) r += g.ri[q];
                    g.reff = 0.5 * r;
                }
            }
            if (s.key) {
                if (nleg == 2) {
                    if (j == 1) s.two[atomicAdd(&s.head->two, 1)] = (int)(i0 + l);
                } else if (j < nleg) {
                    s.key[(i0 + l) * s.nsc_max + j - 1] = share_key(g, j);
                }
            }
        }
        if constexpr (!KEYS) {
            for (int t = tid; t < cnt * T.nterm * 49; t += 128) {
                const int l = t / (T.nterm * 49), q = t % (T.nterm * 49), e = q % 49;
                rec(l).dterm[q / 49][e] = (R)wigner_small(T.term_l[q / 49], e / 7 - 3, e % 7 - 3, half[2 * l],
                                                          half[2 * l + 1], seed_table(T));
            }
            __syncthreads();
            for (size_t t = tid; t < cnt * s.rec_bytes / 16; t += 128)
                reinterpret_cast<uint4 *>(s.rec + i0 * s.rec_bytes)[t] = reinterpret_cast<const uint4 *>(smem)[t];
        }
        __syncthreads();
    }
}

// D of every class: a thread per (class, table entry), path_setup's recursion.
template <typename R, int KIND> __global__ void __launch_bounds__(128) k_share_tables(Tables<R> T, Share<R> s)
{
    constexpr int MM = lamtab(KIND).MM, NC = ncanon(MM), DS = dstride(MM);
    if (s.refused()) return;
    if (!share_chunks<R, KIND>(s)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) s.head->general = 1;       // the staged kernels that follow run
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
                    C2<R> f[20];
                    to_blocks<R, KIND, L.N, L.N>(acc, f);
                    store_f<R, 20>(s.F + (c * G + (it - n_two) % ng) * f_chunk_bytes<R, KIND>(), lane, f);
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
    constexpr int N0 = L.N0;
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
            C2<R> P[N0][6];                                  // columns, in the flip basis
            for (int k = 1; k <= nsc; ++k) {
                C2<R> f[20];
                load_f<R, 20>(s.F + ((int64_t)cls_sh[w][k - 1] * G + gc) * f_chunk_bytes<R, KIND>(), lane, f);
                const C2<R> e1 = g.phs[k + 1], e2 = cmul(e1, e1);
                if (k == 1) {
#pragma unroll
                    for (int c = 0; c < N0; ++c) block_first<R, KIND>(f, e1, e2, c, P[c]);
                } else {
#pragma unroll
                    for (int c = 0; c < N0; ++c) block_step<R, KIND>(f, e1, e2, k < nsc, P[c]);
                }
            }
            C2<R> Q[N0][N0];
            from_blocks<R, KIND>([&](int c, int i) { return P[c][i]; }, Q);
            const C2<R> ptrac = termination<R, KIND>(g, T, e, nleg, ck, [&](int b, int a) { return Q[b][a]; });
            out[o + e] = cmul(ptrac, cfac(g, T, e, nleg, ck));
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------------------------------------ staged form
// Lists of up to three legs (MD trajectories) share nothing, but k_fused spends more than half its time there on what is
// done once per path -- geometry, rotation tables, the fine grid -- at the eight warps per SM that its energy loop allows.
// The staged form gives each part a kernel of its own shape: k_share_geom, the tables by a thread per (scatterer, entry)
// into the workspace, the energies by a warp per path with record and tables copied in, then k_share_fine.  537,000 paths
// of 2,048 absorbers, 60 energies, 401 points, mixed: 15.0 -> 9.5 ms (energies 5.5, fine grid 1.9, tables 1.1, geometry
// 0.7 ms); 4,438 paths of up to four legs: 178 -> 140 us.  What bounds it: the energies' FP32 multiply-adds and their
// fixed latencies at 12 (three legs) and 8 warps per SM.
//
// The kernels take the positions i0 .. i0 + n of the sub-batch, whose tables (tab_len entries a scatterer) are at tab; gate:
// they return at once unless *gate is set (the shared form's kernels, which ran before them, found too little to share).
template <typename R> struct StagePart {
    R *tab;
    int tab_len;
    int64_t i0, n;
    const int *gate;
    __device__ __forceinline__ bool off(const Share<R> &s) const
    {
        return s.refused() || (gate && !*(volatile const int *)gate);
    }
};

template <typename R, int EDGE>
__global__ void __launch_bounds__(128) k_stage_tables(Tables<R> T, Share<R> s, StagePart<R> part)
{
    using K = Kinds<EDGE>;
    constexpr int NC = ncanon(K::MM);
    if (part.off(s)) return;
    const int64_t tasks = part.n * s.nsc_max * NC;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < tasks; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = t / NC, i = part.i0 + c / s.nsc_max;
        const int r = (int)(t % NC), k = (int)(c % s.nsc_max) + 1, nleg = s.legs(s.path(i));
        const int MM = nleg == 2 ? K::MMSS : K::MMMS;
        if (k >= nleg || r >= ncanon(MM)) continue;
        const WarpPath<R> &g = *reinterpret_cast<const WarpPath<R> *>(s.rec + i * s.rec_bytes);
        rotation_column<R>(part.tab + c * part.tab_len, T, g.beta[k], MM, dstride(MM), r);
    }
}

// SHORT: no path has more than three legs
template <typename R, int EDGE, bool SHORT>
__global__ void __launch_bounds__(128, FusedMinBlocks<R>::def) k_stage_energies(Tables<R> T, Share<R> s, StagePart<R> part,
                                                                                int split, C2<R> *__restrict__ out,
                                                                                size_t wbytes)
{
    using K = Kinds<EDGE>;
    if (part.off(s)) return;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5, E = T.E;
    unsigned char *base = smem + (size_t)w * wbytes;
    const WarpPath<R> &g = *reinterpret_cast<const WarpPath<R> *>(base);
    R *dh = reinterpret_cast<R *>(base + s.rec_bytes);
    // all paths' first part of the energies, then the next part: parts differ by a chunk, and every warp gets of each
    for (int64_t it = (int64_t)blockIdx.x * nw + w; it < part.n * split; it += (int64_t)gridDim.x * nw) {
        const int64_t j = it % part.n, i = part.i0 + j, o = s.row(i) * E;
        const int nleg = s.legs(s.path(i)), MM = nleg == 2 ? K::MMSS : K::MMMS;
        copy16(base, s.rec + i * s.rec_bytes, s.rec_bytes, lane);
        // the tables of a path's scatterers, one after the other as the energies read them
        const int len = (T.L1 + 1) * dstride(MM);
        for (int k = 0; k < nleg - 1; ++k)
            copy16(dh + k * len, part.tab + (j * s.nsc_max + k) * part.tab_len, (size_t)len * sizeof(R), lane);
        __syncwarp();
        for (int gc = (int)(it / part.n); gc < s.chunks; gc += split) {
            const int e = first_chunk(E) + 32 * gc + lane;
            if (e < 0 || e >= E) continue;
            if (nleg > 2) {
                if constexpr (SHORT) out[o + e] = energy_ms3<R, K::MS>(g, dh, T, e);
                else out[o + e] = energy_ms<R, K::MS>(g, dh, T, e, nleg);
            } else {
                if constexpr (K::SS_SYM) out[o + e] = energy_ss_sym<R, K::SS>(g, dh, T, e);
                else out[o + e] = energy_ss_col<R, K::SS>(g, dh, T, e);
            }
        }
        __syncwarp();
    }
}

// A fine-grid point's interpolation: the weights of its first two energies (S rows with more are read from S)
struct __align__(16) FinePoint {
    double w0, w1, q;
    int lo, n;
};
static __global__ void k_fine_points(int NK, int E, const double *__restrict__ q, const double *__restrict__ S,
                              const int *__restrict__ span, FinePoint *__restrict__ out)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= NK) return;
    FinePoint f;
    f.lo = span[2 * k];
    f.n = span[2 * k + 1] - f.lo;
    f.q = q[k];
    f.w0 = f.n > 0 ? S[(size_t)k * E + f.lo] : 0.0;
    f.w1 = f.n > 1 ? S[(size_t)k * E + f.lo + 1] : 0.0;
    out[k] = f;
}

// Fine grid and exact row sums of the fused calls from the paths' signals, value for value as k_fused forms them
// (path_terms).  A warp takes a contiguous range of the sub-batch's paths, PG at a time, so that a fine-grid point's
// interpolation is read once for all of them.  Integer sums give the same in any order: with ACC the terms of one row are
// added in the warp's shared memory, and only its sums go to the row's words, those of neighbouring warps first added
// together -- a row's 401 points take one addition each per block and not per path, which is what a small batch on one row
// waits for: 4,438 paths on 60 energies 84 -> 25 us; 537,000 paths on 64 rows 2.29 -> 1.94 ms (4.3 ms a warp per path with
// S read in place).  On 401 energies (128,844 paths, 1.29 ms) the FP64 arc tangents and square roots of the phases bound it.
template <typename R, int PG, bool ACC>
__global__ void __launch_bounds__(256, PG == 1 ? 4 : 2)          // the blocks that the records and sums leave room for
    k_share_fine(Share<R> s, PathsDev P, int E, int NK, const double *__restrict__ S, const FinePoint *__restrict__ pts,
                 const C2<R> *__restrict__ cchi, unsigned long long *__restrict__ racc, double *__restrict__ reff_save,
                 int *status, int64_t range, size_t wbytes)
{
    if (s.refused()) return;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int last_row[8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5, E2 = (E + 1) & ~1;
    auto words = [&](int v) {
        return reinterpret_cast<ulonglong2 *>(smem + (size_t)v * wbytes + (size_t)2 * PG * E2 * sizeof(double));
    };
    double *pha = reinterpret_cast<double *>(smem + (size_t)w * wbytes), *amp = pha + PG * E2;
    const size_t stride = (size_t)P.nrows * NK;
    auto add = [&](int row, int k, unsigned long long hi, unsigned long long lo) {
        atomicAdd(racc + (size_t)row * NK + k, hi);
        atomicAdd(racc + (size_t)row * NK + k + stride, lo);
    };
    const int64_t lo_i = min(s.n, ((int64_t)blockIdx.x * nw + w) * range), hi_i = min(s.n, lo_i + range);
    int cur = -1;                                    // the row whose terms the warp's words hold (ACC)
    for (int64_t i0 = lo_i; i0 < hi_i; i0 += PG) {
        const int cnt = (int)min((int64_t)PG, hi_i - i0);
        double rf[PG], wdeg[PG], s2[PG];
        int row[PG];
#pragma unroll
        for (int j = 0; j < PG; ++j) {
            if (j >= cnt) break;
            const int64_t p = s.path(i0 + j);
            const C2<R> *c = cchi + (s.by_path ? p : i0 + j) * E;
            amp_phase<R>(E, lane, [&](int e) { return c[e]; }, amp + j * E2, pha + j * E2);
            rf[j] = reinterpret_cast<const WarpPath<R> *>(s.rec + (i0 + j) * s.rec_bytes)->reff * kBohr;
            wdeg[j] = P.deg[p];
            s2[j] = P.sigma2 ? P.sigma2[p] : 0.0;
            row[j] = P.row[p];
            if (lane == 0 && reff_save) reff_save[p] = rf[j];
        }
        __syncwarp();
        int next = cur;
        for (int k0 = 0; k0 < NK; k0 += 32) {
            const int k = k0 + lane;
            next = cur;
            if (k < NK) {
                const FinePoint f = pts[k];
                unsigned long long hi = 0, lo = 0;
                if (ACC && cur >= 0) {
                    const ulonglong2 v = words(w)[k];
                    hi = v.x;
                    lo = v.y;
                }
#pragma unroll
                for (int j = 0; j < PG; ++j) {
                    if (j >= cnt) break;
                    if (row[j] != next) {            // the sums so far go to their row
                        if (next >= 0) add(next, k, hi, lo);
                        hi = lo = 0;
                        next = row[j];
                    }
                    const double *a_ = amp + j * E2 + f.lo, *p_ = pha + j * E2 + f.lo;
                    double a = 0.0, ph = 0.0;
                    if (f.n <= 2) {
                        if (f.n > 0) { a += f.w0 * a_[0]; ph += f.w0 * p_[0]; }
                        if (f.n > 1) { a += f.w1 * a_[1]; ph += f.w1 * p_[1]; }
                    } else {
                        for (int m = 0; m < f.n; ++m) {
                            const double sv = S[(size_t)k * E + f.lo + m];
                            a += sv * a_[m];
                            ph += sv * p_[m];
                        }
                    }
                    const double damp = s2[j] != 0.0 ? exp(-2.0 * s2[j] * f.q * f.q) : 1.0;   // exact 1 without sigma^2
                    const double v = wdeg[j] * a * sin_arg<R>(ph + 2.0 * f.q * rf[j]) * damp;
                    if (!fixed_words(v, hi, lo)) atomicOr(status, kBadRange);
                }
                if (ACC) words(w)[k] = make_ulonglong2(hi, lo);
                else add(next, k, hi, lo);
            }
        }
        if (ACC) cur = row[cnt - 1];
        __syncwarp();
    }
    if (!ACC) return;
    if (lane == 0) last_row[w] = cur;
    __syncthreads();
    for (int k = threadIdx.x; k < NK; k += blockDim.x) {
        unsigned long long hi = 0, lo = 0;
        for (int v = 0; v < nw; ++v) {
            if (last_row[v] < 0) continue;
            const ulonglong2 x = words(v)[k];
            hi += x.x;
            lo += x.y;
            if (v + 1 == nw || last_row[v + 1] != last_row[v]) {
                add(last_row[v], k, hi, lo);
                hi = lo = 0;
            }
        }
    }
}

// reff of the drop-in call from the records
template <typename R> __global__ void k_share_reff(Share<R> s, R *__restrict__ reff)
{
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < s.n; p += (int64_t)gridDim.x * blockDim.x)
        reff[p] = (R)(reinterpret_cast<const WarpPath<R> *>(s.rec + p * s.rec_bytes)->reff * kBohr);
}

// ------------------------------------------------------------------------------------------------ launches
// Records, keys and two-leg list (or the keys alone): paths per block such that a thread has a leg, fewer where the paths
// do not fill the chip that way.
template <bool KEYS, typename R, typename CT>
fg_status launch_geom(const StageView &sv, const Tables<R> &T, const Share<R> &s, const CT *coords, const int64_t *ipots,
                      int *status, cudaStream_t st)
{
    const int PB = (int)std::max<int64_t>(1, std::min<int64_t>(128 / (s.nsc_max + 1), s.n / (sv.num_sms * 4)));
    const size_t gb = PB * (geom_bytes<R, KEYS>(s.rec_bytes) + 16);
    int blocks = 0;
    auto kg = k_share_geom<R, CT, KEYS>;
    if (fg_status rc = grid_for(kg, 128, gb, sv.num_sms, (s.n + PB - 1) / PB * 4, blocks)) return rc;
    kg<<<blocks, 128, gb, st>>>(T, s, coords, ipots, status, PB);
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

// The staged form's tables and energies of a part of the sub-batch
template <typename R, int EDGE>
fg_status launch_stage(const StageView &sv, const Tables<R> &T, const Share<R> &s, const StagePart<R> &part, int split,
                       C2<R> *out, cudaStream_t st)
{
    using K = Kinds<EDGE>;
    const int64_t tasks = part.n * s.nsc_max * ncanon(K::MM);
    auto kt = k_stage_tables<R, EDGE>;
    int tb = 0;
    if (fg_status rc = grid_for(kt, 128, 0, sv.num_sms, (tasks + 31) / 32, tb)) return rc;
    kt<<<tb, 128, 0, st>>>(T, s, part);
    FG_CUDA(cudaGetLastError());
    auto ke = s.nsc_max <= 2 ? k_stage_energies<R, EDGE, true> : k_stage_energies<R, EDGE, false>;
    const size_t wb = s.rec_bytes + align_up((size_t)s.nsc_max * part.tab_len * sizeof(R), 16);
    const int ew = fit_warps(4, wb, sv.max_smem);
    int eb = 0;
    if (fg_status rc = grid_for(ke, 32 * ew, wb * ew, sv.num_sms, part.n * split, eb)) return rc;
    ke<<<eb, 32 * ew, wb * ew, st>>>(T, s, part, split, out, wb);
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

template <typename R, int EDGE>
template <typename CT>
fg_status ShareLaunch<R, EDGE>::signals(const StageView &sv, const Tables<R> &T, const SharePlan &pl, Share<R> &s, const CT *coords,
                        const int64_t *ipots, int *status, C2<R> *out, cudaStream_t st)
{
    using K = Kinds<EDGE>;
    constexpr int KIND = K::MS;
    if (pl.staged) {
        if (fg_status rc = launch_geom<false>(sv, T, s, coords, ipots, status, st)) return rc;
        return launch_stage<R, EDGE>(sv, T, s, StagePart<R>{s.tab, s.tab_len, 0, s.n, nullptr}, pl.split, out, st);
    }
    const size_t wb = std::max(s.rec_bytes + align_up((size_t)(sv.L1 + 1) * dstride(K::MMSS) * sizeof(R), 16),
                               align_up((size_t)s.tab_len * sizeof(R), 16));
    auto kf = k_share_f<R, EDGE>;
    auto kc = k_share_chain<R, EDGE>;
    const int fw = fit_warps(4, wb, sv.max_smem);
    int fb = 0, cb = 0;
    if (fg_status rc = grid_for(kf, 32 * fw, wb * fw, sv.num_sms, s.n * s.nsc_max * pl.chunks, fb)) return rc;
    const int split = pl.split;
    const size_t wc = 4 * s.rec_bytes;
    if (fg_status rc = grid_for(kc, 128, wc, sv.num_sms, s.n * split, cb)) return rc;
    FG_CUDA(cudaMemsetAsync(s.head, 0, sizeof(ShareHead), st));
    FG_CUDA(cudaMemsetAsync(s.hash, 0xff, (size_t)pl.hcap * sizeof(unsigned), st));
    if (fg_status rc = launch_geom<false>(sv, T, s, coords, ipots, status, st)) return rc;
    if (fg_status rc = launch_share_insert(s, st)) return rc;
    const int64_t tasks = std::min<int64_t>(s.n * s.nsc_max, s.cls_cap) * ncanon(K::MMMS);
    k_share_tables<R, KIND><<<(int)std::min<int64_t>((tasks + 127) / 128, (int64_t)sv.num_sms * 16), 128, 0, st>>>(T, s);
    FG_CUDA(cudaGetLastError());
    for (int pass = 0; pass < pl.passes; ++pass) {
        kf<<<fb, 32 * fw, wb * fw, st>>>(T, s, pass, out, wb);
        kc<<<cb, 128, wc, st>>>(T, s, pass, split, out);
    }
    FG_CUDA(cudaGetLastError());
    if (pl.force) return FG_OK;
    // Nothing of this happens where the form was taken; where it was not, the records are there already, and the matrices'
    // memory holds the tables.  (Handing such a list to k_fused instead, which does its own geometry, cost what the search
    // had taken: 1,500 paths of 3-4 legs, 401 energies: 496 us without the search, 551 with it, 428 now; 5,000 paths 1,020,
    // 1,083 and 983; 20,000 paths on 60 energies 859, 1,005 and 778.)
    const int len = (sv.L1 + 1) * dstride(K::MM);
    static_assert(K::MM <= (EDGE == 1 ? 2 : 3), "the tables that share_plan makes room for");
    for (int64_t i0 = 0; i0 < s.n; i0 += pl.part) {
        const StagePart<R> part{reinterpret_cast<R *>(s.F), len, i0, std::min<int64_t>(pl.part, s.n - i0), &s.head->general};
        if (fg_status rc = launch_stage<R, EDGE>(sv, T, s, part, pl.part_split, out, st)) return rc;
    }
    return FG_OK;
}

template <typename R, int EDGE>
fg_status ShareLaunch<R, EDGE>::fine(const StageView &sv, const Share<R> &s, const PathsDev &pd, int NK, const double *q,
                                     const double *S, const int *span, unsigned char *pts, bool first, const C2<R> *sig,
                                     unsigned long long *racc, double *reff_save, int *status, cudaStream_t st)
{
    FinePoint *fp = reinterpret_cast<FinePoint *>(pts);
    if (first) k_fine_points<<<(NK + 127) / 128, 128, 0, st>>>(NK, sv.E, q, S, span, fp);
    // Four paths at a time where their amplitudes and phases are small (537,000 paths, 60 energies: 2.3 ms, two at a time
    // 2.6) and there are paths enough; the rows' sums in shared memory up to 1,024 points.
    const bool four = sv.E <= 128 && s.n >= (int64_t)sv.num_sms * 64, acc = NK <= 1024;
    auto kern = four ? (acc ? k_share_fine<R, 4, true> : k_share_fine<R, 4, false>)
                     : (acc ? k_share_fine<R, 1, true> : k_share_fine<R, 1, false>);
    const size_t wb = (size_t)2 * (four ? 4 : 1) * ((sv.E + 1) & ~1) * sizeof(double) + (acc ? (size_t)NK * 16 : 0);
    const int warps = fit_warps(8, wb, sv.max_smem / 2);
    int blocks = 0;
    if (fg_status rc = grid_for(kern, 32 * warps, wb * warps, sv.num_sms, s.n, blocks)) return rc;
    const int64_t range = (s.n + (int64_t)blocks * warps - 1) / ((int64_t)blocks * warps);
    kern<<<blocks, 32 * warps, wb * warps, st>>>(s, pd, sv.E, NK, S, fp, sig, racc, reff_save, status, range, wb);
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

template <typename R, int EDGE> fg_status ShareLaunch<R, EDGE>::reff(const Share<R> &s, R *out, cudaStream_t st)
{
    k_share_reff<R><<<(int)std::min<int64_t>((s.n + 255) / 256, 148 * 4), 256, 0, st>>>(s, out);
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

// ------------------------------------------------------------------------------------------------ shared matrices
// The adjoint with shared scattering matrices (fg_shared.cuh): a class keeps, per energy, F~ and its derivatives along
// beta and the lengths of its two legs, so that a path's sweep 2 contracts its orbit weights with them instead of
// running the partial waves again: 60 complex multiply-adds and 480 bytes per scatterer and energy (FP32) against
// about 25 x 60 multiply-adds.
//
//   k_share_geom        the keys (k_share_insert then finds the classes)
//   k_share_geom_adj    a warp per path, once the form is taken: the record with the frame and d/dbeta of the termination
//   k_share_tables_adj  a thread per (class, entry): D and D'
//   k_share_f_adj       two warps per (class, 32 energies): (F~, dF~/dbeta) and (dF~/drho_in, dF~/drho_out)
//   k_share_chain_adj   a warp per (path, energies): energy_ms_adj's sweeps with the matrices read
//   k_share_two_adj     a warp per (two-leg path, energies)
//   k_share_coord_grad  a warp per path: parameter gradients summed in a fixed order, carried to the coordinates
template <typename R> __device__ __forceinline__ AdjExtra<R> &adj_extra(unsigned char *rec)
{
    return *reinterpret_cast<AdjExtra<R> *>(rec + geo_bytes<R>());
}

// taken: the form is taken whatever the keys show, so this kernel writes them (a launch less); otherwise they are there and
// decide whether the records are needed
template <typename R, int KIND, typename CT>
__global__ void __launch_bounds__(128) k_share_geom_adj(Tables<R> T, Share<R> s, const CT *__restrict__ coords,
                                                        const int64_t *__restrict__ ipots, int *status, int MM_ss,
                                                        int MM_ms, int taken)
{
    if (s.refused() || (!taken && !share_chunks<R, KIND>(s))) return;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned char *base = smem + (size_t)w * s.rec_bytes;
    WarpPath<R> &g = *reinterpret_cast<WarpPath<R> *>(base);
    for (int64_t i = (int64_t)blockIdx.x * 4 + w; i < s.n; i += (int64_t)gridDim.x * 4) {
        const int64_t p = s.path(i);
        const int nleg = s.legs(p);
        path_setup<R, CT>(g, nullptr, T, coords + p * s.stride * 3, ipots + p * s.stride, nleg, lane, status,
                          nleg == 2 ? MM_ss : MM_ms, false);
        term_dbeta<R>(g, adj_extra<R>(base).dterm_db, T, nleg, lane);
        const int frame = choose_frame<R>(g, nleg, lane);
        if (frame) reframe_path<R>(g, nleg, lane, frame);
        if (lane == 0) adj_extra<R>(base).frame = frame;
        __syncwarp();
        copy16(s.rec + i * s.rec_bytes, base, s.rec_bytes, lane);
        if (taken) share_keys(s, g, i, nleg, lane);
        __syncwarp();
    }
}

template <typename R, int KIND> __global__ void __launch_bounds__(128) k_share_tables_adj(Tables<R> T, Share<R> s)
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
        R *t = s.tab + c * 2 * s.tab_len;
        rotation_column_adj<R>(t, t + s.tab_len, T, __longlong_as_double((long long)s.key[s.owner[c]].z), MM, DS,
                               (int)(i % NC));
    }
}

// F~ (accumulate_f's operations) and dF~/dbeta of one class and energy, from its two rotation tables
template <typename R, int KIND>
__device__ __forceinline__ void accumulate_f_beta(C2<R> (&acc)[RepTab<KIND, lamtab(KIND).N, lamtab(KIND).N>().n],
                                                  C2<R> (&accb)[RepTab<KIND, lamtab(KIND).N, lamtab(KIND).N>().n],
                                                  const R *dh, const R *dhd, const C2<R> *tlk, int E, int ilx,
                                                  C2<R> z_in, C2<R> z_out)
{
    constexpr LamTab L = lamtab(KIND);
    constexpr RepTab<KIND, L.N, L.N> RT{};
    constexpr int DS = dstride(L.MM), NCAN = ncanon(L.MM), CI = L.CI, CO = L.CO;
#pragma unroll
    for (int r = 0; r < RT.n; ++r) acc[r] = accb[r] = cz<R>();
    C2<R> pi[CI + 1], ci[CI + 1], po[CO + 1], co[CO + 1];
#pragma unroll
    for (int j = 0; j <= CI; ++j) pi[j] = ci[j] = cz<R>();
#pragma unroll
    for (int j = 0; j <= CO; ++j) po[j] = co[j] = cz<R>();
    pi[1] = ci[1] = po[1] = co[1] = C2<R>{R(1), R(0)};
    C2<R> t1 = tlk[E];
    for (int il = 1; il <= ilx; ++il) {
        const C2<R> t = t1;
        if (il < ilx) t1 = tlk[(size_t)(il + 1) * E];
        R d[NCAN], dd[NCAN];
        load_row<R, NCAN>(dh + (size_t)il * DS, d);
        load_row<R, NCAN>(dhd + (size_t)il * DS, dd);
        C2<R> tco[CO + 1];
#pragma unroll
        for (int j = 1; j <= CO; ++j) tco[j] = pmul(t, co[j]);
#pragma unroll
        for (int r = 0; r < RT.n; ++r) {
            const C2<R> u = pmul(ci[RT.ci[r]], tco[RT.co[r]]);
            acc[r] = pfmr(u, d[RT.d[r]], acc[r]);
            accb[r] = pfmr(u, dd[RT.d[r]], accb[r]);
        }
        const R w = R(2 * il - 1);
        const C2<R> wi = cscl(z_in, w), wo = cscl(z_out, w);
        C2<R> ni[CI + 1], no[CO + 1];
        ni[1] = cfms(wi, ci[1], pi[1]);
#pragma unroll
        for (int j = 2; j <= CI; ++j) ni[j] = cfms(wi, cadd(ci[j], ci[j - 1]), pi[j]);
        no[1] = cfms(wo, co[1], po[1]);
#pragma unroll
        for (int j = 2; j <= CO; ++j) no[j] = cfms(wo, cadd(co[j], co[j - 1]), po[j]);
#pragma unroll
        for (int j = 1; j <= CI; ++j) { pi[j] = ci[j]; ci[j] = ni[j]; }
#pragma unroll
        for (int j = 1; j <= CO; ++j) { po[j] = co[j]; co[j] = no[j]; }
    }
}

// dF~/drho_in and dF~/drho_out of one class and energy (the spherical waves' derivatives as in contract_f_adj)
template <typename R, int KIND>
__device__ __forceinline__ void accumulate_f_rho(C2<R> (&ai)[RepTab<KIND, lamtab(KIND).N, lamtab(KIND).N>().n],
                                                 C2<R> (&ao)[RepTab<KIND, lamtab(KIND).N, lamtab(KIND).N>().n],
                                                 const R *dh, const C2<R> *tlk, int E, int ilx, C2<R> z_in, C2<R> z_out)
{
    constexpr LamTab L = lamtab(KIND);
    constexpr RepTab<KIND, L.N, L.N> RT{};
    constexpr int DS = dstride(L.MM), NCAN = ncanon(L.MM), CI = L.CI, CO = L.CO;
#pragma unroll
    for (int r = 0; r < RT.n; ++r) ai[r] = ao[r] = cz<R>();
    C2<R> pi[CI + 2], ci[CI + 2], po[CO + 2], co[CO + 2];
#pragma unroll
    for (int j = 0; j <= CI + 1; ++j) pi[j] = ci[j] = cz<R>();
#pragma unroll
    for (int j = 0; j <= CO + 1; ++j) po[j] = co[j] = cz<R>();
    pi[1] = ci[1] = po[1] = co[1] = C2<R>{R(1), R(0)};
    C2<R> t1 = tlk[E];
    for (int il = 1; il <= ilx; ++il) {
        const C2<R> t = t1;
        if (il < ilx) t1 = tlk[(size_t)(il + 1) * E];
        R d[NCAN];
        load_row<R, NCAN>(dh + (size_t)il * DS, d);
        C2<R> tco[CO + 1], tdco[CO + 1], dci[CI + 1];
#pragma unroll
        for (int j = 1; j <= CO; ++j) {
            tco[j] = pmul(t, co[j]);
            tdco[j] = pmul(t, mi_z(z_out, pfmr(co[j], R(j - 1), cscl(co[j + 1], R(j)))));
        }
#pragma unroll
        for (int j = 1; j <= CI; ++j) dci[j] = mi_z(z_in, pfmr(ci[j], R(j - 1), cscl(ci[j + 1], R(j))));
#pragma unroll
        for (int r = 0; r < RT.n; ++r) {
            ai[r] = pfmr(pmul(dci[RT.ci[r]], tco[RT.co[r]]), d[RT.d[r]], ai[r]);
            ao[r] = pfmr(pmul(ci[RT.ci[r]], tdco[RT.co[r]]), d[RT.d[r]], ao[r]);
        }
        const R w = R(2 * il - 1);
        const C2<R> wi = cscl(z_in, w), wo = cscl(z_out, w);
        C2<R> ni[CI + 2], no[CO + 2];
#pragma unroll
        for (int j = 1; j <= CI + 1; ++j) ni[j] = pfms(wi, j > 1 ? padd(ci[j], ci[j - 1]) : ci[j], pi[j]);
#pragma unroll
        for (int j = 1; j <= CO + 1; ++j) no[j] = pfms(wo, j > 1 ? padd(co[j], co[j - 1]) : co[j], po[j]);
#pragma unroll
        for (int j = 1; j <= CI + 1; ++j) { pi[j] = ci[j]; ci[j] = ni[j]; }
#pragma unroll
        for (int j = 1; j <= CO + 1; ++j) { po[j] = co[j]; co[j] = no[j]; }
    }
}

// Items (class, chunk of the pass, half): the class's four matrices over the chunk lie one after the other (F~, beta,
// rho_in, rho_out).  Entries outside a lower lambda order's set are stored as zeros, derivatives too, so a path's
// weights need no masking.
template <typename R, int EDGE>
__global__ void __launch_bounds__(128) k_share_f_adj(Tables<R> T, Share<R> s, int pass, size_t wbytes)
{
    using K = Kinds<EDGE>;
    constexpr int KIND = K::MS;
    constexpr LamTab L = lamtab(KIND);
    constexpr RepTab<KIND, L.N, L.N> RT{};
    const int G = s.refused() ? 0 : share_chunks<R, KIND>(s), g0 = pass * G;
    const int ng = min(G, s.chunks - g0), E = T.E;          // <= 0: nothing to do
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    R *dh = reinterpret_cast<R *>(smem + (size_t)w * wbytes);
    const int64_t items = ng > 0 ? (int64_t)s.head->classes * ng * 2 : 0;
    for (int64_t it = (int64_t)blockIdx.x * nw + w; it < items; it += (int64_t)gridDim.x * nw) {
        const int half = (int)(it & 1), gc = (int)((it >> 1) % ng);
        const int64_t c = (it >> 1) / ng;
        const int e = first_chunk(E) + 32 * (g0 + gc) + lane;
        copy16(dh, s.tab + c * 2 * s.tab_len, (size_t)s.tab_len * sizeof(R) * (half ? 1 : 2), lane);
        const ShareKey key = s.key[s.owner[c]];
        __syncwarp();
        if (e >= 0 && e < E) {
            const C2<R> ck = T.ck[e];
            if (fabs((double)ck.x) + fabs((double)ck.y) > 1e-16) {
                const int ip = (int)key.w;
                const C2<R> *tl = T.tl + (size_t)ip * (T.L1 + 1) * E + e;
                const int ilx = T.lmax[ip * E + e] + 1;
                const C2<R> z_in = zfac(cscl(ck, (R)__longlong_as_double((long long)key.y)));
                const C2<R> z_out = zfac(cscl(ck, (R)__longlong_as_double((long long)key.x)));
                C2<R> a[RT.n], b[RT.n];
                if (half) accumulate_f_rho<R, KIND>(a, b, dh, tl, E, ilx, z_in, z_out);
                else accumulate_f_beta<R, KIND>(a, b, dh, dh + s.tab_len, tl, E, ilx, z_in, z_out);
                mask_lambda<R, KIND, L.N, L.N>(a, T.nlam);
                mask_lambda<R, KIND, L.N, L.N>(b, T.nlam);
                unsigned char *at = s.F + ((c * G + gc) * 4 + 2 * half) * f_chunk_bytes<R, KIND>();
                C2<R> f[20];
                to_blocks<R, KIND, L.N, L.N>(a, f);
                store_f<R, 20>(at, lane, f);
                to_blocks<R, KIND, L.N, L.N>(b, f);
                store_f<R, 20>(at + f_chunk_bytes<R, KIND>(), lane, f);
            }
        }
        __syncwarp();
    }
    // the kernel that this one may run beside (k_share_two_adj) has ended before this one does
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

// g + sum of w[r] f[r] over a stored matrix's canonical entries
template <typename R, int NE>
__device__ __forceinline__ C2<R> dot_f(const unsigned char *at, int lane, const C2<R> (&w)[NE])
{
    C2<R> f[NE], g0 = cz<R>(), g1 = cz<R>();
    load_f<R, NE>(at, lane, f);
#pragma unroll
    for (int r = 0; r < NE; r += 2) {
        g0 = pfma(w[r], f[r], g0);
        g1 = pfma(w[r + 1], f[r + 1], g1);
    }
    return cadd(g0, g1);
}

// One energy of a path of three and more legs: energy_ms_adj with its matrices and their derivatives read (cls: the
// path's classes, at(c): where class c's four matrices of this chunk lie).
template <typename R, int KIND, class AT>
__device__ __forceinline__ void shared_energy_adj(const WarpPath<R> &g, const R (*dterm_db)[49], const Tables<R> &T, int e,
                                                  int nleg, int lane, C2<R> gbar, const AT &at, ParGrad &pg)
{
    constexpr LamTab L = lamtab(KIND);
    constexpr int N0 = L.N0;
    using B = Flip<KIND>;
    constexpr size_t FB = f_chunk_bytes<R, KIND>();
    const int nsc = nleg - 1;
    const C2<R> ck = T.ck[e];
    if (fabs((double)ck.x) + fabs((double)ck.y) <= 1e-16) return;
    auto add_re = [](double &acc, C2<R> s, C2<R> v) { acc += (double)s.x * v.x - (double)s.y * v.y; };
    const C2<R> cf = cfac(g, T, e, nleg, ck);
    const C2<R> sd = cmul(C2<R>{gbar.x, -gbar.y}, cf);      // s = conj(gbar) cfac: dL = Re(s dptrac)
    const C2<R> sck = cmul(sd, ck);
    // everything in the flip basis: P_k by columns (k = 0: the N0 unit columns), R_k by rows
    C2<R> Pst[kMaxLeg][N0][6];
    C2<R> Rst[N0][6];
#pragma unroll
    for (int c = 0; c < N0; ++c)
#pragma unroll
        for (int i = 0; i < 6; ++i)
            Pst[0][c][i] = (c < B::NE0 ? i == c : i == 4 + c - B::NE0) ? C2<R>{R(1), R(0)} : cz<R>();
    for (int k = 1; k <= nsc; ++k) {
        C2<R> f[20];
        load_f<R, 20>(at(k), lane, f);
        const C2<R> e1 = g.phs[k + 1], e2 = cmul(e1, e1);
#pragma unroll 1
        for (int c = 0; c < N0; ++c) {
            C2<R> x[6];
#pragma unroll
            for (int i = 0; i < 6; ++i) x[i] = Pst[k - 1][c][i];
            block_step<R, KIND>(f, e1, e2, true, x);
#pragma unroll
            for (int i = 0; i < 6; ++i) Pst[k][c][i] = x[i];
        }
    }
    {
        TermLegs<R, KIND> tl;
        term_legs<R, KIND>(g, T, e, nleg, ck, tl);
        C2<R> ge1 = cz<R>(), gbn = cz<R>(), gr1 = cz<R>(), grn = cz<R>();
        C2<R> Q[N0][N0], Tm[N0][N0];
        from_blocks<R, KIND>([&](int c, int i) { return Pst[nsc][c][i]; }, Q);
        const C2<R> ptrac = term_adj<R, KIND>(g, dterm_db, T, e, tl, [&](int b, int a) { return Q[b][a]; }, ge1, gbn, gr1,
                                              grn, &Tm[0][0], N0);
        add_re(pg.eta[1], sd, ge1);
        add_re(pg.beta[nleg], sd, gbn);
        add_re(pg.ri[1], sck, gr1);
        add_re(pg.ri[nleg], sck, grn);
        cfac_grad(g, T, e, nleg, gbar, cmul(ptrac, cf), pg);
        // R_nsc = [T 0] in the flip basis: rows u, w of T, then its columns halved back
        auto mix = [](C2<R> p, C2<R> m, int am, bool w) {      // p +- (-1)^am m
            return ((am & 1) != 0) != w ? csub(p, m) : cadd(p, m);
        };
#pragma unroll
        for (int c = 0; c < N0; ++c) {
            const bool cw = c >= B::NE0;
            const int cm = cw ? c - B::NE0 + 1 : B::em(c), cn = cw ? 0 : B::en(c);
            C2<R> row[N0];
#pragma unroll
            for (int b = 0; b < N0; ++b)
                row[b] = cm == 0 ? Tm[B::at(0, cn)][b] : mix(Tm[B::at(cm, 0)][b], Tm[B::at(-cm, 0)][b], cm, cw);
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                const bool iw = i >= 4;
                const int im = iw ? i - 3 : B::em(i), in = iw ? 0 : B::en(i);
                C2<R> v = cz<R>();
                if (iw ? i - 4 < B::NO0 : i < B::NE0)
                    v = im == 0 ? row[B::at(0, in)] : cscl(mix(row[B::at(im, 0)], row[B::at(-im, 0)], im, iw), R(0.5));
                Rst[c][i] = v;
            }
        }
    }
    for (int k = nsc; k >= 1; --k) {
        const C2<R> e1 = g.phs[k + 1], e2 = cmul(e1, e1);
        // weights of F~_k's block entries, (P_(k-1) R_k Phi)[j][i], and the Euler angle's derivative
        // -i sum_m m (P_k R_k)(m, m), which in this basis pairs u_m with w_m
        C2<R> Wh[20], tm = cz<R>();
#pragma unroll
        for (int r = 0; r < 20; ++r) Wh[r] = cz<R>();
#pragma unroll 1
        for (int c = 0; c < N0; ++c) {
            C2<R> p[6], rr[6];
#pragma unroll
            for (int i = 0; i < 6; ++i) { p[i] = Pst[k - 1][c][i]; rr[i] = Rst[c][i]; }
            tm = pfma(rr[2], Pst[k][c][4], pfma(rr[4], Pst[k][c][2], tm));
            tm = pfma(cscl(rr[3], R(2)), Pst[k][c][5], pfma(cscl(rr[5], R(2)), Pst[k][c][3], tm));
            turn(e1, rr[2], rr[4]);
            turn(e2, rr[3], rr[5]);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) Wh[4 * i + j] = pfma(p[j], rr[i], Wh[4 * i + j]);
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) Wh[16 + 2 * i + j] = pfma(p[4 + j], rr[4 + i], Wh[16 + 2 * i + j]);
        }
        add_re(pg.eta[k + 1], sd, C2<R>{tm.y, -tm.x});   // -i tm
        const unsigned char *m = at(k);
        add_re(pg.beta[k], sd, dot_f<R, 20>(m + FB, lane, Wh));
        add_re(pg.ri[k + 1], sck, dot_f<R, 20>(m + 2 * FB, lane, Wh));
        add_re(pg.ri[k], sck, dot_f<R, 20>(m + 3 * FB, lane, Wh));
        if (k > 1) {
            // R_(k-1) = R_k Phi F~_k, one row at a time
            C2<R> f[20];
            load_f<R, 20>(m, lane, f);
#pragma unroll 1
            for (int c = 0; c < N0; ++c) {
                C2<R> rr[6];
#pragma unroll
                for (int i = 0; i < 6; ++i) rr[i] = Rst[c][i];
                turn(e1, rr[2], rr[4]);
                turn(e2, rr[3], rr[5]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    C2<R> v = cz<R>();
#pragma unroll
                    for (int i = 0; i < 4; ++i) v = pfma(rr[i], f[4 * i + j], v);
                    Rst[c][j] = v;
                }
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    Rst[c][4 + j] = pfma(rr[5], f[18 + j], pfma(rr[4], f[16 + j], cz<R>()));
            }
        }
    }
}

// The parameter gradients of one item summed over the warp's energies into the path's entry of its part (gpar), added
// to what earlier passes left there.
__device__ __forceinline__ void store_par(double *o, const ParGrad &pg, int nleg, int lane, bool first)
{
    for (int j = 1; j <= nleg; ++j) {
        double v[3] = {pg.ri[j], pg.beta[j], pg.eta[j]};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
#pragma unroll
            for (int h = 16; h > 0; h >>= 1) v[c] += __shfl_xor_sync(0xffffffffu, v[c], h);
        }
        if (lane < 3) {
            const double x = lane == 0 ? v[0] : (lane == 1 ? v[1] : v[2]);
            double &at = o[lane * (kMaxLeg + 1) + j];
            at = first ? x : at + x;
        }
    }
}

template <typename R, int EDGE>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 3 : 2) k_share_chain_adj(Tables<R> T, Share<R> s, int pass, int split,
                                                         const C2<R> *__restrict__ gbar, double *__restrict__ gpar)
{
    using K = Kinds<EDGE>;
    constexpr int KIND = K::MS;
    if (s.refused()) return;
    const int G = share_chunks<R, KIND>(s), g0 = pass * G;
    if (!G || g0 >= s.chunks) return;
    const int ng = min(G, s.chunks - g0), E = T.E;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int cls_sh[4][kMaxLeg];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned char *base = smem + (size_t)w * s.rec_bytes;
    const WarpPath<R> &g = *reinterpret_cast<const WarpPath<R> *>(base);
    // all paths of one part of the energies, then the next: the classes of neighbouring paths over few energies stay in L2
    for (int64_t it = (int64_t)blockIdx.x * 4 + w; it < s.n * split; it += (int64_t)gridDim.x * 4) {
        const int part = (int)(it / s.n);
        const int64_t i = it % s.n, p = s.path(i);
        const int nleg = s.legs(p);
        if (nleg == 2) continue;
        copy16(base, s.rec + i * s.rec_bytes, s.rec_bytes, lane);
        if (lane < nleg - 1) cls_sh[w][lane] = s.cls[s.slot_of[i * s.nsc_max + lane]];
        __syncwarp();
        ParGrad pg;
        for (int j = 0; j <= kMaxLeg; ++j) pg.ri[j] = pg.beta[j] = pg.eta[j] = 0.0;
        for (int gc = part; gc < ng; gc += split) {
            const int e = first_chunk(E) + 32 * (g0 + gc) + lane;
            if (e >= 0 && e < E)
                shared_energy_adj<R, KIND>(
                    g, adj_extra<R>(base).dterm_db, T, e, nleg, lane, gbar[p * E + e],
                    [&](int k) { return s.F + ((int64_t)cls_sh[w][k - 1] * G + gc) * 4 * f_chunk_bytes<R, KIND>(); },
                    pg);
            __syncwarp();
        }
        store_par(gpar + (part * s.n + i) * kGparStride, pg, nleg, lane, pass == 0);
        __syncwarp();
    }
}

// Two-leg paths, all their energies in one launch
template <typename R, int EDGE>
__global__ void __launch_bounds__(128) k_share_two_adj(Tables<R> T, Share<R> s, int split,
                                                       const C2<R> *__restrict__ gbar, double *__restrict__ gpar,
                                                       size_t wbytes)
{
    using K = Kinds<EDGE>;
    if (s.refused() || !share_chunks<R, K::MS>(s)) return;
    extern __shared__ __align__(16) unsigned char smem[];
    // k_share_f_adj, which needs nothing of this kernel, may start beside it (its launch allows it)
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5, E = T.E;
    unsigned char *base = smem + (size_t)w * wbytes;
    const WarpPath<R> &g = *reinterpret_cast<const WarpPath<R> *>(base);
    R *dh = reinterpret_cast<R *>(base + s.rec_bytes), *dhd = dh + (size_t)(T.L1 + 1) * dstride(K::MMSS);
    for (int64_t it = (int64_t)blockIdx.x * nw + w; it < (int64_t)s.head->two * split; it += (int64_t)gridDim.x * nw) {
        const int64_t i = s.two[it / split], p = s.path(i);
        copy16(base, s.rec + i * s.rec_bytes, s.rec_bytes, lane);
        __syncwarp();
        for (int r = lane; r < ncanon(K::MMSS); r += 32)
            rotation_column_adj<R>(dh, dhd, T, g.beta[1], K::MMSS, dstride(K::MMSS), r);
        __syncwarp();
        ParGrad pg;
        for (int j = 0; j <= kMaxLeg; ++j) pg.ri[j] = pg.beta[j] = pg.eta[j] = 0.0;
        for (int gc = (int)(it % split); gc < s.chunks; gc += split) {
            const int e = first_chunk(E) + 32 * gc + lane;
            if (e >= 0 && e < E)
                path_energy_adj<R, EDGE>(g, dh, dhd, adj_extra<R>(base).dterm_db, T, e, 2, gbar[p * E + e], pg);
            __syncwarp();
        }
        store_par(gpar + ((it % split) * s.n + i) * kGparStride, pg, 2, lane, true);
        __syncwarp();
    }
}

// The paths' parameter gradients (their parts summed in order) carried to the coordinates, as k_adjoint and
// k_coord_grad do it; the atoms come from the record, already in the path's frame.
template <typename R, int KIND>
__global__ void __launch_bounds__(128) k_share_coord_grad(Share<R> s, int split, const double *__restrict__ gpar,
                                                          const double *__restrict__ greff_d,
                                                          const R *__restrict__ greff_r, double *__restrict__ gout_d,
                                                          R *__restrict__ gout_r)
{
    __shared__ double s_gpar[4][3 * (kMaxLeg + 1)], s_cg[4][9 * kMaxLeg];
    if (s.refused() || !share_chunks<R, KIND>(s)) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int64_t i = (int64_t)blockIdx.x * 4 + w; i < s.n; i += (int64_t)gridDim.x * 4) {
        const int64_t p = s.path(i);
        const int nleg = s.legs(p);
        const unsigned char *rec = s.rec + i * s.rec_bytes;
        const WarpPath<R> &g = *reinterpret_cast<const WarpPath<R> *>(rec);
        const int frame = reinterpret_cast<const AdjExtra<R> *>(rec + geo_bytes<R>())->frame;
        const double gr = greff_d ? greff_d[p] : (greff_r ? (double)greff_r[p] : 0.0);
        for (int t = lane; t < 3 * (kMaxLeg + 1); t += 32) {
            const int j = t % (kMaxLeg + 1);
            double v = 0.0;
            if (j >= 1 && j <= nleg) {
                for (int q = 0; q < split; ++q) v += gpar[((int64_t)q * s.n + i) * kGparStride + t];
                if (t < kMaxLeg + 1) v += gr * kBohr * 0.5;          // reff (A) = BOHR sum ri (bohr) / 2
            }
            s_gpar[w][t] = v;
        }
        __syncwarp();
        double gc = coord_grad(g.xyz, s_gpar[w], s_cg[w], nleg, lane);
        if (frame) gc = unframe_grad(gc, lane, frame);
        if (lane < 3 * s.stride) {
            const int64_t o = p * s.stride * 3 + lane;
            const double v = lane < 3 * nleg ? gc : 0.0;
            if (gout_d) gout_d[o] = v;
            else gout_r[o] = (R)v;
        }
        __syncwarp();
    }
}

// One sub-batch's coordinate gradients in the shared form; head->general is set and nothing written where it is not
// taken.  coords, ipots, gbar, greff and the outputs are indexed by path.
template <typename R, int EDGE>
template <typename CT>
fg_status ShareLaunch<R, EDGE>::adjoint(const StageView &sv, const Tables<R> &T, const SharePlan &pl, Share<R> &s, unsigned char *ws,
                        const CT *coords, const int64_t *ipots, int *status, const C2<R> *gbar, const double *greff_d,
                        const R *greff_r, double *gout_d, R *gout_r, cudaStream_t st)
{
    using K = Kinds<EDGE>;
    constexpr int KIND = K::MS;
    double *gpar = reinterpret_cast<double *>(ws + pl.gpar);
    s.rec_bytes = geo_bytes<R>() + align_up(sizeof(AdjExtra<R>), 16);
    // the launches' shapes before the first of them: the short kernels ahead of the matrices leave the host no time
    auto kf = k_share_f_adj<R, EDGE>;
    auto kc = k_share_chain_adj<R, EDGE>;
    auto k2 = k_share_two_adj<R, EDGE>;
    const size_t wf = align_up(2 * (size_t)s.tab_len * sizeof(R), 16);
    const size_t w2 = s.rec_bytes + align_up(2 * (size_t)(sv.L1 + 1) * dstride(K::MMSS) * sizeof(R), 16);
    const int nf = fit_warps(4, wf, sv.max_smem), n2 = fit_warps(4, w2, sv.max_smem), split = pl.split;
    int bf = 0, bc = 0, b2 = 0;
    if (fg_status rc = grid_for(kf, 32 * nf, wf * nf, sv.num_sms, s.n * s.nsc_max * pl.chunks * 2, bf)) return rc;
    const size_t wc = 4 * s.rec_bytes;
    if (fg_status rc = grid_for(kc, 128, wc, sv.num_sms, s.n * split, bc)) return rc;
    if (fg_status rc = grid_for(k2, 32 * n2, w2 * n2, sv.num_sms, s.n * split, b2)) return rc;
    FG_CUDA(cudaMemsetAsync(s.head, 0, sizeof(ShareHead), st));
    FG_CUDA(cudaMemsetAsync(s.hash, 0xff, (size_t)pl.hcap * sizeof(unsigned), st));
    const int pb = (int)std::min<int64_t>((s.n + 3) / 4, (int64_t)sv.num_sms * 16);
    auto records = [&]() -> fg_status {
        k_share_geom_adj<R, KIND, CT><<<pb, 128, 4 * s.rec_bytes, st>>>(T, s, coords, ipots, status, K::MMSS, K::MMMS, pl.force);
        FG_CUDA(cudaGetLastError());
        return FG_OK;
    };
    if (fg_status rc = pl.force ? records() : launch_geom<true>(sv, T, s, coords, ipots, status, st)) return rc;
    if (fg_status rc = launch_share_insert(s, st)) return rc;
    if (!pl.force)
        if (fg_status rc = records()) return rc;
    const int64_t tasks = std::min<int64_t>(s.n * s.nsc_max, s.cls_cap) * ncanon(K::MMMS);
    k_share_tables_adj<R, KIND><<<(int)std::min<int64_t>((tasks + 127) / 128, (int64_t)sv.num_sms * 16), 128, 0, st>>>(T, s);
    FG_CUDA(cudaGetLastError());
    k2<<<b2, 32 * n2, w2 * n2, st>>>(T, s, split, gbar, gpar, w2);
    for (int pass = 0; pass < pl.passes; ++pass) {
        if (pass == 0) {                                     // beside the two-leg paths' kernel, not after it
            cudaLaunchAttribute beside{};
            beside.id = cudaLaunchAttributeProgrammaticStreamSerialization;
            beside.val.programmaticStreamSerializationAllowed = 1;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = bf; cfg.blockDim = 32 * nf; cfg.dynamicSmemBytes = wf * nf; cfg.stream = st;
            cfg.attrs = &beside; cfg.numAttrs = 1;
            FG_CUDA(cudaLaunchKernelEx(&cfg, kf, T, s, pass, wf));
        } else {
            kf<<<bf, 32 * nf, wf * nf, st>>>(T, s, pass, wf);
        }
        kc<<<bc, 128, wc, st>>>(T, s, pass, split, gbar, gpar);
    }
    k_share_coord_grad<R, KIND><<<pb, 128, 0, st>>>(s, split, gpar, greff_d, greff_r, gout_d, gout_r);
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

}  // namespace fg

#define FG_SHARE_INSTANCE(R, EDGE)                                                                                     \
    template struct fg::ShareLaunch<R, EDGE>;                                                                         \
    template fg_status fg::ShareLaunch<R, EDGE>::signals<float>(                                                      \
        const StageView &, const Tables<R> &, const SharePlan &, Share<R> &, const float *, const int64_t *, int *,   \
        C2<R> *, cudaStream_t);                                                                                       \
    template fg_status fg::ShareLaunch<R, EDGE>::signals<double>(                                                     \
        const StageView &, const Tables<R> &, const SharePlan &, Share<R> &, const double *, const int64_t *, int *,  \
        C2<R> *, cudaStream_t);                                                                                       \
    template fg_status fg::ShareLaunch<R, EDGE>::adjoint<float>(                                                      \
        const StageView &, const Tables<R> &, const SharePlan &, Share<R> &, unsigned char *, const float *,          \
        const int64_t *, int *, const C2<R> *, const double *, const R *, double *, R *, cudaStream_t);               \
    template fg_status fg::ShareLaunch<R, EDGE>::adjoint<double>(                                                     \
        const StageView &, const Tables<R> &, const SharePlan &, Share<R> &, unsigned char *, const double *,         \
        const int64_t *, int *, const C2<R> *, const double *, const R *, double *, R *, cudaStream_t);
