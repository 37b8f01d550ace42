// fg_shared.cu -- classes of equal scatterers (fg_shared.cuh) and the sizes of their workspace.
#include <algorithm>

#include "fg_forward.cuh"
#include "fg_launch.h"

namespace fg {
namespace {
__device__ __forceinline__ unsigned key_hash(const ShareKey &k)
{
    // each word's bits spread by an odd multiplier (2^64 / the golden ratio; the second and third primes of xxHash64, Collet,
    // BSD), folded by the finaliser of MurmurHash3 (Appleby, public domain)
    unsigned long long h = k.x * 0x9e3779b97f4a7c15ull ^ (k.y * 0xc2b2ae3d27d4eb4full + k.w) ^ (k.z * 0x165667b19e3779f9ull);
    h ^= h >> 33; h *= 0xff51afd7ed558ccdull;
    h ^= h >> 33; h *= 0xc4ceb9fe1a85ec53ull;
    return (unsigned)(h ^ (h >> 33));
}

// A thread per scatterer: linear probing; a slot belongs to the first scatterer that claimed it, and every scatterer
// whose key equals the owner's bit for bit is of its class.  The table has at least twice as many slots as scatterers.
__global__ void __launch_bounds__(256) k_share_insert(ShareIdx s)
{
    if (s.refused()) return;
    const int64_t total = s.n * s.nsc_max;
    unsigned mine = 0;                                   // scatterers of this thread, at most 2^21 in all
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t / s.nsc_max;
        const int nleg = s.legs(s.order ? s.order[i] : i);
        if (nleg <= 2 || (int)(t % s.nsc_max) >= nleg - 1) continue;
        ++mine;
        const ShareKey k = s.key[t];
        unsigned h = key_hash(k) & s.hmask;
        for (unsigned probe = 0; probe <= s.hmask; ++probe, h = (h + 1) & s.hmask) {
            const unsigned was = atomicCAS(s.hash + h, 0xffffffffu, (unsigned)t);
            if (was == 0xffffffffu) {
                const int c = atomicAdd(&s.head->classes, 1);
                s.cls[h] = c;
                if (c < s.cls_cap) s.owner[c] = (unsigned)t;
                break;
            }
            const ShareKey o = s.key[was];
            if (o.x == k.x && o.y == k.y && o.z == k.z && o.w == k.w) break;
        }
        s.slot_of[t] = (int)h;
    }
    mine = __reduce_add_sync(0xffffffffu, mine);         // after the loop, where the whole warp is together again
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd((unsigned long long *)&s.head->scatterers, (unsigned long long)mine);
}
}  // namespace

fg_status launch_share_insert(const ShareIdx &s, cudaStream_t st)
{
    const int64_t total = s.n * s.nsc_max;
    k_share_insert<<<(int)std::min<int64_t>((total + 255) / 256, 148 * 8), 256, 0, st>>>(s);
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

SharePlan share_plan(int64_t n, int nleg_max, int E, int L1, bool fp64, int iorder, int ilinit, bool adjoint, int NK)
{
    SharePlan p;
    if (iorder > 2 || n < 1) return p;
    // Lists of up to three legs share nothing (every scatterer has the absorber on one side and the path's only other
    // atom on the other), so they take this form only where few paths leave the chip idle and it spreads their energies
    // over warps: many energies, or the fifteen-column single scattering of L and M edges (897 paths, L3, 59 energies:
    // 342 -> 245 us; at the K edge on 60 energies the extra launches cost what the spreading gains: 396 paths forward
    // 421 -> 474 us, backward of 396 and 4,438 paths 445 -> 472 and 1355 -> 1420 us).  Longer paths take it wherever
    // the call is worth the launches that find the classes (about 40 us): at two chunks of energies and 4,438 paths of
    // up to four legs, 1.27 scatterers per class, looking for them cost 5 %.  Where they are not found, the call goes on in
    // the staged form (3-4 legs, nothing shared, 401 energies, against the one-kernel form without a search: 700 paths 320
    // -> 309 us, 1,000 paths, which fill one wave of it, 332 -> 352, 5,000 paths 1,020 -> 983).
    const int chunks = (E + 31) / 32;
    const bool small = n * chunks <= kShareSmall && (chunks >= 4 || ilinit > 1);
    // What is left and large enough takes the staged form (4,438 paths on 60 energies 1.35 -> 1.08 ms a refinement step,
    // its rows' sums in shared memory then another 0.05; at 396 paths its launches cost what it gains).
    const bool classes = small || (nleg_max >= 4 && (chunks >= 4 || n * chunks > kShareWorth));
    p.staged = !adjoint && !classes && n * chunks > kStageWorth;
    if (!classes && !p.staged) return p;
    const size_t real = fp64 ? 8 : 4;
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t o = at; at += align_up(bytes, 256); return o; };
    const size_t rec = align_up(fp64 ? sizeof(WarpPath<double>) : sizeof(WarpPath<float>), 16);
    p.nsc_max = nleg_max - 1;
    p.chunks = chunks;
    p.pts = take((size_t)NK * 32);
    if (p.staged) {
        p.sub = std::min<int64_t>(n, kStageSub);
        p.force = p.passes = 1;
        p.split = (int)std::min<int64_t>(chunks, (kShareItems / 4 + p.sub - 1) / p.sub);
        p.rec = take((size_t)p.sub * rec);
        p.tab = take((size_t)p.sub * p.nsc_max * (L1 + 1) * dstride(3) * real);
        p.sig = take((size_t)p.sub * E * 2 * real);
        p.total = at;
        return p;
    }
    p.sub = std::min<int64_t>(n, kShareSub);
    const int64_t scat = p.sub * p.nsc_max;
    p.mats = adjoint ? 4 : 1;
    const size_t per = p.mats * 20 * 2 * real * 32;          // one class, one chunk: 20 canonical entries (orders 0-2)
    const size_t all = (size_t)scat * p.chunks * per;
    p.f_bytes = std::min(all, adjoint ? 2 * kShareMatrixBytes : kShareMatrixBytes);
    if (!adjoint) {
        // one path's tables in the staged form (as few parts as can be: where the form is taken, each is two idle launches)
        const size_t tables = (size_t)p.nsc_max * (L1 + 1) * dstride(ilinit == 1 ? 2 : 3) * real;
        p.f_bytes = std::max(p.f_bytes, tables);
        p.part = std::min<int64_t>(p.sub, (int64_t)(p.f_bytes / tables));
        p.part_split = (int)std::min<int64_t>(chunks, (kShareItems / 4 + p.part - 1) / p.part);
    }
    p.cls_cap = std::min<int64_t>(scat, (int64_t)(p.f_bytes / per));
    const int fit = (int)std::min<size_t>(p.chunks, p.f_bytes / ((size_t)scat * per));   // chunks per pass at worst
    p.passes = fit ? (p.chunks + fit - 1) / fit : p.chunks;
    p.force = small && fit == p.chunks;
    // a path's energies are spread over warps until the items fill the chip many times over (10,007 paths x 13 chunks,
    // backward: k_share_chain_adj 4.0 ms unsplit, the last of its six waves nearly empty)
    p.split = (int)std::min<int64_t>(chunks, (kShareItems + p.sub - 1) / p.sub);
    p.hcap = 64;
    while ((int64_t)p.hcap < 2 * scat) p.hcap *= 2;
    const size_t ext = align_up(fp64 ? sizeof(AdjExtra<double>) : sizeof(AdjExtra<float>), 16);
    p.rec = take((size_t)p.sub * (adjoint ? rec + ext : rec));
    p.key = take((size_t)scat * sizeof(ShareKey));
    p.slot = take((size_t)scat * 4);
    p.hash = take((size_t)p.hcap * 4);
    p.cls = take((size_t)p.hcap * 4);
    p.owner = take((size_t)p.cls_cap * 4);
    p.two = take((size_t)p.sub * 4);
    p.tab = take((size_t)p.cls_cap * (L1 + 1) * dstride(2) * real * (adjoint ? 2 : 1));
    p.F = take(p.f_bytes);
    if (adjoint) p.gpar = take((size_t)p.split * p.sub * kGparStride * sizeof(double));
    else p.sig = take((size_t)p.sub * E * 2 * real);
    p.total = at;
    return p;
}

}  // namespace fg
