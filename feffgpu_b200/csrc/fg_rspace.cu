// fg_rspace.cu -- the R-space misfit of chi(k) rows and its gradient in one kernel (the loss of the reference's
// refinement, src/feffgpu/exafs/transform.py:104-145: windowed, k-weighted, zero-padded FFT restricted to the R window,
// then sum |chi_R - target_R|^2 / sum |target_R|^2).
//
// The transform restricted to the kept R points is a dense complex matrix F (NR, NK) built once by the host.  A cluster
// of eight blocks takes a row: block b forms chi_R - target at the R points m = b, b + 8, ... (a warp per R point,
// coalesced over k) and leaves it in every block's shared memory; after the cluster's barrier the misfit's partial sums
// are added in order and block b forms the gradient dR/dx_k = 2/norm Re sum_m conj(d_m) F[m][k] over its eighth of the k
// (a thread per k and quarter of the m) -- so a refinement step needs no further launch for the loss's backward.  FP64,
// fixed-order sums.  A refinement evaluates one or two rows, and one block per row reads the 163 x 401 transform twice
// through one SM's L2 path: 43.6 us for a row on B200, against 9.1 us with eight blocks (the transform is 1 MB; what is
// left are two cluster barriers and the latency of the two passes).
//
// More rows than one wave of clusters (148, at eight blocks an SM) take one block each: it goes through the eight blocks'
// shares one after the other, with the same sums in the same order, and has no cluster to wait for (148 rows: 48 us a
// block each, 34 a cluster each; 500 rows: 80 and 110; 4,096 rows: 528 and 779).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "fg_launch.h"

namespace fg {
namespace {

namespace cg = cooperative_groups;
constexpr int kThreads = 256, kWarps = kThreads / 32, kShares = 8;
constexpr int64_t kClusterRows = 148;

// NB blocks per row (a cluster of them): 8 or 1
template <int NB>
__device__ __forceinline__ void rspace_row(int NK, int NR, const double *__restrict__ rows, const double2 *__restrict__ F,
                                           const double2 *__restrict__ target, double inv_norm, double *__restrict__ R,
                                           double *__restrict__ grad)
{
    static_assert(NB == 1 || NB == kShares, "a block per share, or one for all");
    extern __shared__ __align__(16) unsigned char smem[];
    double *x = reinterpret_cast<double *>(smem);                 // (NK) the row
    double2 *d = reinterpret_cast<double2 *>(x + ((NK + 1) & ~1));  // (NR) chi_R - target
    __shared__ double wsum[kShares][kWarps], part[kShares], red[kThreads];   // part: the shares' sums (block 0's copy is read)
    cg::cluster_group cl = cg::this_cluster();
    const int rank = NB == 1 ? 0 : (int)cl.block_rank();
    const int64_t b = blockIdx.x / NB;
    auto sync = [&] { if constexpr (NB == 1) __syncthreads(); else cl.sync(); };
    for (int k = threadIdx.x; k < NK; k += blockDim.x) x[k] = rows[b * NK + k];
    sync();                                                       // every block's shared memory is there to be written
    // chi_R - target: lanes over k (coalesced rows of F), a fixed-order shuffle reduction
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int share = rank; share < kShares; share += NB) {
        double s = 0.0;
        for (int m = share + kShares * warp; m < NR; m += kShares * kWarps) {
            const double2 *f = F + (int64_t)m * NK;
            double re = 0.0, im = 0.0;
            for (int k = lane; k < NK; k += 32) {
                const double2 v = f[k];
                re = fma(v.x, x[k], re);
                im = fma(v.y, x[k], im);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                re += __shfl_xor_sync(0xffffffffu, re, o);
                im += __shfl_xor_sync(0xffffffffu, im, o);
            }
            const double2 t = target[m];
            const double2 dm = make_double2(re - t.x, im - t.y);
            if constexpr (NB == 1) {
                if (lane == 0) d[m] = dm;
            } else {
                if (lane < NB) cl.map_shared_rank(d, lane)[m] = dm;   // lane i to block i
            }
            s = fma(dm.x, dm.x, fma(dm.y, dm.y, s));
        }
        if (lane == 0) wsum[share][warp] = s;
    }
    __syncthreads();
    if (threadIdx.x < kShares && (NB == 1 || (int)threadIdx.x == rank)) {
        const double *v = wsum[threadIdx.x];
        const double sum = ((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7]));
        if constexpr (NB == 1) part[threadIdx.x] = sum;
        else cl.map_shared_rank(part, 0)[rank] = sum;
    }
    sync();                                                       // every share of d and its sum is written
    if (rank == 0 && threadIdx.x == 0) {
        double sum = 0.0;
        for (int i = 0; i < kShares; ++i) sum += part[i];
        R[b] = sum * inv_norm;
    }
    if (!grad) return;
    // 64 k by four quarters of the m; the quarters are added in order
    const int per = (NK + NB - 1) / NB, kt = threadIdx.x & 63, qt = threadIdx.x >> 6;
    for (int k0 = rank * per; k0 < min(NK, (rank + 1) * per); k0 += 64) {
        const int k = k0 + kt;
        const bool live = k < min(NK, (rank + 1) * per);
        double g = 0.0;
        if (live)
            for (int m = qt * ((NR + 3) / 4); m < min(NR, (qt + 1) * ((NR + 3) / 4)); ++m) {
                const double2 v = F[(int64_t)m * NK + k];
                g = fma(d[m].x, v.x, fma(d[m].y, v.y, g));        // Re(conj(d) F)
            }
        __syncthreads();
        red[threadIdx.x] = g;
        __syncthreads();
        if (live && qt == 0) grad[b * NK + k] = 2.0 * inv_norm * (red[kt] + red[64 + kt] + red[128 + kt] + red[192 + kt]);
    }
}

__global__ void __cluster_dims__(kShares, 1, 1) __launch_bounds__(kThreads)
    k_rspace_cluster(int NK, int NR, const double *__restrict__ rows, const double2 *__restrict__ F,
                     const double2 *__restrict__ target, double inv_norm, double *__restrict__ R, double *__restrict__ grad)
{
    rspace_row<kShares>(NK, NR, rows, F, target, inv_norm, R, grad);
}

__global__ void __launch_bounds__(kThreads)
    k_rspace_block(int NK, int NR, const double *__restrict__ rows, const double2 *__restrict__ F,
                   const double2 *__restrict__ target, double inv_norm, double *__restrict__ R, double *__restrict__ grad)
{
    rspace_row<1>(NK, NR, rows, F, target, inv_norm, R, grad);
}

}  // namespace
}  // namespace fg

using namespace fg;

extern "C" fg_status fg_rspace_misfit(int64_t B, int32_t NK, int32_t NR, const double *rows, const double *F,
                                      const double *target, double inv_norm, double *R, double *grad, void *stream)
{
    if (B < 0 || NK < 0 || NR < 0) return fail(FG_ERR_VALUE, "negative size");
    if (B == 0) return FG_OK;
    if (!rows || !F || !target || !R) return fail(FG_ERR_VALUE, "null argument");
    if (B > 0x7fffffffLL) return fail(FG_ERR_VALUE, "too many rows for one call");
    const size_t smem = (size_t)((NK + 1) & ~1) * sizeof(double) + (size_t)NR * sizeof(double2);
    if (smem > 200 * 1024) return fail(FG_ERR_VALUE, "NK and NR too large for one block's shared memory");
    const bool cluster = B <= kClusterRows;
    auto kern = cluster ? k_rspace_cluster : k_rspace_block;
    if (smem > 40 * 1024) FG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<(unsigned)(cluster ? B * kShares : B), kThreads, smem, static_cast<cudaStream_t>(stream)>>>(
        NK, NR, rows, reinterpret_cast<const double2 *>(F), reinterpret_cast<const double2 *>(target), inv_norm, R,
        grad);
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}
