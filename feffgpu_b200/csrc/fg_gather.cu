// fg_gather.cu -- the coordinates of paths held as atom indices, and their gradient summed onto the atoms (the reference
// forms them with torch indexing at every evaluation, src/feffgpu/exafs/forward.py:99-163, 664-725).
//
// Forward: a thread per (path, atom slot), relative vector to the absorber under the minimum image.  Backward: a block per
// atom over the path slots that hold it (a compressed list built once per path list), partial sums per thread and a
// fixed-order reduction -- no atomics, the same bits every time.  Bound by the latency of one pass over a few hundred
// kilobytes; as torch operations (index, subtract, divide, round, multiply, and the sorting backward of the index) the
// pair took about 200 us of a 4,438-path refinement step.
#include <cuda_runtime.h>

#include <algorithm>

#include "fg_launch.h"

namespace fg {
namespace {

constexpr int kThreads = 128;

// cell: null, or 18 doubles (the cell's rows, then its inverse); box: a cubic length, or not positive
__global__ void __launch_bounds__(kThreads) k_gather(int64_t total, int nleg_max, const double *__restrict__ pos,
                                                     const int64_t *__restrict__ atoms, const int *__restrict__ nleg,
                                                     double box, const double *__restrict__ cell, double *__restrict__ out)
{
    for (int64_t t = (int64_t)blockIdx.x * kThreads + threadIdx.x; t < total; t += (int64_t)gridDim.x * kThreads) {
        const int64_t p = t / nleg_max;
        const int j = (int)(t % nleg_max);
        double r[3] = {0.0, 0.0, 0.0};
        if (j > 0 && j < nleg[p]) {
            const double *a = pos + 3 * atoms[t], *a0 = pos + 3 * atoms[p * nleg_max];
#pragma unroll
            for (int c = 0; c < 3; ++c) r[c] = a[c] - a0[c];
            if (cell) {
                double f[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    f[c] = fma(r[2], cell[9 + 6 + c], fma(r[1], cell[9 + 3 + c], r[0] * cell[9 + c]));
                    f[c] -= rint(f[c]);
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) r[c] = fma(f[2], cell[6 + c], fma(f[1], cell[3 + c], f[0] * cell[c]));
            } else if (box > 0.0) {
#pragma unroll
                for (int c = 0; c < 3; ++c) r[c] = __dsub_rn(r[c], __dmul_rn(box, rint(r[c] / box)));
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) out[3 * t + c] = r[c];
    }
}

__global__ void __launch_bounds__(kThreads) k_scatter(int64_t natoms, int nleg_max, const int64_t *__restrict__ off,
                                                      const int *__restrict__ entry, const int *__restrict__ nleg,
                                                      const double *__restrict__ g, double *__restrict__ out)
{
    __shared__ double red[kThreads / 32][3];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int64_t a = blockIdx.x; a < natoms; a += gridDim.x) {
        double s[3] = {0.0, 0.0, 0.0};
        for (int64_t i = off[a] + threadIdx.x; i < off[a + 1]; i += kThreads) {
            const int t = entry[i], j = t % nleg_max;
            const double *v = g + 3 * (int64_t)t;
            if (j > 0) {
#pragma unroll
                for (int c = 0; c < 3; ++c) s[c] += v[c];
            } else {                                   // the absorber: minus every other slot of the path
                const int n = nleg[t / nleg_max];
                for (int q = 1; q < n; ++q)
#pragma unroll
                    for (int c = 0; c < 3; ++c) s[c] -= v[3 * q + c];
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int c = 0; c < 3; ++c) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
        if (lane == 0)
#pragma unroll
            for (int c = 0; c < 3; ++c) red[w][c] = s[c];
        __syncthreads();
        if (threadIdx.x < 3) out[3 * a + threadIdx.x] = (red[0][threadIdx.x] + red[1][threadIdx.x]) + (red[2][threadIdx.x] + red[3][threadIdx.x]);
        __syncthreads();
    }
}

}  // namespace
}  // namespace fg

using namespace fg;

extern "C" fg_status fg_path_gather(int64_t n, int32_t nleg_max, const double *pos, const int64_t *atoms,
                                    const int32_t *nleg, double box, const double *cell, double *coords, void *stream)
{
    if (n < 0 || nleg_max < 2 || nleg_max > kMaxLeg) return fail(FG_ERR_VALUE, "bad size");
    if (n == 0) return FG_OK;
    if (!pos || !atoms || !nleg || !coords) return fail(FG_ERR_VALUE, "null argument");
    const int64_t total = n * nleg_max;
    k_gather<<<(int)std::min<int64_t>((total + kThreads - 1) / kThreads, 148 * 32), kThreads, 0,
               static_cast<cudaStream_t>(stream)>>>(total, nleg_max, pos, atoms, nleg, box, cell, coords);
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

extern "C" fg_status fg_path_scatter(int64_t natoms, int32_t nleg_max, const int64_t *off, const int32_t *entry,
                                     const int32_t *nleg, const double *grad_coords, double *grad_pos, void *stream)
{
    if (natoms < 0 || nleg_max < 2 || nleg_max > kMaxLeg) return fail(FG_ERR_VALUE, "bad size");
    if (natoms == 0) return FG_OK;
    if (!off || !entry || !nleg || !grad_coords || !grad_pos) return fail(FG_ERR_VALUE, "null argument");
    k_scatter<<<(int)std::min<int64_t>(natoms, 148 * 64), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        natoms, nleg_max, off, entry, nleg, grad_coords, grad_pos);
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}
