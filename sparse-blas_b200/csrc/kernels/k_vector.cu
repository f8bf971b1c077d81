// k_vector.cu — K1: vector CSR SpMV, V lanes per row (V = 2..32).
//
// Replaces cusparseDcsrmv (SparseBLAS/src/dspmv_mgpu_v1.cu:200-204,
// src/dspmv_mgpu_baseline.cu:163-167).  A warp takes chunks of rows; in a
// chunk a group of V lanes owns one row at a time, reads its col/val with
// coalesced streaming loads (V consecutive nnz per step), gathers x through
// the read-only path and reduces with warp shuffles (xor butterfly: the order
// is fixed for a given V), with several rows' loads in flight per group
// (vector_rows).  Good for regular matrices whose row lengths are close to
// V; long rows serialise on one group.
#include <algorithm>

#include "../sbb_internal.h"
#include "common.cuh"
#include "spmv_device.cuh"

namespace sbb {

namespace {

constexpr int VT = 256;  // threads per CTA

// Warp w of the grid takes rows [w * share, (w + 1) * share), the chunks shared out
// evenly.  The share follows from the grid: as an eleventh parameter it made every
// call 0.25 us longer (2.9 and 3.2 us of the host's time).
template <typename PT, typename ACC, int V, bool AHEAD>
__global__ void __launch_bounds__(VT, 4)
vector_kernel(int m, int n, const int *__restrict__ rowptr, const int *__restrict__ col,
              const typename PT::V *__restrict__ val, const typename PT::V *__restrict__ x,
              double *__restrict__ y, double alpha, double beta, unsigned *status)
{
    constexpr unsigned CR = vector_chunk(V);
    const unsigned warps = gridDim.x * (VT / 32), chunks = ((unsigned)m + CR - 1) / CR;
    // the smallest k (8 at most) with k * warps >= chunks, without a division
    unsigned k = (unsigned)__fdividef((float)chunks, (float)warps);
    k += k * warps < chunks;
    k += k * warps < chunks;
    const int share = (int)(CR * k);
    const long long r0 = ((long long)blockIdx.x * (VT / 32) + (threadIdx.x >> 5)) * share;
    if (r0 >= m) return;
    unsigned bad = 0;
    vector_rows<PT, ACC, V, AHEAD>((int)r0, (int)min((long long)share, m - r0), n, rowptr, col, val,
                                   x, y, alpha, beta, l2_evict_first(), bad);
    if (bad) atomicOr(status, ST_BAD_COL);
}

template <typename PT, typename ACC, int V>
void launch_vector_v(const CsrView &A, double alpha, const typename PT::V *x, double beta,
                     double *y, unsigned *status, cudaStream_t s)
{
    // FP32 storage when a warp has several chunks: nothing runs ahead in a row or
    // into L2 (us with both, with neither: 1M rows of 38 120.9 and 108.7, 1.3M of 2
    // 19.1 and 18.4, 100,000 of 150 37.9 and 37.3; 30,000 of 60, a chunk a warp, 8.4
    // and 8.9).
    constexpr bool kAhead = sizeof(typename PT::V) == 8;
    constexpr auto kern = vector_kernel<PT, ACC, V, true>;
    constexpr auto plain = vector_kernel<PT, ACC, V, kAhead>;
    const LaunchShape ls = cached_launch_shape<kern>(VT, 0);
    // Shares of a few chunks: enough for the prefetches to run ahead, small
    // enough that the warps end together.
    const long long warps = (long long)ls.sms * ls.occ * (VT / 32);
    const long long chunks = ((long long)A.m + vector_chunk(V) - 1) / vector_chunk(V);
    const long long share = std::min<long long>(8, std::max<long long>(1, chunks / (2 * warps)));
    const long long need = (chunks + share - 1) / share;
    hook_start(s);
    (share > 1 ? plain : kern)<<<(int)((need * 32 + VT - 1) / VT), VT, 0, s>>>(
        A.m, A.n, A.rowptr, A.col, static_cast<const typename PT::V *>(A.val), x, y, alpha, beta,
        status);
    hook_stop(s);
}

template <typename PT, typename ACC>
void launch_vector_t(const CsrView &A, int V, double alpha, const typename PT::V *x,
                     double beta, double *y, unsigned *status, cudaStream_t s)
{
    if (A.m <= 0) return;
    switch (V) {
    case 2: launch_vector_v<PT, ACC, 2>(A, alpha, x, beta, y, status, s); break;
    case 4: launch_vector_v<PT, ACC, 4>(A, alpha, x, beta, y, status, s); break;
    case 8: launch_vector_v<PT, ACC, 8>(A, alpha, x, beta, y, status, s); break;
    case 16: launch_vector_v<PT, ACC, 16>(A, alpha, x, beta, y, status, s); break;
    case 32: launch_vector_v<PT, ACC, 32>(A, alpha, x, beta, y, status, s); break;
    default: break;
    }
}

}  // namespace

void launch_vector(const CsrView &A, int V, double alpha, const double *x, double beta,
                   double *y, unsigned *status, cudaStream_t s)
{
    launch_vector_t<ProdF64, AccF64>(A, V, alpha, x, beta, y, status, s);
}

void launch_vector_f32(const CsrView &A, int V, double alpha, const float *x, double beta,
                       double *y, unsigned *status, cudaStream_t s)
{
    launch_vector_t<ProdF32, AccF32>(A, V, alpha, x, beta, y, status, s);
}

}  // namespace sbb
