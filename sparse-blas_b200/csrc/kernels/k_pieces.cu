// k_pieces.cu — K6: long rows in pieces of at most 256 to 1,024 nnz, a warp each
// (FP64 and FP32-storage forms).
//
// For matrices whose rows are long (hundreds of nnz and more in the mean): a
// warp reads its piece straight from the caller's arrays, 32 nnz a step on 32-nnz
// boundaries, each lane sums its own nnz and the warp's sums meet in one
// butterfly at the end.  A row of one piece is written at once.  A row of several
// keeps one partial sum per piece; the warp that finishes last (an atomic count
// per row that wraps to 0 by itself) adds them in piece order, so the result does
// not depend on which warp that was, and no second kernel is needed.  The plan is
// the list of pieces, 28 bytes each, and no copy of the matrix.
//
// Why: on such rows the tiles' instructions (217 a 128-nnz tile) and L1 traffic
// (76 % of its data pipe) come before HBM, and every tile carries its row on; here
// 32 nnz take about 14 instructions.  FP64, against 32 x 4 tiles and their fix-up
// (us): 4,284 rows of 2,770 in the mean 28.4 vs 32.1, 20,000 of 2,670 114 vs 124
// (5.6 TB/s), 2,000 of 1,590 12.9 vs 14.4, 20,000 of 1,020 52.9 vs 53.0; rows of
// 310 17.0 vs 14.8, and with FP32 storage no difference, so both keep the tiles.
// What bounds it: HBM on large matrices, the chain of column and x loads of a
// piece on small ones.
#include <stdint.h>

#include <algorithm>

#include "../sbb_internal.h"
#include "common.cuh"
#include "spmv_device.cuh"

namespace sbb {

namespace {

constexpr int NT = 256;  // threads per CTA
// Steps whose loads are in flight together, and the CTAs per SM that the launch
// bounds aim at (40 registers).  12M nnz in 4,284 rows, us: 4 steps at 4, 5, 6 and
// 7 CTAs 33.7, 33.8, 28.4, 37.3; 3 at 7 31.0; 6 at 5 32.3; 8 at 3 29.9.
constexpr int kPieceSteps = 4;
constexpr int kMinCtas = 6;
// Piece sizes (multiples of 32): 1,024 nnz where that makes a piece for every
// resident warp, smaller ones for smaller matrices (12M nnz, pieces of 512, 768,
// 1,024, 2,048: 31.1, 30.8, 28.4, 36.8 us; 0.7M nnz, 512 and 1,024: 7.9, 10.8).
int piece_size(int nnz)
{
    return nnz >= 1024 * 148 * 48 ? 1024 : (nnz >= 512 * 148 * 16 ? 512 : 256);
}

struct PiecesPlan {
    int pieces = 0, size = 0;
    int4 *piece = nullptr;       // row, first nnz, end, first slot of a row of several or -1
    double *carry = nullptr;     // partial sum of each piece of a row of several
    unsigned *ticket = nullptr;  // per row of several pieces (at its first slot): pieces done
};

__device__ __forceinline__ int pieces_of(int lo, int hi, int size)
{
    const long long n = ((long long)hi - (lo & ~31) + size - 1) / size;
    return n > 1 ? (int)n : 1;  // an empty row has one too: it writes beta*y
}

template <typename PT, typename ACC>
__global__ void __launch_bounds__(NT, kMinCtas)
pieces_spmv_kernel(int n, int pieces, const int4 *__restrict__ piece,
                   const int *__restrict__ rowptr, const int *__restrict__ col,
                   const typename PT::V *__restrict__ val, const typename PT::V *__restrict__ x,
                   double *__restrict__ y, double alpha, double beta, double *carry,
                   unsigned *ticket, int size, unsigned *status)
{
    using V = typename PT::V;
    constexpr int U = kPieceSteps;
    const int i = (int)(((long long)blockIdx.x * NT + threadIdx.x) >> 5);
    if (i >= pieces) return;
    const int lane = threadIdx.x & 31;
    const uint64_t keep = l2_evict_last(), stream = l2_evict_first();
    const int4 pc = __ldg(piece + i);
    const unsigned first = (unsigned)pc.y, end = (unsigned)pc.z;
    // unsigned: a lane's index runs to less than 64 * U past the last nnz
    unsigned k = (first & ~31u) + lane, bad = 0;
    ACC acc;
    acc.zero();
    int c[U];
    V v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const bool p = k + 32 * u - first < end - first;
        c[u] = ld_stream_if(col + k + 32 * u, p);
        v[u] = ld_stream_if(val + k + 32 * u, p);
    }
#pragma unroll 1
    for (unsigned b = first & ~31u; b < end; b += 32 * U) {
        V xv[U], vn[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool p = k + 32 * u - first < end - first, ok = (unsigned)c[u] < (unsigned)n;
            bad |= p && !ok;
            xv[u] = ld_keep_if(x + c[u], p && ok, keep);
        }
        const unsigned kn = k + 32 * U;
#pragma unroll
        for (int u = 0; u < U; ++u) {  // the next steps, while x is on its way
            const bool p = kn + 32 * u < end;
            c[u] = ld_stream_if(col + kn + 32 * u, p);
            vn[u] = ld_stream_if(val + kn + 32 * u, p);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (k + 32 * u - first < end - first) acc.mac(v[u], xv[u]);
            v[u] = vn[u];
        }
        k = kn;
    }
    if (bad) atomicOr(status, ST_BAD_COL);
    double sum = warp_sum(acc.get());
    if (pc.w < 0) {
        if (lane == 0) write_y(y + pc.x, alpha, sum, beta, stream);
        return;
    }
    const int np = pieces_of(__ldg(rowptr + pc.x), __ldg(rowptr + pc.x + 1), size);
    unsigned done = 0;
    if (lane == 0) {
        __stcg(carry + i, sum);
        __threadfence();
        done = atomicInc(ticket + pc.w, (unsigned)np - 1u);
    }
    done = __shfl_sync(0xffffffffu, done, 0);
    if (done != (unsigned)np - 1u) return;
    __threadfence();
    sum = 0.0;
#pragma unroll 4
    for (int j = lane; j < np; j += 32) sum += __ldcg(carry + pc.w + j);
    sum = warp_sum(sum);
    if (lane == 0) write_y(y + pc.x, alpha, sum, beta, stream);
}

// Numbers the pieces of every row by a device counter: which slots a row gets
// depends on the order of the atomics, its sum does not.
__global__ void __launch_bounds__(256)
pieces_list_kernel(const int *__restrict__ rowptr, int m, int size, int4 *__restrict__ piece,
                   int cap, int *count)
{
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < m;
         r += (long long)gridDim.x * blockDim.x) {
        const int lo = __ldg(rowptr + r), hi = __ldg(rowptr + r + 1);
        const int np = pieces_of(lo, hi, size);
        const int slot = atomicAdd(count, np);
        for (int j = 0; j < np && slot + j < cap; ++j) {
            const long long a = (long long)(lo & ~31) + (long long)j * size;
            piece[slot + j] = make_int4((int)r, j == 0 ? lo : (int)a,
                                        (int)(a + size < hi ? a + size : hi),
                                        np > 1 ? slot : -1);
        }
    }
}

template <typename PT, typename ACC>
void launch_pieces_t(const PiecesPlan &S, const Plan *p, double alpha, const void *x, double beta,
                     double *y, cudaStream_t s)
{
    using V = typename PT::V;
    hook_start(s);
    pieces_spmv_kernel<PT, ACC><<<(int)(((long long)S.pieces * 32 + NT - 1) / NT), NT, 0, s>>>(
        p->n, S.pieces, S.piece, p->rowptr, p->col, static_cast<const V *>(p->val),
        static_cast<const V *>(x), y, alpha, beta, S.carry, S.ticket, S.size,
        p->status);
    hook_stop(s);
}

}  // namespace

// The plan's status word gets ST_BAD_COL for a column out of range.
int pieces_build(Plan *p, cudaStream_t s)
{
    auto *S = new PiecesPlan();
    p->pieces = S;
    S->size = piece_size(p->nnz);
    const long long cap = (long long)p->nnz / S->size + 2LL * p->m;
    if (cap > 0x7fffffffLL / 32) {
        set_error("row-piece plan: too many rows");
        return SBB_ERR_ARG;
    }
    int *count = nullptr;
    auto al = [&](void **ptr, size_t bytes) {
        bytes = bytes ? bytes : 16;
        p->scratch_bytes += bytes;
        return dev_malloc_async(ptr, bytes, s) == cudaSuccess;
    };
    if (!al((void **)&count, 4 * sizeof(int)) || !al((void **)&S->piece, sizeof(int4) * cap) ||
        !al((void **)&S->carry, sizeof(double) * cap) ||
        !al((void **)&S->ticket, sizeof(unsigned) * cap)) {
        set_error("row-piece plan: device allocation failed");
        return SBB_ERR_NOMEM;
    }
    SBB_CUDA(cudaMemsetAsync(count, 0, 4 * sizeof(int), s));
    SBB_CUDA(cudaMemsetAsync(S->ticket, 0, sizeof(unsigned) * cap, s));
    if (p->m > 0) {
        const int grid = (int)std::min<long long>(((long long)p->m + 255) / 256, 148 * 16);
        pieces_list_kernel<<<grid, 256, 0, s>>>(p->rowptr, p->m, S->size, S->piece, (int)cap, count);
        launch_csr_check(p->rowptr, p->m, p->nnz, p->col, p->n, p->status, count + 2, s);
    }
    SBB_CUDA(cudaMemcpyAsync(&S->pieces, count, sizeof(int), cudaMemcpyDeviceToHost, s));
    SBB_CUDA(cudaStreamSynchronize(s));
    p->tiles = S->pieces;
    SBB_CUDA(cudaFreeAsync(count, s));
    SBB_CUDA(cudaGetLastError());
    return SBB_OK;
}

int pieces_run(Plan *p, double alpha, const void *x, double beta, double *y, cudaStream_t s)
{
    auto *S = static_cast<PiecesPlan *>(p->pieces);
    if (!S) {
        set_error("row-piece plan missing");
        return SBB_ERR_ARG;
    }
    if (p->f32)
        launch_pieces_t<ProdF32, AccF32>(*S, p, alpha, x, beta, y, s);
    else
        launch_pieces_t<ProdF64, AccF64>(*S, p, alpha, x, beta, y, s);
    SBB_CUDA(cudaGetLastError());
    return SBB_OK;
}

void pieces_free(Plan *p, cudaStream_t s)
{
    auto *S = static_cast<PiecesPlan *>(p->pieces);
    if (!S) return;
    for (void *q : {(void *)S->piece, (void *)S->carry, (void *)S->ticket})
        if (q) cudaFreeAsync(q, s);
    delete S;
    p->pieces = nullptr;
}

}  // namespace sbb
