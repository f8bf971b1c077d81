// k_pieces.cu — K6: rows in pieces: long rows in pieces of at most 256 to 1,024
// nnz, a warp each, and the rows of small matrices in pieces of at most 64, eight
// lanes each (FP64 and FP32-storage forms).
//
// A group of 32 lanes (or 8, with 8 for 32 in what follows) reads its piece
// straight from the caller's arrays, 32 nnz a step on 32-nnz boundaries; each lane
// sums its own nnz and the group's sums meet in one butterfly at the end.  A row of one piece is written at once.  A row of several
// keeps one partial sum per piece; the group that finishes last (an atomic count
// per row that wraps to 0 by itself) adds them in piece order, so the result does
// not depend on which that was, and no second kernel is needed.  The plan is
// the list of pieces, 28 bytes each, and no copy of the matrix.
//
// Why: on such rows the tiles' instructions (217 a 128-nnz tile) and L1 traffic
// (76 % of its data pipe) come before HBM, and every tile carries its row on; here
// 32 nnz take 29 instructions in all (tiles 51).  FP64, against 32 x 4 tiles and their fix-up
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
// Pieces of groups of 8 lanes: 64 nnz.
int piece_size(int nnz, int width)
{
    if (width == 8) return 64;
    return nnz >= 1024 * 148 * 48 ? 1024 : (nnz >= 512 * 148 * 16 ? 512 : 256);
}

struct PiecesPlan {
    int pieces = 0, size = 0, width = 32;  // width: lanes per piece, 32 or 8
    int4 *piece = nullptr;       // row, first nnz, end, first slot of a row of several or -1
    double *carry = nullptr;     // partial sum of each piece of a row of several
    unsigned *ticket = nullptr;  // per row of several pieces (at its first slot): pieces done
};

// Pieces of row [lo, hi), cut on multiples of `width` nnz.
__device__ __forceinline__ int pieces_of(int lo, int hi, int size, int width)
{
    const long long n = ((long long)hi - (lo & -width) + size - 1) / size;
    return n > 1 ? (int)n : 1;  // an empty row has one too: it writes beta*y
}

// W lanes a piece; the 32 / W pieces of a warp run in step.
template <typename PT, typename ACC, int W>
__global__ void __launch_bounds__(NT, kMinCtas)
pieces_spmv_kernel(int n, int pieces, const int4 *__restrict__ piece,
                   const int *__restrict__ rowptr, const int *__restrict__ col,
                   const typename PT::V *__restrict__ val, const typename PT::V *__restrict__ x,
                   double *__restrict__ y, double alpha, double beta, double *carry,
                   unsigned *ticket, int size, unsigned *status)
{
    using V = typename PT::V;
    constexpr int U = kPieceSteps;
    const long long i = ((long long)blockIdx.x * NT + threadIdx.x) / W;
    if (((long long)blockIdx.x * NT + (threadIdx.x & ~31)) / W >= pieces) return;  // whole warps
    const int sub = threadIdx.x % W;
    const uint64_t keep = l2_evict_last(), stream = l2_evict_first();
    const int4 pc = i < pieces ? __ldg(piece + i) : make_int4(-1, 0, 0, -1);
    const unsigned first = (unsigned)pc.y, end = (unsigned)pc.z;
    // unsigned: a lane's index runs to less than 64 * U past the last nnz
    unsigned k = (first & -(unsigned)W) + sub, bad = 0;
    unsigned steps = (end - (first & -(unsigned)W) + W - 1) / W;
    if (W < 32) steps = __reduce_max_sync(0xffffffffu, steps);
    ACC acc;
    acc.zero();
    int c[U];
    V v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const bool p = k + W * u - first < end - first;
        c[u] = ld_stream_if(col + k + W * u, p);
        v[u] = ld_stream_if(val + k + W * u, p);
    }
#pragma unroll 1
    for (unsigned b = 0; b < steps; b += U) {
        V xv[U], vn[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool p = k + W * u - first < end - first, ok = (unsigned)c[u] < (unsigned)n;
            bad |= p && !ok;
            xv[u] = ld_keep_if(x + c[u], p && ok, keep);
        }
        const unsigned kn = k + W * U;
#pragma unroll
        for (int u = 0; u < U; ++u) {  // the next steps, while x is on its way
            const bool p = kn + W * u < end;
            c[u] = ld_stream_if(col + kn + W * u, p);
            vn[u] = ld_stream_if(val + kn + W * u, p);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (k + W * u - first < end - first) acc.mac(v[u], xv[u]);
            v[u] = vn[u];
        }
        k = kn;
    }
    if (bad) atomicOr(status, ST_BAD_COL);
    double sum = acc.get();
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o, W);
    if (pc.w < 0) {
        if (sub == 0 && pc.x >= 0) write_y(y + pc.x, alpha, sum, beta, stream);
        return;
    }
    // the lanes of a piece stay together from here
    const unsigned mine = W == 32 ? 0xffffffffu : ((1u << (W & 31)) - 1u) << ((threadIdx.x & 31) / W * W);
    const int np = pieces_of(__ldg(rowptr + pc.x), __ldg(rowptr + pc.x + 1), size, W);
    unsigned done = 0;
    if (sub == 0) {
        __stcg(carry + i, sum);
        __threadfence();
        done = atomicInc(ticket + pc.w, (unsigned)np - 1u);
    }
    done = __shfl_sync(mine, done, 0, W);
    if (done != (unsigned)np - 1u) return;
    __threadfence();
    sum = 0.0;
#pragma unroll 4
    for (int j = sub; j < np; j += W) sum += __ldcg(carry + pc.w + j);
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(mine, sum, o, W);
    if (sub == 0) write_y(y + pc.x, alpha, sum, beta, stream);
}

// Numbers the pieces of every row, those of 32 consecutive rows in order, by a
// device counter: which slots the rows get depends on the order of the atomics,
// their sums do not.
__global__ void __launch_bounds__(256)
pieces_list_kernel(const int *__restrict__ rowptr, int m, int size, int width,
                   int4 *__restrict__ piece, int cap, int *count)
{
    const int lane = threadIdx.x & 31;
    for (long long r0 = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); r0 < m;
         r0 += (long long)gridDim.x * blockDim.x) {
        const long long r = r0 + lane;
        int lo = 0, hi = 0, np = 0;
        if (r < m) {
            lo = __ldg(rowptr + r);
            hi = __ldg(rowptr + r + 1);
            np = pieces_of(lo, hi, size, width);
        }
        int slot = np;  // inclusive scan over the 32 rows
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, slot, o);
            if (lane >= o) slot += u;
        }
        int base = 0;
        if (lane == 31) base = atomicAdd(count, slot);
        slot += __shfl_sync(0xffffffffu, base, 31) - np;
        for (int j = 0; j < np && slot + j < cap; ++j) {
            const long long a = (long long)(lo & -width) + (long long)j * size;
            piece[slot + j] = make_int4((int)r, j == 0 ? lo : (int)a,
                                        (int)(a + size < hi ? a + size : hi), np > 1 ? slot : -1);
        }
    }
}

template <typename PT, typename ACC>
void launch_pieces_t(const PiecesPlan &S, const Plan *p, double alpha, const void *x, double beta,
                     double *y, cudaStream_t s)
{
    using V = typename PT::V;
    hook_start(s);
    const auto kern =
        S.width == 8 ? pieces_spmv_kernel<PT, ACC, 8> : pieces_spmv_kernel<PT, ACC, 32>;
    kern<<<(int)(((long long)S.pieces * S.width + NT - 1) / NT), NT, 0, s>>>(
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
    S->width = p->vector_width;
    S->size = piece_size(p->nnz, S->width);
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
        pieces_list_kernel<<<grid, 256, 0, s>>>(p->rowptr, p->m, S->size, S->width, S->piece,
                                            (int)cap, count);
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
