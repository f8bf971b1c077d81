// k_pieces.cu — K6: rows in pieces: long rows in pieces of 256 to 2,048 nnz, a
// warp each, and the rows of small matrices in pieces of 64, eight lanes each
// (larger ones where a row would have more than 2,048 or 1,024 pieces).  FP64 and
// FP32-storage forms.
//
// A group of 32 lanes (or 8, with 8 for 32 in what follows) reads its piece
// straight from the caller's arrays, 32 nnz a step on 32-nnz boundaries; each lane
// sums its own nnz and the group's sums meet in one butterfly at the end.  A row of
// one piece is written at once.  A row of several keeps one partial sum per piece;
// the warp with the piece that finishes last (an atomic count per row that wraps to
// 0 by itself) adds them in piece order, so the result does not depend on which
// that was, and no second kernel is needed.  The plan is the list of pieces, 28
// bytes each, and no copy of the matrix.
//
// Why: on long rows the tiles' instructions (217 a 128-nnz tile) and L1 traffic
// (76 % of its data pipe) come before HBM, and every tile carries its row on; here
// 32 nnz take 32 instructions in all (tiles 51).  FP64, beta = 0, us on the device
// with 32 x 4 tiles and their fix-up and here: rows of lognormal length with
// columns in runs, 4,284 of 2,640 nnz in the mean 33.0 and 27.9, 20,000 of 2,000 108
// and 85; with random columns 5,000 x 2,000 nnz 48.5 and 44.0, 1,000 x 10,000 49.1
// and 46.9, 20,000 x 1,100 102.7 and 89.2, one row of 10M 67.0 and 47.7, of 1M 10.6
// and 10.9; lognormal with random columns, where L2's sectors bound both, 500 rows
// of 3,000 12.7 and 11.0, 2,000 of 1,600 19.5 and 20.0, 4,284 of 2,640 55.1 and 58.4
// (beta = 0.5: 59.7 and 58.5), 20,000 of 2,000 178 and 184 (187 and 184).  Rows of
// 310 17.0 vs 14.8, and with FP32 storage no difference, so both keep the tiles.
// Small matrices (a launch fewer): 60k power-law nnz 4.7 and 4.7 (beta = 0.5: 6.3
// and 5.2), one row of 65,536 among 300 rows 6.6 and 5.6.
// What bounds it: HBM on large matrices, the chain of column and x loads of a
// piece on small ones.  The count is one atomic with release and acquire: with
// fences around it 60k nnz took 5.0.
#include <stdint.h>

#include <algorithm>

#include "../sbb_internal.h"
#include "common.cuh"
#include "spmv_device.cuh"

namespace sbb {

namespace {

constexpr int NT = 64;  // threads per CTA
// Steps whose loads are in flight together, and the CTAs per SM that the launch
// bounds aim at (48 warps, 40 registers).  12M nnz in 4,284 rows, us, CTAs of 8
// warps: 4 steps at 32, 40, 48 and 56 warps 33.7, 33.8, 28.4, 37.3; 3 at 56 31.0; 6
// at 40 32.3; 8 at 24 29.9.  CTAs of 2 warps free their place sooner than of 8 and
// spread evenly over the SMs: 5,000 x 2,000 nnz 44.4 and 50.2, 2,000 rows of 1,600
// in pieces of 512 21.9 and 24.8.
constexpr int kPieceSteps = 4;
constexpr int kMinCtas = 24;
constexpr int kSumSteps = 8;  // partial sums of a row that a lane loads together

// Piece sizes, multiples of 32.  Of 32 lanes (`warps`: resident on the device): one
// piece a row when the rows are short enough and fill the device; else, when
// pieces of at most about 2,048 do, as many as fill 0.7 of it (3.3M nnz in 2,000
// rows, pieces of 256, 512, 768, 1,024: 21.9, 21.9, 20.5, 21.5 us; 1.6M in 500,
// 256, 384, 512, 1,024: 11.7, 11.5, 11.7, 13.3; 10M in 1,000, 768, 1,024, 2,048:
// 51.8, 52.0, 47.5); else 1,024 (11M nnz in 4,284 rows, 512, 768, 1,024, 1,536,
// 2,048: 29.7, 29.5, 27.9, 31.7, 31.8).  A row has at most kRowPieces8 or
// kRowPieces32 pieces, whose sums one warp adds (a row of 65,536 nnz, 256, 512 and
// 1,024 pieces of 8 lanes: 7.5, 6.1, 5.5 us).
constexpr int kRowPieces8 = 1024, kRowPieces32 = 2048;
int piece_size(int m, int nnz, int max_row, int width, long long warps)
{
    const int most = width == 8 ? kRowPieces8 : kRowPieces32;
    long long size = 64;
    if (width == 32) {
        const double room = 0.7 * warps - 0.5 * m;
        size = 1024;
        if (max_row <= 2048 - 31 && m >= 0.7 * warps)
            size = max_row + 31LL;
        else if (room > 0 && nnz <= 2304.0 * room)
            size = std::min(2048LL, std::max(256LL, (long long)(nnz / room)));
    }
    size = std::max(size, ((long long)max_row + most - 1) / most);
    return (int)((size + 31) / 32 * 32);
}

struct PiecesPlan {
    int pieces = 0, size = 0, width = 32;  // width: lanes per piece, 32 or 8
    int4 *piece = nullptr;       // row, first nnz, end, first slot of a row of several or -1
    double *carry = nullptr;     // partial sum of each piece of a row of several
    unsigned *ticket = nullptr;  // per row of several pieces (at its first slot): pieces done
    int *count = nullptr;        // counters of the build
};

// Pieces of row [lo, hi), cut on multiples of `width` nnz.
__device__ __forceinline__ int pieces_of(int lo, int hi, int size, int width)
{
    const long long n = ((long long)hi - (lo & -width) + size - 1) / size;
    return n > 1 ? (int)n : 1;  // an empty row has one too: it writes beta*y
}

// One more piece of a row done: the count before it, which wraps to 0 after
// `last`.  Release for this thread's partial sum, acquire for those counted.
__device__ __forceinline__ unsigned ticket_take(unsigned *t, unsigned last)
{
    unsigned old;
    asm volatile("atom.acq_rel.gpu.global.inc.u32 %0, [%1], %2;"
                 : "=r"(old)
                 : "l"(t), "r"(last)
                 : "memory");
    return old;
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
    // Of a row of several pieces: its ends, for the number of its pieces, on their
    // way while the piece is read.
    int row_lo = 0, row_hi = 0;
    if (pc.w >= 0) {
        row_lo = __ldg(rowptr + pc.x);
        row_hi = __ldg(rowptr + pc.x + 1);
    }
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
    if (sub == 0 && pc.w < 0 && pc.x >= 0) write_y(y + pc.x, alpha, sum, beta, stream);
    if (!__any_sync(0xffffffffu, pc.w >= 0)) return;
    const int np = pc.w >= 0 ? pieces_of(row_lo, row_hi, size, W) : 0;
    bool last = false;
    if (sub == 0 && pc.w >= 0) {
        __stcg(carry + i, sum);
        last = ticket_take(ticket + pc.w, (unsigned)np - 1u) == (unsigned)np - 1u;
    }
    // The sums of rows that are complete now; with __syncwarp() what the ticket
    // ordered for the lane that took it holds for the whole warp.
    unsigned rows = __ballot_sync(0xffffffffu, last);
    __syncwarp();
    while (rows) {
        const int src = __ffs(rows) - 1;
        rows &= rows - 1;
        const int first_slot = __shfl_sync(0xffffffffu, pc.w, src);
        const int count = __shfl_sync(0xffffffffu, np, src);
        double total = 0.0;
#pragma unroll 1
        for (int j = threadIdx.x & 31; j < count; j += 32 * kSumSteps) {
            double t[kSumSteps];
#pragma unroll
            for (int u = 0; u < kSumSteps; ++u)
                t[u] = j + 32 * u < count ? __ldcg(carry + first_slot + j + 32 * u) : 0.0;
#pragma unroll
            for (int u = 0; u < kSumSteps; ++u) total += t[u];
        }
        total = warp_sum(total);
        if (sub == 0 && (threadIdx.x & 31) == src) write_y(y + pc.x, alpha, total, beta, stream);
    }
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

// Warps of the 32-lane form that the device holds at a time.
long long resident_warps(bool f32)
{
    const LaunchShape ls =
        f32 ? cached_launch_shape<pieces_spmv_kernel<ProdF32, AccF32, 32>>(NT, 0)
            : cached_launch_shape<pieces_spmv_kernel<ProdF64, AccF64, 32>>(NT, 0);
    return (long long)ls.sms * ls.occ * (NT / 32);
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
    S->size = piece_size(p->m, p->nnz, p->max_row, S->width, resident_warps(p->f32));
    const long long cap = (long long)p->nnz / S->size + 2LL * p->m;
    if (cap > 0x7fffffffLL / 32) {
        set_error("row-piece plan: too many rows");
        return SBB_ERR_ARG;
    }
    auto al = [&](void **ptr, size_t bytes) {
        bytes = bytes ? bytes : 16;
        p->scratch_bytes += bytes;
        return dev_malloc_async(ptr, bytes, s) == cudaSuccess;
    };
    if (!al((void **)&S->count, 4 * sizeof(int)) || !al((void **)&S->piece, sizeof(int4) * cap) ||
        !al((void **)&S->carry, sizeof(double) * cap) ||
        !al((void **)&S->ticket, sizeof(unsigned) * cap)) {
        set_error("row-piece plan: device allocation failed");
        return SBB_ERR_NOMEM;
    }
    SBB_CUDA(cudaMemsetAsync(S->count, 0, 4 * sizeof(int), s));
    SBB_CUDA(cudaMemsetAsync(S->ticket, 0, sizeof(unsigned) * cap, s));
    if (p->m > 0) {
        const int grid = (int)std::min<long long>(((long long)p->m + 255) / 256, 148 * 16);
        pieces_list_kernel<<<grid, 256, 0, s>>>(p->rowptr, p->m, S->size, S->width, S->piece,
                                            (int)cap, S->count);
        launch_csr_check(p->rowptr, p->m, p->nnz, p->col, p->n, p->status, S->count + 2, s);
    }
    SBB_CUDA(cudaMemcpyAsync(&S->pieces, S->count, sizeof(int), cudaMemcpyDeviceToHost, s));
    SBB_CUDA(cudaStreamSynchronize(s));
    p->tiles = S->pieces;
    SBB_CUDA(cudaFreeAsync(S->count, s));
    S->count = nullptr;
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
    for (void *q : {(void *)S->piece, (void *)S->carry, (void *)S->ticket, (void *)S->count})
        if (q) cudaFreeAsync(q, s);
    delete S;
    p->pieces = nullptr;
}

}  // namespace sbb
