// k_sliced.cu — K5: row slices for short, even rows (FP64 and FP32-storage
// forms).
//
// W lanes own a row and a warp a slice of 32/W consecutive rows; lane i of a
// row takes its nnz i, i + W, i + 2W, ...  The plan keeps a copy of the nnz in
// the order in which a warp needs them: step j of a slice holds the nnz of
// every lane that has a j-th one, in lane order, without padding.  So the
// columns and values of a step are contiguous whatever the row lengths, a
// lane's place in them is a count of the lanes before it, and a row's sum
// takes log2(W) shuffles.  Row lengths and the slice's place come from the
// caller's row pointer; the copy is all that the plan adds.
//
// Why: the vector kernel reads the caller's arrays with V lanes a row, and on
// short rows its issue slots (61 % used; 96 warp instructions per 24-nnz row,
// most of them in the butterflies and the ragged ends of each row) and
// latency come before HBM (24 %).  Here 32 nnz take 40 instructions in
// all, 128 there.  Measured against it (FP64, beta = 0.5; us): 200k rows of 24
// nnz in a band 13.6 vs 26.7; 500k rows of 6 10.6 vs 19.1; 100k rows of 50 in
// diagonal blocks 14.4 vs 21.5; 1M rows of 40 in a band 91.6 vs 136.5 (5.5 TB/s);
// 700k rows of 0 to 8, half of them empty, 12.0 vs 16.3; FP32 storage, 200k
// rows of 24, 12.7 vs 24.3.  What bounds it now: HBM on the largest of these,
// on the others the chain of row pointer, column and x loads of each slice and
// one to three waves of warps.
#include <stdint.h>

#include "../sbb_internal.h"
#include "common.cuh"
#include "lane_index.cuh"

namespace sbb {

namespace {

constexpr int ST = 256;  // threads per CTA
// Steps whose loads are in flight together, and the CTAs per SM that the
// launch bounds aim at (40 registers).  What counts is warps times loads in
// flight: 4 steps at 6 CTAs ran the 200k-row banded matrix in 14.4 us, 8 steps
// at 5 and 4 CTAs in 18.6 and 17.7, 4 steps at 8 CTAs (32 registers) in 16.9;
// with no bound the compiler unrolls the step loops to 148 registers, 53 us.
constexpr int kSteps = 4;
constexpr int kMinCtas = 6;
// Slices of up to this many nnz in the mean are brought into L2 as a whole
// when their place is known, so that HBM's latency is paid once and not every
// kSteps steps (us, without and with: 100k rows of 12 7.1 and 5.9, 500k of 6
// 11.8 and 10.6, 200k of 24 14.4 and 13.6, 100k of 50 14.9 and 14.4); in longer
// ones the loads in flight are enough and the prefetches only crowd L2 (rows of
// 100, 800 nnz a slice: 26.4 and 32.7; of 40, 640 nnz: 91.9 and 97.3).
constexpr int kPrefetchNnz = 448;

struct SlicedPlan {
    int width = 1;  // lanes per row
    int *col = nullptr;
    void *val = nullptr;
};

// What a lane knows of its slice: its row (-1: none; sub-lane 0 writes it), the
// slice's first nnz and their number, how many nnz the lane takes, the steps of
// the slice and those that every lane takes part in.  J counts steps: int, and
// unsigned for rows of more than 2^30 nnz, where a count runs past int (us with
// int and unsigned: 80,000 rows of 105 26.6 and 28.0, FP32 storage 22.3 and 23.1).
template <typename J> struct SliceLane {
    int row;
    unsigned base, total;
    int start, len;
    J mine, steps, full;
};
template <int W, typename J>
__device__ __forceinline__ SliceLane<J> slice_lane(int s, int m, const int *__restrict__ rowptr)
{
    constexpr int R = 32 / W;
    const int lane = threadIdx.x & 31, sub = lane % W;
    const int in_slice = min(R, m - s * R);  // rows; s * R < m
    SliceLane<J> L;
    L.row = s * R + lane / W;
    L.start = 0;
    L.len = 0;
    if (lane / W < in_slice) {
        L.start = __ldg(rowptr + L.row);
        L.len = __ldg(rowptr + L.row + 1) - L.start;
    } else {
        L.row = -1;
    }
    L.base = (unsigned)__shfl_sync(0xffffffffu, L.start, 0);
    L.total = __reduce_add_sync(0xffffffffu, sub == 0 ? (unsigned)L.len : 0u);
    L.mine = (J)lane_share((unsigned)L.len, sub, W);
    L.steps = __reduce_max_sync(0xffffffffu, L.mine);
    L.full = __reduce_min_sync(0xffffffffu, L.mine);
    return L;
}

template <typename PT, typename ACC, int W, bool PREFETCH, typename J>
__global__ void __launch_bounds__(ST, kMinCtas)
sliced_kernel(int m, int slices, const int *__restrict__ rowptr, const int *__restrict__ col,
              const typename PT::V *__restrict__ val, const typename PT::V *__restrict__ x,
              double *__restrict__ y, double alpha, double beta)
{
    using V = typename PT::V;
    const int s = (int)(((long long)blockIdx.x * ST + threadIdx.x) >> 5);
    if (s >= slices) return;
    const int lane = threadIdx.x & 31;
    const uint64_t keep = l2_evict_last(), stream = l2_evict_first();
    const SliceLane<J> L = slice_lane<W, J>(s, m, rowptr);
    if (PREFETCH && L.steps > kSteps && lane == 0) {
        prefetch_l2(col + L.base, 4 * (size_t)L.total);
        prefetch_l2(val + L.base, sizeof(V) * (size_t)L.total);
    }
    const bool writes = L.row >= 0 && lane % W == 0;
    double yv = 0.0;
    if (writes && beta != 0.0) yv = ld_y(y + L.row, stream);
    ACC acc;
    acc.zero();
    // steps of all 32 lanes: no predicates, constant offsets
    const int *cp = col + L.base + lane;
    const V *vp = val + L.base + lane;
    J j = 0;
#pragma unroll 1
    for (; j + kSteps <= L.full; j += kSteps) {
        int c[kSteps];
        V v[kSteps], xv[kSteps];
#pragma unroll
        for (int u = 0; u < kSteps; ++u) {
            c[u] = ld_stream(cp + 32 * u);
            v[u] = ld_stream(vp + 32 * u);
        }
#pragma unroll
        for (int u = 0; u < kSteps; ++u) xv[u] = ld_keep(x + c[u], keep);
#pragma unroll
        for (int u = 0; u < kSteps; ++u) acc.mac(v[u], xv[u]);
        cp += 32 * kSteps;
        vp += 32 * kSteps;
    }
    unsigned at = L.base + 32u * (unsigned)j;
    const unsigned before = (1u << lane) - 1u;
#pragma unroll 1
    for (; j < L.steps; j += kSteps) {
        int c[kSteps];
        V v[kSteps], xv[kSteps];
#pragma unroll
        for (int u = 0; u < kSteps; ++u) {
            const bool p = j + u < L.mine;
            const unsigned who = __ballot_sync(0xffffffffu, p);
            const unsigned k = at + __popc(who & before);
            at += __popc(who);
            c[u] = ld_stream_if(col + k, p);
            v[u] = ld_stream_if(val + k, p);
        }
#pragma unroll
        for (int u = 0; u < kSteps; ++u) xv[u] = ld_keep_if(x + c[u], j + u < L.mine, keep);
#pragma unroll
        for (int u = 0; u < kSteps; ++u)
            if (j + u < L.mine) acc.mac(v[u], xv[u]);
    }
    double sum = acc.get();
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o, W);
    if (writes) st_y(y + L.row, y_update(alpha, sum, beta, yv), stream);
}

constexpr int kFillWarps = 4;
constexpr int kFillNnz = 1024;  // nnz of a slice staged in shared memory

// Copies a slice's nnz into step order, one warp per slice: read in order,
// staged in shared memory and written in step order, so both sides coalesce;
// a slice of more than kFillNnz nnz is read step by step.  Columns are
// range-checked here, so the product trusts the copy.
template <typename V, int W>
__global__ void __launch_bounds__(kFillWarps * 32)
slice_fill_kernel(const int *__restrict__ rowptr, int m, int n, int slices,
                  const int *__restrict__ col, const V *__restrict__ val, int *__restrict__ scol,
                  V *__restrict__ sval, unsigned *status)
{
    __shared__ V s_val[kFillWarps][kFillNnz];
    __shared__ int s_col[kFillWarps][kFillNnz];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s = (int)((long long)blockIdx.x * kFillWarps + warp);
    if (s >= slices) return;  // no block-wide barrier follows
    const SliceLane<unsigned> L = slice_lane<W, unsigned>(s, m, rowptr);
    const unsigned total = L.total;
    const bool staged = total <= kFillNnz;
    bool bad = false;
    if (staged) {
        for (unsigned k = lane; k < total; k += 32) {
            int c = ld_stream(col + L.base + k);
            if ((unsigned)c >= (unsigned)n) bad = true, c = 0;
            s_col[warp][k] = c;
            s_val[warp][k] = ld_stream(val + L.base + k);
        }
        __syncwarp();
    }
    unsigned at = L.base;
    const unsigned before = (1u << lane) - 1u;
    for (unsigned j = 0; j < L.steps; ++j) {
        const bool p = j < L.mine;
        const unsigned who = __ballot_sync(0xffffffffu, p);
        if (p) {
            const unsigned from = (unsigned)L.start + j * W + lane % W;
            int c;
            V v;
            if (staged) {
                c = s_col[warp][from - L.base];
                v = s_val[warp][from - L.base];
            } else {
                c = __ldg(col + from);
                v = __ldg(val + from);
                if ((unsigned)c >= (unsigned)n) bad = true, c = 0;
            }
            const unsigned k = at + __popc(who & before);
            scol[k] = c;
            sval[k] = v;
        }
        at += __popc(who);
    }
    if (bad) atomicOr(status, ST_BAD_COL);
}

template <int W> int slices_of(int m) { return (int)(((long long)m + 32 / W - 1) / (32 / W)); }

template <typename V, int W> void fill_w(Plan *p, SlicedPlan *S, cudaStream_t s)
{
    const int slices = slices_of<W>(p->m);
    slice_fill_kernel<V, W><<<(slices + kFillWarps - 1) / kFillWarps, kFillWarps * 32, 0, s>>>(
        p->rowptr, p->m, p->n, slices, p->col, static_cast<const V *>(p->val), S->col,
        static_cast<V *>(S->val), p->status);
}

template <typename PT, typename ACC, int W>
void run_w(const SlicedPlan &S, const Plan *p, double alpha, const void *x, double beta, double *y,
           cudaStream_t s)
{
    using V = typename PT::V;
    const int slices = slices_of<W>(p->m);
    const auto kern = p->max_row > 1 << 30 ? sliced_kernel<PT, ACC, W, false, unsigned>
                      : (long long)p->nnz <= (long long)kPrefetchNnz * slices
                          ? sliced_kernel<PT, ACC, W, true, int>
                          : sliced_kernel<PT, ACC, W, false, int>;
    hook_start(s);
    kern<<<(int)(((long long)slices * 32 + ST - 1) / ST), ST, 0, s>>>(
        p->m, slices, p->rowptr, S.col, static_cast<const V *>(S.val), static_cast<const V *>(x), y,
        alpha, beta);
    hook_stop(s);
}

}  // namespace

#define SBB_SLICED_W(CALL)                                                       \
    switch (S->width) {                                                          \
    case 1: CALL(1); break;                                                      \
    case 2: CALL(2); break;                                                      \
    case 4: CALL(4); break;                                                      \
    case 8: CALL(8); break;                                                      \
    default: CALL(16); break;                                                    \
    }

int sliced_build(Plan *p, cudaStream_t s)
{
    auto *S = new SlicedPlan();
    p->sliced = S;
    S->width = p->vector_width;
    const size_t vb = p->f32 ? 4 : 8;
    auto al = [&](void **ptr, size_t bytes) {
        bytes = bytes ? bytes : 16;
        p->scratch_bytes += bytes;
        return dev_malloc_async(ptr, bytes, s) == cudaSuccess;
    };
    // 16 bytes more than the nnz: prefetches run to the next 16-byte boundary
    if (!al((void **)&S->col, sizeof(int) * (size_t)p->nnz + 16) ||
        !al(&S->val, vb * (size_t)p->nnz + 16)) {
        set_error("sliced plan: device allocation failed");
        return SBB_ERR_NOMEM;
    }
    if (p->m > 0) {
#define SBB_FILL(W) (p->f32 ? fill_w<float, W>(p, S, s) : fill_w<double, W>(p, S, s))
        SBB_SLICED_W(SBB_FILL)
#undef SBB_FILL
    }
    SBB_CUDA(cudaGetLastError());
    return SBB_OK;
}

int sliced_run(Plan *p, double alpha, const void *x, double beta, double *y, cudaStream_t s)
{
    auto *S = static_cast<SlicedPlan *>(p->sliced);
    if (!S) {
        set_error("sliced plan missing");
        return SBB_ERR_ARG;
    }
#define SBB_RUN(W)                                                               \
    (p->f32 ? run_w<ProdF32, AccF32, W>(*S, p, alpha, x, beta, y, s)             \
            : run_w<ProdF64, AccF64, W>(*S, p, alpha, x, beta, y, s))
    SBB_SLICED_W(SBB_RUN)
#undef SBB_RUN
    SBB_CUDA(cudaGetLastError());
    return SBB_OK;
}

void sliced_free(Plan *p, cudaStream_t s)
{
    auto *S = static_cast<SlicedPlan *>(p->sliced);
    if (!S) return;
    void *ptrs[] = {S->col, S->val};
    for (void *q : ptrs)
        if (q) cudaFreeAsync(q, s);
    delete S;
    p->sliced = nullptr;
}

}  // namespace sbb
