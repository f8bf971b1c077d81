// spmv_device.cuh — per-row (K1) and per-segment (K2) device code shared by
// the standalone kernels and the batched persistent kernel, so a matrix gets
// bit-identical results whichever way it is run.
#pragma once
#include <climits>

#include "../sbb_internal.h"
#include "common.cuh"

namespace sbb {

constexpr int kLongRow = 32;  // K2: rows longer than this in a segment are summed by the warp

// The sums of U rows held by a group of V lanes (acc[u] = this lane's part of
// row u): lane li ends with the total of row li / (V / U).  At each step a
// lane keeps half of the rows it still holds and hands the other half to the
// lane o away, so U rows take U - 1 + log2(V / U) exchanges instead of
// U * log2(V); a row's total is formed by the additions of the xor butterfly
// over V lanes, so it has the butterfly's bits.
template <int V, int U> __device__ __forceinline__ double group_row_sums(double (&acc)[U], int li)
{
#pragma unroll
    for (int h = U / 2, o = V / 2; h > 0; h >>= 1, o >>= 1) {
        const bool upper = li & o;
#pragma unroll
        for (int j = 0; j < h; ++j) {
            const double send = upper ? acc[j] : acc[j + h];
            const double keep = upper ? acc[j + h] : acc[j];
            acc[j] = keep + __shfl_xor_sync(0xffffffffu, send, o, V);
        }
    }
    double sum = acc[0];
#pragma unroll
    for (int o = V / U / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o, V);
    return sum;
}

// K1: rows [r0, r0 + count) by one warp, V lanes per row, a chunk of
// vector_chunk(V) rows at a time.  Lane l loads rowptr[r+l], rowptr[r+l+1] and
// y[r+l] of a chunk (coalesced) and ends with row r+l's sum, so y is written
// with one coalesced store; row q of a chunk is reduced by lane group
// q % (32/V), with the U rows of a group in flight together.  Three things run
// ahead: the row pointers by one chunk; the nnz of the next chunk, when it has
// at most kVectorPrefetch of them, into L2; and in a row the next V columns and
// values, loaded while x is gathered for the current ones.  Per row the order
// of the sum is fixed for a given V: lane i of the group adds the products of
// nnz lo+i, lo+i+V, lo+i+2V, ... in that order, then the group's partial sums
// meet in an xor butterfly.  All 32 lanes call this together (full-mask
// shuffles).
//
// What bounds it: the latency of column and x loads in turn, and issue in the
// row ends.  Against loads that wait for the rows before them, branches around
// each load and a butterfly per row (us, FP64, beta = 0.5): 200k rows of 24 in
// a band with 8, 16, 32 lanes 18.6, 18.8, 25.5 (21.2, 21.4, 26.9 before); 100k
// rows of 100 in blocks with 16, 32 lanes 30.9, 30.9 (36.1, 31.4); 100k
// power-law rows of 30 with 16, 32 lanes 64, 44 (81, 54).  Without the bound on
// the L2 prefetch rows of 100 took 42, without the loads ahead in a row 38.
constexpr unsigned kVectorPrefetch = 256;
template <typename PT, typename ACC, int V>
__device__ __forceinline__ void vector_rows(int r0, int count, int n,
                                            const int *__restrict__ rowptr,
                                            const int *__restrict__ col,
                                            const typename PT::V *__restrict__ val,
                                            const typename PT::V *__restrict__ x,
                                            double *__restrict__ y, double alpha, double beta,
                                            uint64_t stream, unsigned &bad)
{
    using T = typename PT::V;
    constexpr int RPW = 32 / V, U = vector_rows_in_flight(V), CR = RPW * U;
    const int lane = threadIdx.x & 31, g = lane / V, li = lane & (V - 1);
    int lo = 0, hi = 0, nlo = 0, nhi = 0;
    // offsets from r0 stay in int
    auto load_rows = [&](int at, int &a, int &b) {
        a = b = 0;
        if (lane < min(CR, count - at)) {
            a = __ldg(rowptr + r0 + at + lane);
            b = __ldg(rowptr + r0 + at + lane + 1);
        }
    };
    auto prefetch = [&](int a, int b) {
        const unsigned first = (unsigned)__shfl_sync(0xffffffffu, a, 0);
        const unsigned end = __reduce_max_sync(0xffffffffu, (unsigned)b);
        if (lane == 0 && end - first - 1u < kVectorPrefetch) {
            prefetch_l2(col + first, 4 * (size_t)(end - first));
            prefetch_l2(val + first, sizeof(T) * (size_t)(end - first));
        }
    };
    load_rows(0, lo, hi);
    if (CR < count) load_rows(CR, nlo, nhi);
    prefetch(lo, hi);
#pragma unroll 1
    for (int at = 0; at < count; at += CR) {
        double yv = 0.0;
        const bool in = lane < min(CR, count - at);
        if (in && beta != 0.0) yv = ld_y(y + r0 + at + lane, stream);
        if (at + CR < count) prefetch(nlo, nhi);
        // nnz indices are unsigned: with nnz up to 2^31 - 1 a lane's index runs
        // to at most nnz - 1 + V (< 2^32), past the int range but never wrapping
        unsigned k[U], end[U];
        ACC acc[U];
        bool any = false;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int q = u * RPW + g;
            k[u] = (unsigned)__shfl_sync(0xffffffffu, lo, q) + (unsigned)li;
            end[u] = (unsigned)__shfl_sync(0xffffffffu, hi, q);
            acc[u].zero();
            any |= k[u] < end[u];
        }
        lo = nlo;
        hi = nhi;
        if (at + 2 * CR < count) load_rows(at + 2 * CR, nlo, nhi);
        int c[U];
        T v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            c[u] = ld_stream_if(col + k[u], k[u] < end[u]);
            v[u] = ld_stream_if(val + k[u], k[u] < end[u]);
        }
        while (any) {
            T xv[U], vn[U];
#pragma unroll
            for (int u = 0; u < U; ++u) xv[u] = gather_x_if(x, c[u], n, k[u] < end[u], bad);
            any = false;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const unsigned kn = k[u] + V;
                any |= kn < end[u];
                c[u] = ld_stream_if(col + kn, kn < end[u]);
                vn[u] = ld_stream_if(val + kn, kn < end[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (k[u] < end[u]) acc[u].mac(v[u], xv[u]);
                v[u] = vn[u];
                k[u] += V;
            }
        }
        double part[U];
#pragma unroll
        for (int u = 0; u < U; ++u) part[u] = acc[u].get();
        const double sum = group_row_sums<V, U>(part, li);
        // row q = u*RPW + g lands in lane q
        const double out =
            __shfl_sync(0xffffffffu, sum, (lane % RPW) * V + (lane / RPW & (U - 1)) * (V / U));
        if (in) st_y(y + r0 + at + lane, y_update(alpha, out, beta, yv), stream);
    }
}

// Carry fix-up arithmetic shared by the standalone fix-up (k_fixup.cu) and
// the batch fix-up (k_batch.cu): a single carry is added as fma(alpha, c, y[r]); a
// run of at most kWarpRunMax carries is summed by one warp (lane i: slots i,
// i + 32, ... in order, then an xor butterfly); a longer run by kFixupThreads
// threads (thread i: slots i, i + kFixupThreads, ... in order) and then a
// shared-memory tree.  Which of the two a run gets depends only on its
// length, so both fix-ups sum every run in the same order.
constexpr int kFixupThreads = 256;
__device__ __forceinline__ void fixup_single(double *y, int r, double alpha, double c)
{
    y[r] = __fma_rn(alpha, c, y[r]);
}
__device__ __forceinline__ double fixup_partial(const double *cval, int first, int len, int i)
{
    double acc = 0.0;
    for (; i < len; i += kFixupThreads) acc += cval[first + i];
    return acc;
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum of a run of at most kWarpRunMax carries by the calling warp (every lane
// gets it).
__device__ __forceinline__ double fixup_run_warp(const double *cval, int first, int len)
{
    double acc = 0.0;
    for (int i = threadIdx.x & 31; i < len; i += 32) acc += cval[first + i];
    return warp_sum(acc);
}

// Sum of the products s_p[lo..hi) by the whole warp (fixed order: lane-strided
// partial sums, then an xor butterfly).
template <typename ACC, typename P>
__device__ __forceinline__ double warp_range_sum(const P *s_p, int lo, int hi, int lane)
{
    ACC acc;
    acc.zero();
    for (int i = lo + lane; i < hi; i += 32) acc.add(s_p[i]);
    return warp_sum(acc.get());
}

template <typename PT, typename ACC, int IPT>
__device__ __forceinline__ void merge_segment(
    int w, int n, const int *__restrict__ rowptr, const int *__restrict__ col,
    const typename PT::V *__restrict__ val, const typename PT::V *__restrict__ x,
    double *__restrict__ y, double alpha, double beta, const int *__restrict__ tile_row,
    const int *__restrict__ tile_nnz, double *__restrict__ carry_val, unsigned *status,
    typename PT::P *s_p, int *s_re, uint64_t keep, uint64_t streaming)
{
    using P = typename PT::P;
    using V = typename PT::V;
    constexpr int SEG = 32 * IPT;
    const int lane = threadIdx.x & 31;
    const int r0 = __ldg(tile_row + w), r1 = __ldg(tile_row + w + 1);
    const int k0 = __ldg(tile_nnz + w), k1 = __ldg(tile_nnz + w + 1);
    const int nrows = r1 - r0, nz = k1 - k0;
    if (nrows < 0 || nz < 0 || nrows + nz > SEG) {  // corrupt coordinates
        if (lane == 0) atomicOr(status, ST_BAD_TILE);
        return;
    }
    unsigned bad = 0;
    // y of the first 32 rows, early: the beta*y read then is off the tail
    double ypre = 0.0;
    if (beta != 0.0 && lane < nrows) ypre = ld_y(y + r0 + lane, streaming);

    // 1. row ends and products (every load of the lane in flight together)
    int cc[IPT];
    V vv[IPT];
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
        const int i = lane + 32 * j;
        if (i < nz) {
            cc[j] = ld_stream(col + k0 + i);
            vv[j] = ld_stream(val + k0 + i);
        }
    }
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
        const int i = lane + 32 * j;
        if (i < nrows) s_re[i] = __ldg(rowptr + r0 + 1 + i);
    }
    V xv[IPT];
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
        const int i = lane + 32 * j;
        if (i < nz) {
            if ((unsigned)cc[j] < (unsigned)n) {
                xv[j] = ld_keep(x + cc[j], keep);
            } else {
                bad = 1u;
                xv[j] = V(0);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
        const int i = lane + 32 * j;
        if (i < nz) s_p[i] = PT::make(vv[j], xv[j]);
    }
    if (bad) atomicOr(status, ST_BAD_COL);
    __syncwarp();

    // 2. complete rows r0 .. r1-1: lane per row, long rows by the warp
    for (int b = 0; b < nrows; b += 32) {
        const int i = b + lane;
        int lo = 0, hi = 0;
        if (i < nrows) {
            lo = i == 0 ? 0 : s_re[i - 1] - k0;  // row r0 may have started before k0
            hi = s_re[i] - k0;
            // a valid row pointer keeps 0 <= lo <= hi <= nz; clamping makes a
            // corrupt one harmless (wrong sums, no out-of-range reads)
            lo = min(max(lo, 0), nz);
            hi = min(max(hi, lo), nz);
        }
        const bool is_long = hi - lo > kLongRow;
        if (i < nrows && !is_long) {
            ACC acc;
            acc.zero();
            for (int k = lo; k < hi; ++k) acc.add(s_p[k]);
            double *yp = y + r0 + i;
            const double v = y_update(alpha, acc.get(), beta,
                                      beta == 0.0 ? 0.0 : (b == 0 ? ypre : ld_y(yp, streaming)));
            st_y(yp, v, streaming);
        }
        unsigned longs = __ballot_sync(0xffffffffu, i < nrows && is_long);
        while (longs) {
            const int src = __ffs(longs) - 1;
            longs &= longs - 1;
            const int llo = __shfl_sync(0xffffffffu, lo, src);
            const int lhi = __shfl_sync(0xffffffffu, hi, src);
            const double s = warp_range_sum<ACC>(s_p, llo, lhi, lane);
            if (lane == src) {
                double *yp = y + r0 + i;
                const double v = y_update(alpha, s, beta,
                                          beta == 0.0 ? 0.0 : (b == 0 ? ypre : ld_y(yp, streaming)));
                st_y(yp, v, streaming);
            }
        }
    }
    // 3. carry: the part of row r1 inside this segment
    const int clo = nrows > 0 ? min(max(s_re[nrows - 1] - k0, 0), nz) : 0;
    const double c = warp_range_sum<ACC>(s_p, clo, nz, lane);
    if (lane == 0) carry_val[w] = c;
    __syncwarp();  // shared memory is reused by this warp's next segment
}


}  // namespace sbb
