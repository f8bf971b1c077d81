// spmv_device.cuh — per-row (K1) and per-segment (K2) device code shared by
// the standalone kernels and the batched persistent kernel, so a matrix gets
// bit-identical results whichever way it is run.
#pragma once
#include <climits>

#include "../sbb_internal.h"
#include "common.cuh"
#include "lane_index.cuh"

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
// the L2 prefetch rows of 100 took 42, without the loads ahead in a row 38.  Rows
// of 150 with 32 lanes are no faster: 43.0 (42.5), FP32 storage 37.3 (35.9).
// AHEAD: with the prefetches and the loads ahead in a row.
constexpr unsigned kVectorPrefetch = 256;
template <typename PT, typename ACC, int V, bool AHEAD = true>
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
        if (!AHEAD) return;
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
        unsigned k[U], end[U], reach[U];
        ACC acc[U];
        unsigned most = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int q = u * RPW + g;
            k[u] = (unsigned)__shfl_sync(0xffffffffu, lo, q) + (unsigned)li;
            end[u] = (unsigned)__shfl_sync(0xffffffffu, hi, q);
            reach[u] = lane_reach(k[u], end[u]);
            acc[u].zero();
            most = max(most, reach[u]);
        }
        lo = nlo;
        hi = nhi;
        if (at + 2 * CR < count) load_rows(at + 2 * CR, nlo, nhi);
        int c[U];
        T v[U], xv[U];
        auto load = [&](unsigned off) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                c[u] = ld_stream_if(col + (k[u] + off), off < reach[u]);
                v[u] = ld_stream_if(val + (k[u] + off), off < reach[u]);
            }
        };
        auto gather = [&](unsigned off) {
#pragma unroll
            for (int u = 0; u < U; ++u) xv[u] = gather_x_if(x, c[u], n, off < reach[u], bad);
        };
        if constexpr (!AHEAD) {
#pragma unroll 1
            for (unsigned off = 0; off < most; off += V) {
                load(off);
                gather(off);
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (off < reach[u]) acc[u].mac(v[u], xv[u]);
            }
        } else if constexpr (sizeof(T) == 8) {
            // FP64: an index per row; FP32 storage: one offset for all (the other way
            // round, us: 9 small matrices as a batch 32.8 and 32.0, FP32 rows of 150 38.4
            // and 36.9)
            load(0);
            bool any = most > 0;
            while (any) {
                T vn[U];
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
                    if (k[u] < end[u]) {
                        acc[u].mac(v[u], xv[u]);
                        k[u] = lane_step(k[u], end[u], V);
                    }
                    v[u] = vn[u];
                }
            }
        } else {
            load(0);
#pragma unroll 1
            for (unsigned off = 0; off < most; off += V) {
                T vn[U];
                gather(off);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const bool p = off + V < reach[u];
                    c[u] = ld_stream_if(col + (k[u] + V + off), p);
                    vn[u] = ld_stream_if(val + (k[u] + V + off), p);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (off < reach[u]) acc[u].mac(v[u], xv[u]);
                    v[u] = vn[u];
                }
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

// K2: `count` (at most kMergeGroup) consecutive merge-path segments by one
// warp, the first of them segment w0.  Lane l reads the coordinates of segment
// w0 + l, all at once, and the nnz of the whole group (contiguous) are brought
// into L2 together, so the segments after the first find them there.
template <typename PT, typename ACC, int IPT>
__device__ __forceinline__ void merge_segments(
    int w0, int count, int n, const int *__restrict__ rowptr, const int *__restrict__ col,
    const typename PT::V *__restrict__ val, const typename PT::V *__restrict__ x,
    double *__restrict__ y, double alpha, double beta, const int *__restrict__ tile_row,
    const int *__restrict__ tile_nnz, double *__restrict__ carry_val, unsigned *status,
    typename PT::P *s_p, uint64_t keep, uint64_t streaming)
{
    using V = typename PT::V;
    constexpr int SEG = 32 * IPT;
    const int lane = threadIdx.x & 31;
    int crow = 0, cnnz = 0;
    if (lane <= count) {
        crow = __ldg(tile_row + w0 + lane);
        cnnz = __ldg(tile_nnz + w0 + lane);
    }
    unsigned bad = 0;
    if (count > 1) {
        const int a = __shfl_sync(0xffffffffu, cnnz, 0), b = __shfl_sync(0xffffffffu, cnnz, count);
        if (lane == 0 && b > a && b - a <= SEG * kMergeGroup) {
            prefetch_l2(col + a, 4 * (size_t)(b - a));
            prefetch_l2(val + a, sizeof(V) * (size_t)(b - a));
        }
    }
#pragma unroll 1
    for (int g = 0; g < count; ++g) {
        const int r0 = __shfl_sync(0xffffffffu, crow, g), r1 = __shfl_sync(0xffffffffu, crow, g + 1);
        const int k0 = __shfl_sync(0xffffffffu, cnnz, g), k1 = __shfl_sync(0xffffffffu, cnnz, g + 1);
        const int nrows = r1 - r0, nz = k1 - k0;
        if (nrows < 0 || nz < 0 || nrows + nz > SEG) {  // corrupt coordinates
            if (lane == 0) atomicOr(status, ST_BAD_TILE);
            continue;
        }
        // 1. products to shared memory: every load of the lane in flight
        // together, with the first 32 row ends and their y
        int c[IPT];
        V v[IPT];
#pragma unroll
        for (int j = 0; j < IPT; ++j) {
            const bool p = lane + 32 * j < nz;
            c[j] = ld_stream_if(col + k0 + lane + 32 * j, p);
            v[j] = ld_stream_if(val + k0 + lane + 32 * j, p);
        }
        int end = k0;  // end of row r0 + b + lane, for the 32 rows from b
        if (lane < nrows) end = __ldg(rowptr + r0 + 1 + lane);
        // the ends of further rows go behind the products, where there is room for
        // one of each of the segment's items
        int *s_end = reinterpret_cast<int *>(s_p + nz);
        for (int i = 32 + lane; i < nrows; i += 32) copy_async(s_end + i, rowptr + r0 + 1 + i);
        double yv = 0.0;
        if (beta != 0.0 && lane < nrows) yv = ld_y(y + r0 + lane, streaming);
        V xv[IPT];
#pragma unroll
        for (int j = 0; j < IPT; ++j) {
            const bool p = lane + 32 * j < nz, ok = (unsigned)c[j] < (unsigned)n;
            bad |= p && !ok;
            xv[j] = ld_keep_if(x + c[j], p && ok, keep);
        }
#pragma unroll
        for (int j = 0; j < IPT; ++j)
            if (lane + 32 * j < nz) s_p[lane + 32 * j] = PT::make(v[j], xv[j]);
        if (nrows > 32) copy_async_wait();
        __syncwarp();

        // 2. complete rows r0 .. r1-1: lane per row, long rows by the warp
        int before = 0;  // where row r0 + b starts (it may have started before k0)
        for (int b = 0; b < nrows; b += 32) {
            const int i = b + lane;
            if (b > 0) {
                if (i < nrows) end = s_end[i];
                if (beta != 0.0 && i < nrows) yv = ld_y(y + r0 + i, streaming);
            }
            // a valid row pointer keeps 0 <= lo <= hi <= nz; clamping makes a
            // corrupt one harmless (wrong sums, no out-of-range reads)
            int hi = min(max(end - k0, 0), nz), lo = __shfl_up_sync(0xffffffffu, hi, 1);
            if (lane == 0) lo = before;
            hi = max(hi, lo);
            const bool in = i < nrows, is_long = hi - lo > kLongRow;
            double sum = 0.0;
            if (in && !is_long) {
                ACC acc;
                acc.zero();
#pragma unroll 4
                for (int k = lo; k < hi; ++k) acc.add(s_p[k]);
                sum = acc.get();
            }
            unsigned longs = __ballot_sync(0xffffffffu, in && is_long);
            while (longs) {
                const int src = __ffs(longs) - 1;
                longs &= longs - 1;
                const int llo = __shfl_sync(0xffffffffu, lo, src);
                const int lhi = __shfl_sync(0xffffffffu, hi, src);
                const double t = warp_range_sum<ACC>(s_p, llo, lhi, lane);
                if (lane == src) sum = t;
            }
            if (in) st_y(y + r0 + i, y_update(alpha, sum, beta, yv), streaming);
            before = __shfl_sync(0xffffffffu, hi, min(31, nrows - b - 1));
        }
        // 3. carry: the part of row r1 inside this segment
        const double t = warp_range_sum<ACC>(s_p, before, nz, lane);
        if (lane == 0) carry_val[w0 + g] = t;
        __syncwarp();  // shared memory is reused by the next segment
    }
    if (bad) atomicOr(status, ST_BAD_COL);
}

}  // namespace sbb
