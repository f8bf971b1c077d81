// lane_index.cuh — index arithmetic of lanes that walk a row, for nnz up to
// 2^31 - 1.  Plain C++ besides, so that the host can check the limits.
#pragma once

#if defined(__CUDACC__)
#define SBB_HD __host__ __device__ __forceinline__
#else
#define SBB_HD inline
#endif

namespace sbb {

// How far a lane that starts at nnz `k` of a row may go: it takes k + off for off =
// 0, step, 2 * step, ... while off < lane_reach(k, end).  Rows that are walked
// together share one `off`, which runs to the longest of them and two steps more,
// less than 2^32.  (With an index per row, tested against the row's end, the index of
// a short row wrapped to 0 beside a row of nearly 2^31 nnz, and its walk began again.)
SBB_HD unsigned lane_reach(unsigned k, unsigned end) { return k < end ? end - k : 0u; }

// How many of a row's `len` nnz lane `sub` of `width` takes: sub, sub + width, ...
SBB_HD unsigned lane_share(unsigned len, unsigned sub, unsigned width)
{
    return len > sub ? (len - sub + width - 1u) / width : 0u;
}

}  // namespace sbb
