// lane_index.cuh — index arithmetic of lanes that walk a row, for nnz up to
// 2^31 - 1.  Plain C++ besides, so that the host can check the limits.
#pragma once

#if defined(__CUDACC__)
#define SBB_HD __host__ __device__ __forceinline__
#else
#define SBB_HD inline
#endif

namespace sbb {

// A lane walks rows of different lengths together, `step` nnz at a time, until the
// longest ends.  Either each row has its index, which moves on only while it is
// in the row (lane_step), so it stays below end + step ...
SBB_HD unsigned lane_step(unsigned k, unsigned end, unsigned step) { return k < end ? k + step : k; }

// ... or all rows share one offset: the lane takes nnz k + off of a row that it
// starts at nnz k, for off = 0, step, 2 * step, ... while off < lane_reach(k, end);
// the offset runs to the longest row and two steps more, less than 2^32.  (With an
// index that went on behind the row's end, it wrapped to 0 beside a row of nearly
// 2^31 nnz, and the short row's walk began again.)
SBB_HD unsigned lane_reach(unsigned k, unsigned end) { return k < end ? end - k : 0u; }

// How many of a row's `len` nnz lane `sub` of `width` takes: sub, sub + width, ...
SBB_HD unsigned lane_share(unsigned len, unsigned sub, unsigned width)
{
    return len > sub ? (len - sub + width - 1u) / width : 0u;
}

}  // namespace sbb
