// The walk of a lane over rows, at the limits of nnz (2^31 - 1), as the vector
// kernel and the row slices do it (lane_index.cuh), on the host.
#include <cstdio>
#include <initializer_list>

#include "lane_index.cuh"

using sbb::lane_reach;
using sbb::lane_share;
using sbb::lane_step;

static int failures = 0;
static void check(bool ok, const char *what, unsigned a, unsigned b)
{
    if (ok) return;
    failures++;
    std::printf("failed: %s (%u, %u)\n", what, a, b);
}

int main()
{
    const unsigned last = 0x7fffffffu;  // the largest nnz
    // A row that is empty (or has one nnz) and starts behind one of `len` nnz, the
    // two walked together by `v` lanes: first and last steps of the walk.
    for (unsigned v = 2; v <= 32; v *= 2)
        for (unsigned len : {last, last - 1, last - 40, 1u << 30})
            for (unsigned li = 0; li < v; li++)
                for (unsigned own = 0; own <= 1; own++) {
                    const unsigned reach = lane_reach(last - own + li, last);
                    const unsigned most = lane_reach(li, len);
                    check(reach == (own && li == 0), "nnz of the short row", reach, li);
                    check(most == len - li, "nnz of the long row", most, li);
                    unsigned long long off = (most - 1) / v * (unsigned long long)v;
                    check(off < most && off + v >= most, "last step", most, v);
                    // the short row's own index, any number of steps on and one ahead
                    unsigned k = last - own + li, taken = 0;
                    for (int i = 0; i < 1000; i++) {
                        taken += k < last;
                        check(k + v > k, "index wraps", k, v);
                        k = lane_step(k, last, v);
                    }
                    check(taken == (own && li == 0) && lane_step(k, last, v) == k,
                          "short row by index", taken, li);
                    for (int i = 0; i < 3; i++, off += v)  // it, and two more loaded ahead
                        check(off <= 0xffffffffull && (unsigned)off >= reach, "walks again", li, v);
                }
    // Shares of the row slices: together the whole row, evenly.
    for (unsigned w = 1; w <= 16; w *= 2)
        for (unsigned len : {0u, 1u, w - 1, w, w + 1, 1000u, last - 16, last - 1, last}) {
            unsigned long long sum = 0;
            for (unsigned sub = 0; sub < w; sub++) {
                const unsigned n = lane_share(len, sub, w);
                check(n <= len / w + 1 && n >= len / w, "share", len, sub);
                sum += n;
            }
            check(sum == len, "shares of a row", len, w);
        }
    if (!failures) std::printf("ok\n");
    return failures != 0;
}
