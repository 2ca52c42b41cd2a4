// Bounded waits whose outcome a whole warp acts on. A wait can run out on some lanes of a warp and be met on the others, at
// the moment of its limit; what the warp then does together (votes, shuffles, loads of tensor memory) needs all
// lanes on one path.
#pragma once

#ifndef GBT_HD
#ifdef __CUDACC__
#define GBT_HD __host__ __device__ __forceinline__
#else
#define GBT_HD inline
#endif
#endif

namespace gbt {

// Polls until no lane of the warp lacks anything (late()), asking for it again in between (ask()), `limit` times at most:
// then ok is false on every lane. A lane whose own wait has run out before (ok false) waits for nothing more, but votes
// on with the others (any: whether some lane's vote is true).
template <typename Any, typename Late, typename Ask>
GBT_HD void poll_together(bool &ok, unsigned limit, Any any, Late late, Ask ask)
{
    for (unsigned polls = 0; any(ok && late()); polls++) {
        if (polls > limit) { ok = false; return; }
        if (ok) ask();
    }
}

}  // namespace gbt
