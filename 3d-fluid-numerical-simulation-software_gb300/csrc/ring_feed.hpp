// The groups of a ring of asynchronous copies, asked for in order by one thread: group g goes into stage
// g % STAGES and completes phase g / STAGES of that stage's barrier. The thread asks for a group once the consumers
// have said that they are done with the group before it in the same stage, and they say so only of a group that
// they have seen land: a barrier armed twice in a phase would lose count of its arrivals, and two copies would write
// the same bytes. After a wait that ran out nothing more is said or asked for, and drain() waits for exactly the
// groups that were asked for, so that no copy is in flight when the block's shared memory goes.
#pragma once

#ifdef __CUDACC__
#define GBT_HD __host__ __device__ __forceinline__
#else
#define GBT_HD inline
#endif

namespace gbt {

template <int STAGES>
struct RingFeed {
    int groups, asked = 0;
    // ok: no wait of the calling thread has run out; ask(group, stage) arms the barrier and starts the copies
    template <typename Ask>
    GBT_HD void next(bool ok, Ask ask)
    {
        if (!ok || asked >= groups) return;
        ask(asked, asked % STAGES);
        asked++;
    }
    template <typename Wait>
    GBT_HD void drain(Wait wait) const
    {
        for (int g = asked < STAGES ? 0 : asked - STAGES; g < asked; g++) wait(g % STAGES, (unsigned)(g / STAGES) & 1u);
    }
};

}  // namespace gbt
