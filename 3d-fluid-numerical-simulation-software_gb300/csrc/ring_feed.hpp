// The groups of a ring of asynchronous copies, asked for in order by one thread: group g goes into stage
// g % STAGES and completes phase g / STAGES of that stage's barrier. A barrier is armed for a group only once the
// group before it in the same stage has landed, also where the consumers gave up waiting and run ahead of the
// copies: armed twice in a phase, its count of arrivals would underflow and two copies would write the same
// bytes. After a wait that ran out nothing more is asked for, and drain() waits for exactly the groups that were,
// so that no copy is in flight when the block's shared memory goes.
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
    // wait(stage, parity): false once a wait has run out; ask(group, stage) arms the barrier and starts the copies
    template <typename Wait, typename Ask>
    GBT_HD void next(bool ok, Wait wait, Ask ask)
    {
        if (!ok || asked >= groups) return;
        const int stage = asked % STAGES;
        if (asked >= STAGES && !wait(stage, (unsigned)(asked / STAGES - 1) & 1u)) return;
        ask(asked++, stage);
    }
    template <typename Wait>
    GBT_HD void drain(Wait wait) const
    {
        for (int g = asked < STAGES ? 0 : asked - STAGES; g < asked; g++) wait(g % STAGES, (unsigned)(g / STAGES) & 1u);
    }
};

}  // namespace gbt
