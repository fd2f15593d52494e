// The books of a producer that fills a ring of stages in two steps, of which the second may still be missing
// when the kernel ends: a running tile's first copy (`issued` tiles) and, for the next iteration's first tiles only
// once that iteration runs, its windows (`windowed` tiles).  A stage's barrier expects the bytes of both, so a
// kernel that ends has to issue the windows that are owed, of the same tiles the barrier was armed for, and wait
// for every copy in flight before its shared memory is released.  No CUDA in here: tests run it on the host.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define RG_HD __host__ __device__ __forceinline__
#else
#define RG_HD inline
#endif

namespace rg {

struct RingBooks {
    int64_t issued = 0, windowed = 0;
    int64_t ahead_base = 0;  // the running number of the first tile issued ahead of its iteration,
    bool ahead_back = false; // and the direction in which that iteration walks

    // the next tiles are issued ahead of an iteration that starts at running tile `base`
    RG_HD void ahead(int64_t base, bool back)
    {
        ahead_base = base;
        ahead_back = back;
    }
    // at the kernel's end: windows(running tile, tile of its iteration, direction) for each tile that is owed them,
    // then wait(running tile) for the latest tile of every stage, consumed or not
    template <class Windows, class Wait>
    RG_HD void drain(int stages, Windows windows, Wait wait)
    {
        for (int64_t c = windowed; c < issued; ++c) windows(c, (int)(c - ahead_base), ahead_back);
        windowed = issued;
        for (int64_t c = issued > stages ? issued - stages : 0; c < issued; ++c) wait(c);
    }
};

}  // namespace rg
