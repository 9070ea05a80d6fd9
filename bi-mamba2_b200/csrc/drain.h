// Which phases of a ring of mbarriers a kernel that gives up still has to see: load i arrives at barrier i % depth, as its phase
// i / depth, and at most the last one on each barrier can be in flight.  Waiting for any other phase would be wrong: a parity
// wait takes one that has not begun for the one before it.
#pragma once

#ifdef __CUDACC__
#define BISSD_DRAIN __device__ __forceinline__
#else
#define BISSD_DRAIN inline
#endif

namespace bissd {

template <class Wait> BISSD_DRAIN void drain_ring(int issued, int depth, Wait wait) {   // wait(barrier, parity)
#ifdef __CUDACC__
#pragma unroll 1
#endif
    for (int i = issued > depth ? issued - depth : 0; i < issued; ++i) wait(i % depth, (i / depth) & 1);
}

// The same for a tile whose dstate comes in `ns` slabs, two ahead, and whose x rows in `nx` pieces once the last slab but one has
// been read: what had been asked for when a wait ran out at `where`, 1 + the slab, or kStages + the stage that was not begun.
constexpr int kStages = 64;
struct Asked {
    int slabs, pieces;
};
BISSD_DRAIN Asked tile_asked(int where, int ns, int nx) {
    const bool early = where > 0 && where < kStages;
    int slabs = ns, pieces = nx;
    if (early) slabs = where < 2 ? 2 : where;
    if (early) pieces = ns > 1 ? 0 : 2;
    else if (where) pieces = where - kStages < 2 ? 2 : where - kStages;
    return {slabs < ns ? slabs : ns, pieces < nx ? pieces : nx};
}

}  // namespace bissd
