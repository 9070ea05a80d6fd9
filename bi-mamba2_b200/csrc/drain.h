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

}  // namespace bissd
