// The order of work in a ring of bulk copies through shared memory: n pieces, each loaded into stage (piece % kStages), waited for, stored
// from there.  Apart from the copies themselves (Ops) so that it can be followed on the host; plain C++.
//   load(i)      starts the load of piece i                  wait(i)     has it landed? false: the bounded wait ran out
//   store(i)     starts the store of piece i                 settle(i)   gives a load in flight a bounded chance to land
//   stores_read  the stores before the last one have read    finish()    every store has landed
//                their stages
#pragma once

#ifdef __CUDACC__
#define GE2_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define GE2_HOST_DEVICE inline
#endif

namespace ge2 {

// false: a load did not land in time.  Loads that are still on their way into the ring then are waited for before the caller may give the
// shared memory back, and so are the stores.
template <int kStages, typename Ops>
GE2_HOST_DEVICE bool copy_ring(int n, Ops& ops) {
    int issued = 0;
    for (; issued < n && issued < kStages - 1; issued++) ops.load(issued);
    int i = 0;
    for (; i < n; i++) {
        if (!ops.wait(i)) break;
        ops.store(i);
        if (issued < n) {
            ops.stores_read();  // the store before this one has read its stage
            ops.load(issued++);
        }
    }
    const bool ok = i == n;
    for (; i < issued; i++) ops.settle(i);
    ops.finish();
    return ok;
}

}  // namespace ge2
