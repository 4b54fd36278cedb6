// Which slot of a warp's ring of copies comes next, and what becomes of the ring when a wait runs out. The copies and the waits are
// the caller's (gemm_stream.cuh gives it tensor-map copies and mbarriers), so the order of both is tested with the host compiler.
//
// A slot is filled again only after its wait came back true, so a barrier is never armed twice in one phase; after a wait that ran
// out nothing is filled any more, and every copy still in flight is waited for once before the warp leaves its shared memory.
#pragma once

#ifdef __CUDACC__
#define B200I_RING_FN __host__ __device__ __forceinline__
#else
#define B200I_RING_FN inline
#endif

namespace b200i {

struct StreamRing {
    int stages;
    int head = 0;       // the slot that the next copy goes to: slot itself while the ring is full
    int slot = 0;       // the slot that is read next
    unsigned phase = 0; // of its barrier

    // fill(slot) asks for the next copy and says whether there was one left to ask for.
    template <class Fill>
    B200I_RING_FN void refill(Fill fill) {
        if (fill(head) && ++head == stages) head = 0;
    }
    template <class Fill>
    B200I_RING_FN void start(Fill fill) {
        for (int s = 0; s < stages; s++) refill(fill);
    }
    // The slot has been read: the next copy may go there.
    template <class Fill>
    B200I_RING_FN void release(Fill fill) {
        refill(fill);
        step();
    }
    // A wait for `slot` ran out: the copies in flight are that one (it is waited for once more) and those up to head.
    template <class Wait>
    B200I_RING_FN void drain(Wait wait) {
        do {
            wait(slot, phase);
            step();
        } while (slot != head);
    }
    B200I_RING_FN void step() {
        if (++slot == stages) {
            slot = 0;
            phase ^= 1u;
        }
    }
};

} // namespace b200i
