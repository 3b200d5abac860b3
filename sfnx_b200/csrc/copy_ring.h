// The bookkeeping of a ring of SLOTS shared-memory buffers that one thread (or the lanes of a warp together) fills by asynchronous copies:
// copy k goes into slot k % SLOTS and completes phase k / SLOTS of the slot's `full` barrier; its readers complete phase
// k / SLOTS of the slot's `empty` barrier when they are done with it.  Plain C++, so that a test on the CPU can run it.
//
// Waits are bounded, and a block must not end while a copy into its memory is under way, also after a wait ran out.  So a
// slot's copy is asked for only when the one before it has landed (whatever the readers say) and been read, nothing is
// asked for once a wait ran out, and drain() waits for the slots' last copies: with no more than one copy of a slot under
// way, a wait by the phase's parity cannot take an older phase for it.
#pragma once

#ifdef __CUDACC__
#define FNX_RING_FN __host__ __device__ __forceinline__
#else
#define FNX_RING_FN inline
#endif

namespace fnxk {

template <int SLOTS> struct CopyRing {
    unsigned slot = 0, round = 0;   // the next copy's; copies asked for: round SLOTS + slot
    bool alive = true;              // false after a wait ran out
    // Waits until the next copy may be asked for; false: it must not.  empty(slot, parity), full(slot, parity): bounded
    // waits, false when they run out.  The copy before has landed by the time it has been read, so it is waited for first
    // and costs nothing; asked for after the readers it was 1 % of a dense kernel's time.
    template <class Empty, class Full> FNX_RING_FN bool acquire(Empty empty, Full full) {
        if (alive && round) alive = full(slot, (round - 1) & 1u) && empty(slot, (round - 1) & 1u);
        return alive;
    }
    FNX_RING_FN void asked() {
        if (++slot == SLOTS) slot = 0, ++round;
    }
    template <class Full> FNX_RING_FN void drain(Full full) const {
        for (unsigned s = 0; s < SLOTS; ++s)
            if (s < slot) full(s, round & 1u);
            else if (round) full(s, (round - 1) & 1u);
    }
};

}  // namespace fnxk
