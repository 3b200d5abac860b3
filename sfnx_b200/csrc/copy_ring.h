// The bookkeeping of a ring of SLOTS shared-memory buffers that one thread fills by asynchronous copies (the TMA unit's):
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
    unsigned n = 0;      // copies asked for
    bool alive = true;   // false after a wait ran out
    FNX_RING_FN unsigned slot() const { return n % SLOTS; }
    // Waits until copy n may be asked for; false: it must not.  empty(slot, parity), full(slot, parity): bounded waits,
    // false when they run out.
    template <class Empty, class Full> FNX_RING_FN bool acquire(Empty empty, Full full) {
        if (alive && n >= SLOTS) alive = empty(slot(), (n / SLOTS - 1) & 1u) && full(slot(), (n / SLOTS - 1) & 1u);
        return alive;
    }
    FNX_RING_FN void asked() { ++n; }
    template <class Full> FNX_RING_FN void drain(Full full) const {
        for (unsigned k = n < SLOTS ? 0 : n - SLOTS; k < n; ++k) full(k % SLOTS, (k / SLOTS) & 1u);
    }
};

}  // namespace fnxk
