// The word that counts bound-and-split's unfinished work: a warp that gives
// ranges away reserves the bundle's slot and adds the bundle's unit in one
// update, so the slot's number exists only once the unit is counted.  The
// bundle is written to the slot and its receiver reads it there, so the
// receiver's own update, which takes the unit off, comes after: no order
// between different addresses is needed, and no fence.  (With the slot and the
// unit in two words, relaxed as they are, the receiver could take the unit off
// before it was added, and a count that passes zero ends the frame early.)
// Plain C++, so that the tests run it on the host.
#pragma once

#ifdef __CUDACC__
#define MP_HANDOVER_FN __host__ __device__ __forceinline__
#else
#define MP_HANDOVER_FN inline
#endif

namespace mp {

// Low half: units of work (root ranges, published bundles) whose split trees
// are not finished.  High half: bundle slots reserved so far.
constexpr unsigned long long kUnitMask = 0xffffffffull;

MP_HANDOVER_FN unsigned long long handover_start(unsigned long long roots) { return roots; }
// What a giver adds; the value before names its slot.
MP_HANDOVER_FN unsigned long long handover_give() { return (1ull << 32) + 1; }
MP_HANDOVER_FN unsigned long long handover_slot(unsigned long long before) { return before >> 32; }
// What a warp adds when `units` of its own are finished (also a giver whose
// slot does not exist: it keeps its pairs, and still holds a unit of its own).
MP_HANDOVER_FN unsigned long long handover_finish(unsigned units) { return 0ull - units; }
// Whether that was the last work, from the value before.
MP_HANDOVER_FN bool handover_ended(unsigned long long before, unsigned units) {
    return ((before + handover_finish(units)) & kUnitMask) == 0;
}

}  // namespace mp
