// Bookkeeping of a ring of shared-memory slots that asynchronous copies fill: copy j goes to slot j % slots and completes that slot's
// phase j / slots; a slot is armed again only after its last copy was waited for.
#pragma once
#include "layout.cuh"

namespace juno {

// The copies [ring_open, issued) may still be in flight when the first `used` of them have been waited for: no two share a slot.  A kernel
// that gave up a wait stops arming and waits for these before the memory is used for anything else or given back.
JHD int ring_open(int issued, int used, int slots) { return used > issued - slots ? used : issued - slots; }
JHD unsigned ring_parity(int j, int slots) { return (unsigned)(j / slots) & 1u; }

}  // namespace juno
