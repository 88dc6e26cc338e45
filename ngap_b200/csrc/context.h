// The calling thread's current CUDA context, for what is kept from one call
// to the next: a device address is only good in the context it was made in.
#pragma once

#include <cstdint>

namespace ngap {

// Identity of the current context (cuCtxGetId, reached through the runtime's
// entry-point lookup so that the library does not link the driver library):
// never the same for two contexts of a process, not even where a new one (after
// cudaDeviceReset, say) gets the handle of an old one. 0: none is current, or
// it cannot be read.
uint64_t current_context_id();

}  // namespace ngap
