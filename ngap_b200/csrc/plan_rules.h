// Host rules of a match that need no GPU to be decided.
#pragma once

#include <cstdint>

namespace ngap {

// What the runtime says about an input address (cudaPointerGetAttributes).
struct InputMemory {
  bool device = false;  // plain device memory (not managed, not host memory)
  int owner = -1;       // the GPU that holds it
};

// Whether an input of a length and an address that the kernels' 16-byte reads and
// bulk copies can cover (multiples of 16) may be read where it is. `memory` is
// asked only for such an input: it must be memory of the engine's own GPU. What
// another GPU holds, or the host, is copied, which works without peer
// access; a kernel that read it in place would fault.
template <class Memory>
bool reads_in_place(const void* input, bool on_device, uint64_t bytes, int engine_device, Memory memory) {
  if (!on_device || bytes == 0 || bytes % 16 != 0 || reinterpret_cast<uintptr_t>(input) % 16 != 0) return false;
  const InputMemory m = memory(input);
  return m.device && m.owner == engine_device;
}

}  // namespace ngap
