// Device memory that a host thread keeps from one call to the next.
//
// A call that has waited for its stream is done with its scratch, so the thread
// may use the same block for its next call instead of allocating and freeing
// one, which waits for the whole device. A block belongs to the context it was
// allocated in: it is used again, and freed, only while that context is current.
// Blocks of other contexts are left alone; one whose context has been
// destroyed (cudaDeviceReset, cuCtxDestroy) went with it, and its address
// may be somebody else's by now. Api: uint64_t context() (0: none is current),
// void init() (makes the device's context current), int device(), void
// set_device(int), int alloc(void**, size_t) (0 = success), void free(void*).
#pragma once

#include <cstddef>
#include <cstdint>

namespace ngap {

template <class Api, int kContexts = 4>
class KeptBlocks {
 public:
  explicit KeptBlocks(Api api = Api()) : api_(api) {}
  KeptBlocks(const KeptBlocks&) = delete;
  KeptBlocks& operator=(const KeptBlocks&) = delete;

  // At least `bytes` of the current context in *out, kept when they are at most
  // `keep` and the context is one of the first kContexts the thread used;
  // otherwise *mine is true and the caller frees *out. Returns Api's status.
  int reserve(size_t bytes, size_t keep, void** out, bool* mine) {
    *out = nullptr;
    *mine = true;
    uint64_t now = api_.context();
    if (now == 0) {
      api_.init();
      now = api_.context();
    }
    Block* b = nullptr;
    if (bytes <= keep && now != 0) {
      for (Block& x : blocks_)
        if (x.context == now) b = &x;
      for (Block& x : blocks_)
        if (!b && x.context == 0) b = &x;
    }
    if (!b) return api_.alloc(out, bytes);
    if (b->cap < bytes) {
      if (b->ptr) api_.free(b->ptr);
      *b = Block();
      void* p = nullptr;
      const int rc = api_.alloc(&p, bytes);
      if (rc != 0) return rc;
      *b = Block{p, bytes, api_.device(), now};
    }
    *out = b->ptr;
    *mine = false;
    return 0;
  }

  // Frees the blocks whose context lives on (the thread ends): the current
  // one's, and those of other devices whose primary context is still theirs.
  ~KeptBlocks() {
    const uint64_t now = api_.context();
    if (now == 0) return;
    const int dev = api_.device();
    for (Block& b : blocks_) {
      if (!b.ptr) continue;
      if (b.context == now) {
        api_.free(b.ptr);
      } else if (b.device != dev) {
        api_.set_device(b.device);
        if (api_.context() == b.context) api_.free(b.ptr);
        api_.set_device(dev);
      }
    }
  }

 private:
  struct Block {
    void* ptr = nullptr;
    size_t cap = 0;
    int device = -1;
    uint64_t context = 0;
  };
  Api api_;
  Block blocks_[kContexts];
};

}  // namespace ngap
