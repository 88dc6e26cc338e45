#include "context.h"

#include <cuda_runtime_api.h>

namespace ngap {

uint64_t current_context_id() {
  using Fn = int (*)(void*, unsigned long long*);
  static Fn fn = []() -> Fn {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<Fn>(f);
  }();
  unsigned long long id = 0;
  if (!fn || fn(nullptr, &id) != 0) return 0;  // a null handle asks for the current context
  return (uint64_t)id + 1;
}

}  // namespace ngap
