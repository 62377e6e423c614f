// alloc.h -- device allocations of the solver and the dense drivers, and the
// list in which finished dense calls leave their buffers for the next one.
#ifndef MR3_ALLOC_H
#define MR3_ALLOC_H

#include <cuda_runtime_api.h>
#include <stddef.h>

// Defined with the dense drivers (mr3_b200.h); weak, so that the solver links
// without them.
extern "C" __attribute__((weak)) int mr3_dense_release(void);

// cudaMalloc; where it fails for lack of memory, the dense drivers' idle
// buffers are given back first and it is tried again.
static inline cudaError_t mr3__alloc(void **p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation && mr3_dense_release && mr3_dense_release() > 0) {
    (void)cudaGetLastError();
    e = cudaMalloc(p, bytes);
  }
  return e;
}

// At most N idle objects, each of a device.  The caller holds a lock.
template <typename T, int N>
struct KeptList {
  T *at[N] = {};

  // An idle object of this device, or null; it leaves the list.
  T *take(int device) {
    for (int k = 0; k < N; k++)
      if (at[k] && at[k]->device == device) return remove(k);
    return nullptr;
  }
  // Any idle object, or null.
  T *take_any() {
    for (int k = 0; k < N; k++)
      if (at[k]) return remove(k);
    return nullptr;
  }
  // Puts x into the list.  Returns the object to free for it: null, or x
  // itself, or, where the list is full and another device holds more of it
  // than x's, one of that device.
  T *give(T *x) {
    int most = -1, mine = 0;
    for (int k = 0; k < N; k++) {
      if (!at[k]) { at[k] = x; return nullptr; }
      mine += at[k]->device == x->device;
      if (most < 0 || held(at[k]->device) > held(at[most]->device)) most = k;
    }
    if (held(at[most]->device) <= mine) return x;
    T *out = at[most];
    at[most] = x;
    return out;
  }

 private:
  T *remove(int k) {
    T *x = at[k];
    at[k] = nullptr;
    return x;
  }
  int held(int device) const {
    int c = 0;
    for (int k = 0; k < N; k++) c += at[k] && at[k]->device == device;
    return c;
  }
};

#endif
