// What the library keeps between calls and what belongs to a CUDA context: events, pinned memory, memory pools.  A
// context made later on a device (after cudaDeviceReset, or another one beside it) gets its own; what belonged to a
// context that is gone went with it and is not touched again.
#pragma once

#include <new>

#include "xk_common.cuh"

// The current context's id, after making the device's primary context current if the thread has none.
xk_status xk_context_here(unsigned long long* id);

// Making what is kept, and trimming a pool, are no stream operations: a capture that another thread has under way
// must not forbid them, nor end by them.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// One T per context.  Ids are not used again, so a found one is of a live context.  T::drop() gives back what T
// holds, in its context.
template <typename T>
class PerContext {
  struct Node {
    unsigned long long ctx;
    T kept;
    Node* next;
  };
  Node* head = nullptr;

 public:
  T* find(unsigned long long ctx) const {
    for (Node* n = head; n; n = n->next)
      if (n->ctx == ctx) return &n->kept;
    return nullptr;
  }
  T* add(unsigned long long ctx) {  // null without memory
    Node* n = new (std::nothrow) Node{ctx, T{}, head};
    if (n) head = n;
    return n ? &n->kept : nullptr;
  }
  xk_status here(T** out) {
    unsigned long long ctx = 0;
    XK_TRY(xk_context_here(&ctx));
    *out = find(ctx);
    if (!*out) *out = add(ctx);
    return *out ? XK_OK : xk_set_error(XK_ERR_OVERFLOW, "out of host memory");
  }
  ~PerContext() {  // a thread's: of the context that it ends in (others may be gone, and give theirs back themselves)
    unsigned long long ctx = 0;
    const bool have = xk_context_id(&ctx);
    while (Node* n = head) {
      head = n->next;
      if (have && n->ctx == ctx) n->kept.drop();
      delete n;
    }
  }
};
