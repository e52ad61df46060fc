// Scratch memory of one call, allocated and freed in stream order, so calls on
// several streams and threads never share it.  It comes from one pool per device
// that exists while the device has handles: omb_create / omb_destroy hold it,
// the last handle's end returns its memory; what it keeps between calls is
// bounded by kScratchKept.  A call that is being captured into a CUDA graph gets
// none: the pair would become memory nodes, and a graph with those can be
// neither cloned nor instantiated twice.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace omb {

constexpr size_t kScratchKept = 512u << 20;

void scratch_hold(int device);
void scratch_drop(int device);

struct StreamScratch {
    void *p = nullptr;
    // p is NULL when there is no pool or memory, the stream is capturing or bytes is 0: the caller does without
    StreamScratch(size_t bytes, cudaStream_t st);
    ~StreamScratch();
    StreamScratch(const StreamScratch &) = delete;
    StreamScratch &operator=(const StreamScratch &) = delete;

  private:
    cudaStream_t stream;
};

}  // namespace omb
