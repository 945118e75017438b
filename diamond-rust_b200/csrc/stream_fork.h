// Streams that a call has forked work to.
#pragma once
#include <cuda_runtime.h>

#include <vector>

namespace drg {

// Between a fork and its join a call's other streams read buffers that the
// call frees in the order of its main stream.  A call that fails in between
// unwinds through this, which waits for them; joined() once the main stream
// waits for all of them.  Declared after the buffers, so that it goes first.
class ForkGuard {
 public:
  ForkGuard() = default;
  ForkGuard(const ForkGuard&) = delete;
  ForkGuard& operator=(const ForkGuard&) = delete;
  ~ForkGuard() {
    for (cudaStream_t s : open_) cudaStreamSynchronize(s);
  }
  void add(cudaStream_t s) { open_.push_back(s); }  // before the first work on s
  void joined() { open_.clear(); }

 private:
  std::vector<cudaStream_t> open_;
};

}  // namespace drg
