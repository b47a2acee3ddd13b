// Scratch of the SpMV calls on one handle or plan.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <memory>

namespace mfp {

// A handle or plan may be used by several streams and threads at once and in
// captured graphs, so a call's scratch must not be another running call's.  A
// call takes a block here and gives it back when its launches are enqueued:
//   - a block belongs to the stream that used it first: the calls of one
//     stream follow each other on the GPU.  The first block is allocated with
//     the handle, one more for each further stream (16 in all, then one per
//     call, freed in stream order);
//   - a captured call takes a block that its graph keeps until the graph and its
//     executable copies are destroyed (a CUDA user object; nothing is allocated
//     in the graph).
// The first `zero` bytes of a block are zero when it is handed out for the first
// time; calls leave them zero.  Blocks are freed with the owner.
class call_blocks {
 public:
  call_blocks();
  ~call_blocks();
  call_blocks(const call_blocks &) = delete;
  call_blocks &operator=(const call_blocks &) = delete;
  // Allocates the first block on the current device; adds its size to *acct.
  cudaError_t init(size_t bytes, size_t zero, size_t *acct);

  struct state;

 private:
  friend class call_scratch;
  std::shared_ptr<state> st_;  // NULL before init
};

// The scratch of one call on `stream`, held while the call enqueues its
// launches.  ptr() is NULL when there is no memory for it.
class call_scratch {
 public:
  call_scratch(const call_blocks &blocks, cudaStream_t stream);
  ~call_scratch();
  call_scratch(const call_scratch &) = delete;
  call_scratch &operator=(const call_scratch &) = delete;
  void *ptr() const { return p_; }

 private:
  const std::shared_ptr<call_blocks::state> &st_;
  cudaStream_t stream_;
  void *p_ = nullptr;
  bool once_ = false;  // allocated for this call alone
};

}  // namespace mfp
