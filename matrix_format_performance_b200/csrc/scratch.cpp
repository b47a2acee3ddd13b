#include "scratch.h"

#include <mutex>
#include <new>
#include <vector>

namespace mfp {

namespace {
constexpr size_t kMaxStreams = 16;

// Calls that are refused to every thread while one captures in global mode
// (cudaMalloc) are made as this thread's own business.
struct relaxed_capture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  relaxed_capture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~relaxed_capture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};
}  // namespace

// No CUDA call is made with `mu` held: give_back() may come from a thread of the
// driver's.
struct call_blocks::state {
  struct block {
    void *p;
    unsigned long long owner;  // stream id; captures: capture id
    cudaStream_t stream;       // captures: the capturing stream
    bool owned;                // has an owner; captures: a graph holds it
    bool busy;                 // a call is enqueueing its launches
  };
  std::mutex mu;
  size_t bytes = 0, zero = 0;
  std::vector<block> streams, captures;

  // The call has enqueued its launches; `unowned`: no graph holds the block either.
  void done(void *p, bool unowned = false) {
    std::lock_guard<std::mutex> g(mu);
    for (auto *v : {&streams, &captures})
      for (block &b : *v)
        if (b.p == p) {
          b.busy = false;
          if (unowned) b.owned = false;
        }
  }

  // A graph's reference to a block; the graph's last owner gives it back.
  struct hold {
    std::shared_ptr<state> st;
    void *p;
  };
  static void CUDART_CB give_back(void *arg) {
    hold *h = static_cast<hold *>(arg);
    {
      std::lock_guard<std::mutex> g(h->st->mu);
      for (block &b : h->st->captures)
        if (b.p == h->p) b.owned = false;
    }
    delete h;
  }

  // A block for a capture, its zeroes in place before any graph can run.
  void *allocate_now() {
    const relaxed_capture relaxed;
    void *p = nullptr;
    cudaStream_t s = nullptr;
    bool ok = cudaMalloc(&p, bytes) == cudaSuccess;
    if (ok && zero) {
      ok = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess &&
           cudaMemsetAsync(p, 0, zero, s) == cudaSuccess && cudaStreamSynchronize(s) == cudaSuccess;
      if (s) cudaStreamDestroy(s);
    }
    if (ok) return p;
    cudaGetLastError();
    cudaFree(p);
    return nullptr;
  }

  static void *take_captured(const std::shared_ptr<state> &st, cudaGraph_t graph, unsigned long long id,
                             cudaStream_t s) {
    void *p = nullptr;
    {
      std::lock_guard<std::mutex> g(st->mu);
      block *spare = nullptr;
      for (block &b : st->captures) {
        // taken earlier by the same stream of the same capture, whose calls follow each other
        if (b.owned && !b.busy && b.owner == id && b.stream == s && s != cudaStreamPerThread) {
          b.busy = true;
          return b.p;
        }
        if (!b.owned && !b.busy) spare = &b;
      }
      if (spare) {
        *spare = block{spare->p, id, s, true, true};
        p = spare->p;
      }
    }
    if (!p) {
      if (!(p = st->allocate_now())) return nullptr;
      std::lock_guard<std::mutex> g(st->mu);
      st->captures.push_back(block{p, id, s, true, true});
    }
    cudaUserObject_t obj = nullptr;
    hold *h = new (std::nothrow) hold{st, p};
    if (h && cudaUserObjectCreate(&obj, h, give_back, 1, cudaUserObjectNoDestructorSync) == cudaSuccess) {
      if (cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove) == cudaSuccess) return p;
      cudaGetLastError();
      cudaUserObjectRelease(obj, 1);
      st->done(p, true);
      return nullptr;
    }
    cudaGetLastError();
    delete h;
    st->done(p, true);
    return nullptr;
  }

  void *take(cudaStream_t s, bool *once) {
    unsigned long long id = 0;
    const bool known = cudaStreamGetId(s, &id) == cudaSuccess;  // unlike a handle, never used again
    if (!known) cudaGetLastError();
    if (known) {
      std::lock_guard<std::mutex> g(mu);
      block *b = nullptr;
      for (block &c : streams) {
        if (c.busy || (c.owned && c.owner != id)) continue;
        b = &c;
        if (c.owned) break;
      }
      if (b) {
        *b = block{b->p, id, s, true, true};
        return b->p;
      }
    }
    void *p = nullptr;
    if (cudaMallocAsync(&p, bytes, s) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    if (zero && cudaMemsetAsync(p, 0, zero, s) != cudaSuccess) {
      cudaGetLastError();
      cudaFreeAsync(p, s);
      return nullptr;
    }
    std::lock_guard<std::mutex> g(mu);
    if (known && streams.size() < kMaxStreams)
      streams.push_back(block{p, id, s, true, true});
    else
      *once = true;
    return p;
  }
};

call_blocks::call_blocks() = default;

call_blocks::~call_blocks() {
  if (!st_) return;
  std::vector<state::block> all;
  {
    std::lock_guard<std::mutex> g(st_->mu);
    all.swap(st_->streams);
    all.insert(all.end(), st_->captures.begin(), st_->captures.end());
    st_->captures.clear();
  }
  for (state::block &b : all) cudaFree(b.p);
}

cudaError_t call_blocks::init(size_t bytes, size_t zero, size_t *acct) {
  auto st = std::make_shared<state>();
  st->bytes = bytes;
  st->zero = zero;
  void *p = nullptr;
  const cudaError_t e = cudaMalloc(&p, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return e;
  }
  st->streams.reserve(kMaxStreams);
  st->streams.push_back(state::block{p, 0, nullptr, false, false});
  st_ = std::move(st);
  *acct += bytes;
  return zero ? cudaMemset(p, 0, zero) : cudaSuccess;
}

call_scratch::call_scratch(const call_blocks &blocks, cudaStream_t stream) : st_(blocks.st_), stream_(stream) {
  if (!st_) return;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  cudaGraph_t graph = nullptr;
  if (cudaStreamGetCaptureInfo(stream, &status, &id, &graph, nullptr, nullptr) != cudaSuccess) {
    cudaGetLastError();  // the launches that follow report it
    return;
  }
  if (status == cudaStreamCaptureStatusNone)
    p_ = st_->take(stream, &once_);
  else if (status == cudaStreamCaptureStatusActive)
    p_ = call_blocks::state::take_captured(st_, graph, id, stream);
}

call_scratch::~call_scratch() {
  if (!p_) return;
  if (once_)
    cudaFreeAsync(p_, stream_);
  else
    st_->done(p_);
}

}  // namespace mfp
