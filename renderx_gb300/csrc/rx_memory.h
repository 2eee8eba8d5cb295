// Device memory: owned allocations (DevBuf), and the renders' buffers (Workspace), which the
// contexts of a device share and keep between calls.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

namespace rx {

// Device memory that a render takes its buffers from, as a stack of blocks.
class Workspace {
  struct Block {
    void* p;
    size_t size, used;
  };

 public:
  Workspace() = default;
  Workspace(const Workspace&) = delete;
  Workspace& operator=(const Workspace&) = delete;
  ~Workspace() { trim(0); }
  // `bytes` of device memory, 256-byte aligned: from the first block with room.
  cudaError_t alloc(size_t bytes, void** out);
  std::vector<size_t> marks() const {
    std::vector<size_t> used;
    for (const Block& b : blocks_) used.push_back(b.used);
    return used;
  }
  // Gives back what was taken since marks() returned `used`.
  void restore(const std::vector<size_t>& used) {
    for (size_t k = 0; k < blocks_.size(); k++) blocks_[k].used = k < used.size() ? used[k] : 0;
  }
  size_t size() const {
    size_t all = 0;
    for (const Block& b : blocks_) all += b.size;
    return all;
  }
  // Frees blocks from the top until at most `keep` bytes stay (nothing taken).
  void trim(size_t keep) {
    for (size_t all = size(); !blocks_.empty() && all > keep;) {
      all -= blocks_.back().size;
      pop();
    }
  }

 private:
  static cudaError_t take(Block& b, size_t bytes, void** out) {
    *out = static_cast<char*>(b.p) + b.used;
    b.used += bytes;
    return cudaSuccess;
  }
  void pop() {
    if (blocks_.back().p) cudaFree(blocks_.back().p);
    blocks_.pop_back();
  }
  std::vector<Block> blocks_;
};

// The workspaces of a device that no render holds: cudaMalloc and cudaFree of a render's
// buffers cost more than many renders do (1.3 of 2.1 ms for a 256^2 x 16 frame, 9 of 65 ms
// for VCM at 512^2). A render takes the workspace that was given back last, whichever
// context that was for, so contexts that render one after another share one, and there are
// as many as renders that ran at the same time. At most kKeep bytes stay in all of them,
// the least recently used are freed first; all are freed when an allocation of the library
// finds no memory, on request, and with the device's last context. Safe with several threads.
class WorkspacePool {
 public:
  static constexpr size_t kKeep = (size_t)8 << 30;
  static WorkspacePool& of(int device) {
    static std::mutex m;
    static auto* pools = new std::map<int, WorkspacePool>;  // outlives every context
    std::lock_guard<std::mutex> lock(m);
    return (*pools)[device];
  }
  std::unique_ptr<Workspace> take() {
    std::lock_guard<std::mutex> lock(m_);
    if (idle_.empty()) return std::unique_ptr<Workspace>(new Workspace);
    std::unique_ptr<Workspace> w = std::move(idle_.back());
    idle_.pop_back();
    return w;
  }
  // `w` with nothing taken from it and no work left that uses it.
  void give(std::unique_ptr<Workspace> w) {
    std::lock_guard<std::mutex> lock(m_);
    idle_.push_back(std::move(w));
    size_t all = 0;
    for (const auto& i : idle_) all += i->size();
    for (size_t k = 0; all > kKeep; k++) {
      const size_t had = idle_[k]->size();
      idle_[k]->trim(had - std::min(had, all - kKeep));
      all -= had - idle_[k]->size();
    }
    idle_.erase(std::remove_if(idle_.begin(), idle_.end(), [](const std::unique_ptr<Workspace>& i) { return i->size() == 0; }),
                idle_.end());
  }
  // Frees what no render holds; whether there was any.
  bool drain() {
    std::lock_guard<std::mutex> lock(m_);
    const bool any = !idle_.empty();
    idle_.clear();
    return any;
  }
  void add_context() {
    std::lock_guard<std::mutex> lock(m_);
    contexts_++;
  }
  void drop_context() {
    std::lock_guard<std::mutex> lock(m_);
    if (--contexts_ == 0) idle_.clear();
  }

 private:
  std::mutex m_;
  std::vector<std::unique_ptr<Workspace>> idle_;  // least recently used first
  int contexts_ = 0;
};

// cudaMalloc that has the memory kept for renders given back before it fails. A failure is
// returned and not left behind as the thread's last error, where a later launch would find it.
inline cudaError_t device_malloc(void** p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  int device = 0;
  cudaGetDevice(&device);
  if (WorkspacePool::of(device).drain()) e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation) cudaGetLastError();
  return e;
}

inline cudaError_t Workspace::alloc(size_t bytes, void** out) {
  bytes = (bytes + 255) & ~(size_t)255;
  for (Block& b : blocks_)
    if (b.p && b.size - b.used >= bytes) return take(b, bytes, out);
  Block b{nullptr, std::max({bytes, std::min(size() / 2, (size_t)512 << 20), (size_t)32 << 20}), 0};
  cudaError_t e = device_malloc(&b.p, b.size);
  if (e == cudaErrorMemoryAllocation) {  // give back the unused blocks, take no more than asked
    for (Block& u : blocks_)  // (an empty block keeps its place: the frames' marks go by it)
      if (u.p && u.used == 0) {
        cudaFree(u.p);
        u = Block{nullptr, 0, 0};
      }
    b.size = bytes;
    e = device_malloc(&b.p, b.size);
  }
  if (e != cudaSuccess) return e;
  blocks_.push_back(b);
  return take(blocks_.back(), bytes, out);
}

// A context's hold on a workspace: from the first Frame (one per render call) to its end. A
// frame gives back when it ends what was taken since it began, so a render made from a
// snapshot callback nests. Buffers are used on the context's stream (and on a side stream
// that the render waits for); the outermost frame waits for that stream, so another
// context can use the memory on its own. Not thread-safe, as calls on one context are not.
class WorkspaceHold {
 public:
  int device = 0;
  cudaStream_t stream = nullptr;
  class Frame {
   public:
    explicit Frame(WorkspaceHold& hold) : h(hold) {
      if (h.depth_++ == 0) h.ws_ = WorkspacePool::of(h.device).take();
      used = h.ws_->marks();
    }
    Frame(const Frame&) = delete;
    Frame& operator=(const Frame&) = delete;
    ~Frame() {
      if (h.depth_ == 1) cudaStreamSynchronize(h.stream);  // a render that failed may have left work
      h.ws_->restore(used);
      if (--h.depth_ == 0) WorkspacePool::of(h.device).give(std::move(h.ws_));
    }

   private:
    WorkspaceHold& h;
    std::vector<size_t> used;
  };
  cudaError_t alloc(size_t bytes, void** out) { return ws_->alloc(bytes, out); }

 private:
  std::unique_ptr<Workspace> ws_;
  int depth_ = 0;
};

// A buffer of a render, from its frame's workspace.
struct WsBuf {
  void* p = nullptr;
  size_t bytes = 0;
  cudaError_t alloc(WorkspaceHold& w, size_t b) {
    p = nullptr;
    bytes = 0;
    if (b == 0) return cudaSuccess;
    cudaError_t e = w.alloc(b, &p);
    if (e == cudaSuccess) bytes = b;
    return e;
  }
  template <class T>
  T* as() const { return static_cast<T*>(p); }
};

// A device allocation, released when its owner goes away (move-only).
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  DevBuf(DevBuf&& o) noexcept : p(o.p), bytes(o.bytes) {
    o.p = nullptr;
    o.bytes = 0;
  }
  DevBuf& operator=(DevBuf&& o) noexcept {
    if (this != &o) {
      release();
      p = o.p;
      bytes = o.bytes;
      o.p = nullptr;
      o.bytes = 0;
    }
    return *this;
  }
  ~DevBuf() { release(); }
  cudaError_t alloc(size_t b) {
    release();
    if (b == 0) return cudaSuccess;
    cudaError_t e = device_malloc(&p, b);
    if (e == cudaSuccess) bytes = b;
    else p = nullptr;
    return e;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
  }
  template <class T>
  T* as() const { return static_cast<T*>(p); }
};

}  // namespace rx
