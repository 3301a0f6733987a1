// Device tables that are built once for a set of matrices and found again by later calls.  A captured CUDA graph bakes in
// the addresses of the entry that its launches used, so an entry must outlive every graph that refers to it: each captured
// use gives the graph a reference (a CUDA user object, which the graph, its executable graphs and their unfinished launches
// hold), and an entry with references is never evicted.  Of the entries without references the least recently used one
// goes when there are too many.
#pragma once
#include <ATen/ATen.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAStream.h>

#include <list>
#include <memory>

#include "host_utils.h"

namespace b200 {

// Counts the captured graphs that refer to some device memory.
class GraphPins {
 public:
  bool pinned() const { return count_->load(std::memory_order_acquire) > 0; }

  // To be called for every use on `stream`: while it captures, the graph under construction gets a reference; otherwise
  // `tensors` are held back from reuse until the stream has passed this use, should they be freed.
  void use(const c10::cuda::CUDAStream& stream, std::initializer_list<at::Tensor> tensors) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    cudaGraph_t graph = nullptr;
    B200_CUDA_CHECK(cudaStreamGetCaptureInfo_v2(stream.stream(), &status, nullptr, &graph, nullptr, nullptr));
    if (status == cudaStreamCaptureStatusActive) {
      retain(graph);
      return;
    }
    for (const at::Tensor& t : tensors) c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(), stream);
  }

 private:
  using Count = std::atomic<int>;

  void retain(cudaGraph_t graph) {
    auto* ref = new std::shared_ptr<Count>(count_);
    count_->fetch_add(1, std::memory_order_relaxed);
    cudaUserObject_t object = nullptr;
    cudaError_t err = cudaUserObjectCreate(&object, ref, &GraphPins::release, 1, cudaUserObjectNoDestructorSync);
    if (err != cudaSuccess) {
      release(ref);
      B200_CUDA_CHECK(err);
    }
    err = cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove);
    if (err != cudaSuccess) {
      cudaUserObjectRelease(object, 1);   // calls release()
      B200_CUDA_CHECK(err);
    }
  }

  // Runs on a thread of the CUDA runtime, where no CUDA call is allowed: the memory itself is freed by a later eviction.
  static void CUDART_CB release(void* p) {
    auto* ref = static_cast<std::shared_ptr<Count>*>(p);
    (*ref)->fetch_sub(1, std::memory_order_release);
    delete ref;
  }

  std::shared_ptr<Count> count_ = std::make_shared<Count>(0);
};

// Entry needs `key` (comparable) and `pins` (GraphPins).  The caller holds its own lock around every call and for as long
// as it uses the returned entry.
// A process-wide cache is to be allocated and never deleted: when static objects are destroyed, the CUDA context may be gone,
// and freeing memory that several streams have used records events there.
template <typename Entry, size_t Capacity>
class PreparedCache {
 public:
  // The entry of `key`, now the most recently used one, or nullptr.
  template <typename Key>
  Entry* find(const Key& key) {
    for (auto it = entries_.begin(); it != entries_.end(); ++it)
      if (it->key == key) {
        entries_.splice(entries_.end(), entries_, it);
        return &entries_.back();
      }
    return nullptr;
  }

  Entry* insert(Entry entry) {
    size_t idle = 0;
    for (const Entry& e : entries_) idle += e.pins.pinned() ? 0 : 1;
    for (auto it = entries_.begin(); it != entries_.end() && idle >= Capacity;) {
      if (it->pins.pinned()) {
        ++it;
      } else {
        it = entries_.erase(it);
        --idle;
      }
    }
    entries_.push_back(std::move(entry));
    return &entries_.back();
  }

  void drop_idle() {
    entries_.remove_if([](const Entry& e) { return !e.pins.pinned(); });
  }

  size_t size() const { return entries_.size(); }
  size_t pinned() const {
    size_t n = 0;
    for (const Entry& e : entries_) n += e.pins.pinned() ? 1 : 0;
    return n;
  }

 private:
  std::list<Entry> entries_;   // least recently used first
};

}  // namespace b200
