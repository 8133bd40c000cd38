// SPDX-License-Identifier: Apache-2.0
// The launches of the engine's steps: onto a stream, or into the launch sequence that the calling
// thread is building. A sequence's graph is made node by node, each after the one before, not by
// capturing a stream: while a stream is captured no thread of the process may synchronise the device,
// and this library's callers are not to know when it captures.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <tuple>

namespace edab {

class Sequence {
 public:
  Sequence();   // the calling thread's launches go into this sequence ..
  ~Sequence();  // .. until here
  Sequence(const Sequence&) = delete;
  Sequence& operator=(const Sequence&) = delete;
  void kernel(const cudaLaunchConfig_t& at, const void* f, void** args);
  void zero(void* p, size_t bytes);
  cudaGraphExec_t instantiate();
  int64_t launches() const { return launches_; }  // its kernels

 private:
  cudaGraphNode_t* after() { return last_ ? &last_ : nullptr; }
  cudaGraph_t graph_ = nullptr;
  cudaGraphNode_t last_ = nullptr;
  int64_t launches_ = 0;
};

bool building_sequence();  // by the calling thread
void enqueue_config(const cudaLaunchConfig_t& at, const void* kernel, void** args);

// kernel<<<grid, block, smem, s>>>(args...) with clusters of cluster_x CTAs, counted and checked; into
// the calling thread's sequence while it builds one.
template <class... P, class... A>
void enqueue_clusters(unsigned cluster_x, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                      const A&... args) {
  static_assert(sizeof...(P) == sizeof...(A));
  std::tuple<P...> values(static_cast<P>(args)...);
  void* at[sizeof...(P)];
  std::apply([&](auto&... v) {
    size_t i = 0;
    ((at[i++] = const_cast<void*>(static_cast<const void*>(&v))), ...);
  }, values);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute cluster{};
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.x = cluster_x;
  cluster.val.clusterDim.y = 1;
  cluster.val.clusterDim.z = 1;
  cfg.attrs = &cluster;
  cfg.numAttrs = cluster_x > 0 ? 1 : 0;
  enqueue_config(cfg, reinterpret_cast<const void*>(kernel), at);
}
template <class... P, class... A>
void enqueue(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, const A&... args) {
  enqueue_clusters(0, kernel, grid, block, smem, s, args...);
}
// Sets bytes at p to zero, in the same way.
void enqueue_zero(void* p, size_t bytes, cudaStream_t s);

}  // namespace edab
