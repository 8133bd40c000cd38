// SPDX-License-Identifier: Apache-2.0
// Replayed launch sequences (replay.hpp).
#include "replay.hpp"

#include "engine.cuh"

namespace edab {

void Replays::clear() {
  for (auto& [key, e] : entries_) {
    if (e.exec) cudaGraphExecDestroy(e.exec);
  }
  entries_.clear();
  if (capture_) cudaStreamDestroy(capture_);
  capture_ = nullptr;
}

void Replays::run(const std::string& key, cudaStream_t s, const std::function<void(cudaStream_t)>& issue) {
  auto it = entries_.find(key);
  if (it == entries_.end()) {
    if (entries_.size() >= kMost) {
      auto old = entries_.begin();
      for (auto k = entries_.begin(); k != entries_.end(); ++k) {
        if (k->second.used < old->second.used) old = k;
      }
      if (old->second.exec) {
        EDAB_CUDA(cudaStreamSynchronize(s));  // its last launch may still run
        cudaGraphExecDestroy(old->second.exec);
      }
      entries_.erase(old);
    }
    entries_[key].used = ++clock_;
    issue(s);
    return;
  }
  Entry& e = it->second;
  e.used = ++clock_;
  if (!e.exec && !e.refused) {
    if (!capture_) EDAB_CUDA(cudaStreamCreateWithFlags(&capture_, cudaStreamNonBlocking));
    cudaGraph_t graph = nullptr;
    bool issued = false;
    EDAB_CUDA(cudaStreamBeginCapture(capture_, cudaStreamCaptureModeRelaxed));
    try {
      issue(capture_);
      issued = true;
    } catch (const std::exception&) {
      // the capture ends below; the sequence is issued directly, where an error that is its own shows
    }
    const cudaError_t ended = cudaStreamEndCapture(capture_, &graph);
    if (issued && ended == cudaSuccess && graph) {
      if (cudaGraphInstantiate(&e.exec, graph, 0) != cudaSuccess) e.exec = nullptr;
    }
    if (graph) cudaGraphDestroy(graph);
    if (!e.exec) {
      e.refused = true;
      (void)cudaGetLastError();
    }
  }
  if (e.exec) EDAB_CUDA(cudaGraphLaunch(e.exec, s));
  else issue(s);
}

}  // namespace edab
