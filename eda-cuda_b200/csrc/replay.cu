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
}

void Replays::run(const std::string& key, cudaStream_t s, const std::function<void()>& issue) {
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
    issue();
    return;
  }
  Entry& e = it->second;
  e.used = ++clock_;
  if (!e.exec && !e.refused) {
    try {
      Sequence q;
      issue();
      e.exec = q.instantiate();
      e.launches = q.launches();
    } catch (const std::exception&) {
      // the sequence is issued directly, where an error that is its own shows
    }
    if (!e.exec) {
      e.refused = true;
      (void)cudaGetLastError();
    }
  }
  if (!e.exec) {
    issue();
    return;
  }
  EDAB_CUDA(cudaGraphLaunch(e.exec, s));
  note_launch(e.launches);
}

}  // namespace edab
