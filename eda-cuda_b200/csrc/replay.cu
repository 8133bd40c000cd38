// SPDX-License-Identifier: Apache-2.0
// Replayed launch sequences (replay.hpp).
#include "replay.hpp"

#include "engine.cuh"

#include <atomic>

namespace edab {
namespace {
std::atomic<int64_t> g_built{0}, g_launched{0}, g_refused{0}, g_evicted{0};
}

ReplayCounts replay_counts() { return {g_built, g_launched, g_refused, g_evicted}; }

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
        ++g_evicted;
      }
      entries_.erase(old);
    }
    Entry& e = entries_[key];
    e.used = ++clock_;
    e.first = call_;
    issue();
    return;
  }
  Entry& e = it->second;
  e.used = ++clock_;
  if (!e.exec && !e.refused && e.first != call_) {
    try {
      Sequence q;
      issue();
      e.exec = q.instantiate();
      e.launches = q.launches();
      ++g_built;
    } catch (const std::exception&) {
      // the sequence is issued directly, where an error that is its own shows
    }
    if (!e.exec) {
      e.refused = true;
      ++g_refused;
      (void)cudaGetLastError();
    }
  }
  if (!e.exec) {
    issue();
    return;
  }
  EDAB_CUDA(cudaGraphLaunch(e.exec, s));
  note_launch(e.launches);
  ++g_launched;
}

}  // namespace edab
