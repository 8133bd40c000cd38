// SPDX-License-Identifier: Apache-2.0
// Launch sequences of a workspace, replayed as CUDA graphs. Between two host reads of a mode the engine
// issues a fixed sequence of launches: it depends on the geometry, the call's constants, the
// workspace's address and a count or two (the rungs), never on the data. For small fields the
// sequence is bound by its launches (one signal of 2048 samples: 533 launches, 2.5 ms of kernels in
// 4.8 ms), so a sequence that a thread's workspace has run in an earlier call is built as a graph (launch.hpp),
// and from then on launched as one.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <functional>
#include <map>
#include <string>

namespace edab {

// What the process's sequences came to: graphs built and launched, sequences that could not be built, and
// graphs that left for others (the tests' evidence that calls replay).
struct ReplayCounts {
  int64_t built, launched, refused, evicted;
};
ReplayCounts replay_counts();

class Replays {
 public:
  ~Replays() { clear(); }
  // A call begins: the modes of one call share their sequences, so uses are counted over calls.
  void begin_call() { ++call_; }
  // Runs `issue`, which enqueues the sequence of `key`, on stream s: directly in the first call that comes to
  // the key, as its graph afterwards.
  void run(const std::string& key, cudaStream_t s, const std::function<void()>& issue);
  void clear();  // the graphs hold addresses of the workspace: none outlives its buffer

 private:
  struct Entry {
    cudaGraphExec_t exec = nullptr;
    bool refused = false;  // could not be built: always issued directly
    uint64_t used = 0;
    uint64_t first = 0;    // the call that came to it first
    int64_t launches = 0;  // of the graph
  };
  // The least recently used sequence leaves beyond this many: a program that cycles through more never
  // comes to a second call's use, so it builds no graph.
  static constexpr size_t kMost = 64;
  std::map<std::string, Entry> entries_;
  uint64_t clock_ = 0, call_ = 0;
};

}  // namespace edab
