// SPDX-License-Identifier: Apache-2.0
// The launches of the engine's steps (launch.hpp).
#include "engine.cuh"

namespace edab {
namespace {

thread_local Sequence* t_building = nullptr;

}  // namespace

bool building_sequence() { return t_building != nullptr; }

Sequence::Sequence() {
  EDAB_CUDA(cudaGraphCreate(&graph_, 0));
  t_building = this;
}

Sequence::~Sequence() {
  t_building = nullptr;
  cudaGraphDestroy(graph_);
}

void Sequence::kernel(const cudaLaunchConfig_t& at, const void* f, void** args) {
  cudaKernelNodeParams p{};
  p.func = const_cast<void*>(f);
  p.gridDim = at.gridDim;
  p.blockDim = at.blockDim;
  p.sharedMemBytes = static_cast<unsigned>(at.dynamicSmemBytes);
  p.kernelParams = args;  // (their values are copied)
  cudaGraphNode_t node = nullptr;
  EDAB_CUDA(cudaGraphAddKernelNode(&node, graph_, after(), last_ ? 1 : 0, &p));
  for (unsigned i = 0; i < at.numAttrs; ++i) EDAB_CUDA(cudaGraphKernelNodeSetAttribute(node, at.attrs[i].id, &at.attrs[i].val));
  last_ = node;
  ++launches_;
}

void Sequence::zero(void* p, size_t bytes) {
  const bool words = bytes % 4 == 0 && reinterpret_cast<uintptr_t>(p) % 4 == 0;
  cudaMemsetParams m{};
  m.dst = p;
  m.elementSize = words ? 4 : 1;
  m.width = words ? bytes / 4 : bytes;
  m.height = 1;
  cudaGraphNode_t node = nullptr;
  EDAB_CUDA(cudaGraphAddMemsetNode(&node, graph_, after(), last_ ? 1 : 0, &m));
  last_ = node;
}

cudaGraphExec_t Sequence::instantiate() {
  cudaGraphExec_t exec = nullptr;
  EDAB_CUDA(cudaGraphInstantiate(&exec, graph_, 0));
  return exec;
}

void enqueue_config(const cudaLaunchConfig_t& at, const void* kernel, void** args) {
  if (t_building) {
    t_building->kernel(at, kernel, args);
    return;
  }
  (void)cudaLaunchKernelExC(&at, kernel, args);
  EDAB_LAUNCH("enqueue");
}

void enqueue_zero(void* p, size_t bytes, cudaStream_t s) {
  if (t_building) t_building->zero(p, bytes);
  else EDAB_CUDA(cudaMemsetAsync(p, 0, bytes, s));
}

}  // namespace edab
