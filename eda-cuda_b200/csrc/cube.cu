// SPDX-License-Identifier: Apache-2.0
// The separable cube filter: along every axis a running max, min or box sum of odd width 2r + 1,
// r = min((w - 1) / 2, n_a - 1), with half-sample reflection, by the van Herk / Gil-Werman scheme
// with the reference's canonical fold structure (cpp/src/field/vhgw.cu:1-36 of eda-cuda), so
// that every output depends only on the line, its length and the window:
//   - the extended line e in [-r, n + r) reads the line through half-sample reflection; it is cut
//     into segments of wa = 2r + 1 samples starting at o + k wa, o = (n (wa + 1) / 2) mod wa;
//   - G (prefix fold of a segment): 32-sample chunks from the segment start, a sequential fold in
//     each chunk, a sequential carry over the chunk totals, G = carry op local; H (suffix fold) is
//     G of the reversed line;
//   - y(x) = op(H(x - r), G(x + r)); a box window aligned with a segment takes (H + G) * 0.5.
// Box sums run axis 0 first and the last pass multiplies by fl_T(1 / prod of the clamped sides);
// max and min fold the integer order keys of the values (the order of max_c / min_c).
//
// A CTA runs one line group of one element: P rows of the contiguous axis, or a panel of P adjacent
// columns of an outer axis, staged in shared memory by 16-byte asynchronous copies (cube.cuh). The
// passes are in cube_ext.cu (max, min), cube_box.cu (sums) and cube_long.cu (1-D lines too long for
// that); this file chooses their launch shapes.
#include "cube.cuh"

#include <algorithm>
#include <mutex>

namespace edab {
using namespace cubes;
namespace {

thread_local void* t_long_lines = nullptr;
thread_local void* t_long_totals = nullptr;

struct DevFacts {
  int sms = 148;
  size_t smem = 227 * 1024;  // dynamic shared memory a CTA may take
};
DevFacts dev_facts() {
  static std::mutex mu;
  static DevFacts f[64];
  static bool have[64] = {};
  int dev = 0;
  EDAB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (!have[dev]) {
    int optin = 0, sms = 0;
    EDAB_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    EDAB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    f[dev].sms = sms;
    f[dev].smem = static_cast<size_t>(optin) - 2048;  // the kernel's static shared memory
    const int most = static_cast<int>(f[dev].smem);
    ext_allow_smem<float>(most);
    ext_allow_smem<double>(most);
    box_allow_smem<float>(most);
    box_allow_smem<double>(most);
    have[dev] = true;
  }
  return f[dev];
}

// A 1-D line is staged whole while two CTAs' lines fit an SM (a box pass's buffers: 9 000 float32 or
// 4 500 float64 samples); a longer one is cut into tiles: one float64 line of 20 011 samples takes
// 8.0 ms per decomposition in tiles, 13.5 ms staged or folded whole. The lines of 2-D and 3-D fields
// are shorter.
bool staged_line(const Geom& g, size_t es, size_t cap) {
  return g.dim > 1 || box_smem_bytes(g.n_last, 1, true, es) <= cap / 2;
}

// Lines per group (a power of two up to 8): 8 lines for column panels (whole sectors) and rows;
// fewer where the element's rows run out or the shared memory would hold fewer than two CTAs.
int lines_per_cta(const Geom& g, int axis, size_t es, size_t cap, size_t (*bytes)(int32_t, int, bool, size_t)) {
  const int32_t n = g.n[axis];
  const bool rows = axis == g.dim - 1;
  int P = 8;
  if (rows) {
    while (P > 1 && P / 2 >= g.rows) P /= 2;
  }
  while (P > 1 && bytes(n, P, rows, es) > cap / 2) P /= 2;
  return P;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <class T>
void launch_pass(cudaStream_t s, const Geom& g, PassArgs<T> a) {
  const DevFacts f = dev_facts();
  const bool rows = a.axis == g.dim - 1;
  const int32_t n = g.n[a.axis];
  const CubeTune tune = cube_tune_for(g, a.axis, sizeof(T));
  if (a.rungs > kMaxRungs) throw std::invalid_argument("edab: more rungs than a cube launch holds");
  if (!staged_line(g, sizeof(T), f.smem)) {
    if (t_long_lines == nullptr || t_long_totals == nullptr) {
      throw std::logic_error("edab: a long-line cube pass needs the thread's long-line scratch");
    }
    a.bytes = cube_bytes_counter();
    profile_cube_launch(s, true);
    launch_long<T>(s, g, a, t_long_lines, t_long_totals, f.sms, f.smem);
    profile_cube_launch(s, false);
    return;
  }
  const bool box = a.op == static_cast<int>(CubeOp::kBox);
  const auto bytes = box ? box_smem_bytes : ext_smem_bytes;
  int P = lines_per_cta(g, a.axis, sizeof(T), f.smem, bytes);
  if (tune.lines > 0 && tune.lines <= 8 && (tune.lines & (tune.lines - 1)) == 0 &&
      bytes(n, tune.lines, rows, sizeof(T)) <= f.smem &&
      (!rows || tune.lines <= std::max<int64_t>(1, g.rows))) {
    P = tune.lines;
  }
  if (box && bytes(n, P, rows, sizeof(T)) > f.smem) {
    throw std::invalid_argument("edab: an axis of " + std::to_string(n) + " samples exceeds the shared-memory line capacity");
  }
  int64_t groups;
  if (rows) {
    groups = (g.rows + P - 1) / P;
  } else {
    int64_t outer = 1;
    for (int ax = 0; ax < a.axis; ++ax) outer *= g.n[ax];
    groups = outer * (g.stride[a.axis] / P);
  }
  const int nf = a.op == static_cast<int>(CubeOp::kMaxMin) ? 2 : 1;
  // A first pass stages its input once for every rung of the ladder and both fields of a max + min
  // cube when the line groups alone fill the GPU; else every rung and field is a CTA of its own (one line
  // of 2048 samples, 7 rungs, max + min: 4.7 us against 64.8 us in one CTA; 64 lines of 4096: 17 against
  // 75 us; at 64 fields of 512 x 512 one staging for all is the faster: 293 against 7 x 66 us).
  const bool fills = groups * g.batch >= int64_t{kCubeCtas} * f.sms;
  // (an output over the input is only written by a CTA that has staged every line it reads and is
  // their only reader)
  const bool shared = a.in_stride == 0 && a.in1 == nullptr;
  const bool in_place = a.in0 != nullptr && (a.in0 == a.out0 || a.in0 == a.out1);
  const bool together = shared && (in_place || fills) && bytes(n, P, rows, sizeof(T)) <= f.smem;
  a.zr = together ? a.rungs : 1;
  a.zf = together ? nf : 1;
  if (groups > 0x7fffffffLL || g.batch > 65535) throw std::invalid_argument("edab: cube launch too large");
  if (!rows) {
    const uint32_t per_outer = static_cast<uint32_t>(g.stride[a.axis] / P);
    a.panels = PanelDiv{make_div31(per_outer), make_div31(static_cast<uint32_t>(g.pitch / P)),
                        static_cast<uint32_t>(groups / per_outer)};
  }
  a.lp = P == 8 ? 3 : (P == 4 ? 2 : (P == 2 ? 1 : 0));
  const int64_t es = static_cast<int64_t>(sizeof(T));
  if (!(aligned16(a.in0) && aligned16(a.in1) && aligned16(a.out0) && aligned16(a.out1) && aligned16(a.epi.aux) &&
        (a.in_stride * es) % 16 == 0 && (a.out_stride * es) % 16 == 0 && (g.field * es) % 16 == 0 &&
        (g.pitch * es) % 16 == 0)) {
    throw std::logic_error("edab: a cube pass needs fields on 16-byte boundaries");
  }
  const dim3 grid(static_cast<unsigned>(groups), static_cast<unsigned>(g.batch),
                  static_cast<unsigned>(a.rungs / a.zr * (nf / a.zf)));
  a.bytes = cube_bytes_counter();
  profile_cube_launch(s, true);
  const size_t smem = bytes(n, P, rows, sizeof(T));
  if (box) launch_box<T>(s, g, a, P, rows, grid, smem);
  else launch_ext<T>(s, g, a, P, rows, grid, smem);
  profile_cube_launch(s, false);
}

}  // namespace

template <class T>
void cube(cudaStream_t s, const Geom& g, CubeOp op, const CubeArgs<T>& c) {
  const int D = g.dim;
  const int32_t rungs = c.rungs < 1 ? 1 : c.rungs;
  PassArgs<T> base{};
  base.win = c.win;
  base.rungs = rungs;
  base.out_stride = c.out_stride;
  base.op = static_cast<int32_t>(op);
  if (op == CubeOp::kBox) {
    for (int ax = 0; ax < D; ++ax) {
      PassArgs<T> a = base;
      a.axis = ax;
      a.epi = c.epi;
      if (ax == 0) {
        a.in0 = c.in;
        a.bits = c.src_bits;
        a.bit = c.bit;
        a.in_stride = 0;
      } else {
        a.in0 = c.out0;
        a.in_stride = c.out_stride;
      }
      a.out0 = ax == D - 1 && c.epi.out ? c.epi.out : c.out0;
      launch_pass<T>(s, g, a);
    }
    return;
  }
  for (int ax = D - 1; ax >= 0; --ax) {
    PassArgs<T> a = base;
    a.axis = ax;
    const bool first = ax == D - 1;
    if (first) {
      a.in0 = c.in;
      a.in1 = nullptr;
      a.in_stride = 0;
    } else {
      a.in0 = c.out0;
      a.in1 = op == CubeOp::kMaxMin ? c.out1 : nullptr;
      a.in_stride = c.out_stride;
    }
    a.out0 = c.out0;
    a.out1 = c.out1;
    a.keys_out = ax > 0;
    launch_pass<T>(s, g, a);
  }
}

void set_long_line_scratch(void* lines, void* totals) {
  t_long_lines = lines;
  t_long_totals = totals;
}

size_t long_line_scratch_bytes(const Geom& g, size_t es) {
  return staged_line(g, es, dev_facts().smem) ? 0 : long_line_part(g, es);
}

size_t fold_scratch_bytes(const Geom& g, size_t es) {
  if (g.dim != 1 || box_smem_bytes(g.n_last, 1, true, es) <= dev_facts().smem) return 0;
  return (static_cast<size_t>(g.batch) * static_cast<size_t>(g.pitch) * es + 255) / 256 * 256 +
         static_cast<size_t>(kMaxRungs) * static_cast<size_t>(g.batch) * 2 * static_cast<size_t>(tot_slots(g.n_last)) * es;
}

size_t long_totals_scratch_bytes(const Geom& g, size_t es) {
  return staged_line(g, es, dev_facts().smem) ? 0 : long_totals_part(g, es);
}

template <class T>
void cube_simple(cudaStream_t s, const Geom& g, CubeOp op, const T* in, T* out0, T* out1, const int32_t* win) {
  CubeArgs<T> a{};
  a.in = in;
  a.out0 = out0;
  a.out1 = out1;
  a.win = win;
  a.rungs = 1;
  cube<T>(s, g, op, a);
}

template void cube<float>(cudaStream_t, const Geom&, CubeOp, const CubeArgs<float>&);
template void cube<double>(cudaStream_t, const Geom&, CubeOp, const CubeArgs<double>&);
template void cube_simple<float>(cudaStream_t, const Geom&, CubeOp, const float*, float*, float*, const int32_t*);
template void cube_simple<double>(cudaStream_t, const Geom&, CubeOp, const double*, double*, double*, const int32_t*);

}  // namespace edab
