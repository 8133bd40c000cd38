// SPDX-License-Identifier: Apache-2.0
// What the cube filter's passes share (cube.cu, cube_ext.cu, cube_box.cu): the window geometry, the
// layouts of a line group in shared memory, its staging, and the arguments of a pass.
#pragma once

#include "engine.cuh"

#include <climits>

namespace edab {
namespace cubes {

// Threads of a cube CTA, and CTAs per SM the registers are bounded for.
constexpr int kCubeThreads = 256;
constexpr int kCubeCtas = 4;
constexpr int kWarps = kCubeThreads / 32;

// The window of one line: r the clamped half width, wa = 2r + 1 the segment length, o the segments'
// offset, k_lo the first segment, nseg their number, cps the 32-sample chunks of a segment.
struct Win {
  int32_t r, wa, o, k_lo, nseg, cps;
};
// 32-bit arithmetic (the 64-bit integer divisions of a general formula are long emulated sequences
// on the GPU): n (wa + 1) / 2 = n (r + 1) modulo wa = 2r + 1, where 2 (r + 1) = 1, is n / 2 for an
// even n and (n - 1) / 2 + (r + 1) for an odd one.
__device__ __forceinline__ int32_t floor_div32(int32_t a, int32_t b) {  // b > 0
  const int32_t q = a / b;
  return (a % b != 0 && a < 0) ? q - 1 : q;
}
__device__ __forceinline__ Win make_win(int32_t n, int32_t w) {
  Win q;
  const int32_t half = (w - 1) >> 1;
  q.r = min(half, n - 1);
  q.wa = 2 * q.r + 1;
  q.o = ((n >> 1) + (n & 1) * (q.r + 1)) % q.wa;
  q.k_lo = floor_div32(q.r - q.o, q.wa);
  const int32_t k_hi = floor_div32(n - 1 + q.r - q.o, q.wa);
  q.nseg = k_hi - q.k_lo + 1;
  q.cps = (q.wa + 31) >> 5;
  return q;
}

// Chunk totals per line and direction (nseg cps <= tot_slots(n) for every window).
__host__ __device__ constexpr int32_t tot_slots(int32_t n) { return n / 8 + 24; }
// Line stride of the row layout in elements: the padded row rounded up, plus 16 bytes (4 words
// modulo 32 for 4-byte samples, 2 elements modulo 16 for 8-byte samples): the 8 lines of a group
// lie in distinct banks, one sample or one 16-byte unit of each.
template <class T>
__host__ __device__ constexpr int32_t row_stride(int32_t n) {
  return sizeof(T) == 4 ? ((n + 31) & ~31) + 4 : ((n + 15) & ~15) + 2;
}
// Elements of one line-group buffer (a multiple of 16 bytes).
template <class T>
__host__ __device__ constexpr int32_t group_elems(int32_t n, int P, bool rows) {
  return rows ? P * row_stride<T>(n) : ((n * P + 3) & ~3);
}

// Order keys are signed integers of the samples' size.
template <class T>
struct KeyType;
template <>
struct KeyType<float> {
  using type = int32_t;
};
template <>
struct KeyType<double> {
  using type = long long;
};
template <class K>
__device__ __forceinline__ K key_min() {
  if constexpr (sizeof(K) == 4) return INT_MIN;
  else return LLONG_MIN;
}

// Order key of v as an integer: integer order = order of max_c / min_c; its own inverse on the bits.
__device__ __forceinline__ int32_t okey_i(float v) {
  const int32_t b = __float_as_int(v);
  return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ __forceinline__ long long okey_i(double v) {
  const long long b = __double_as_longlong(v);
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ float key_back(int32_t k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }
__device__ __forceinline__ double key_back(long long k) {
  return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffLL));
}

// Division of a 31-bit unsigned number by a constant d < 2^31: with 2^(s-1) < d <= 2^s and
// m = floor(2^32 (2^s - d) / d) + 1, x / d = (umulhi(x, m) + x) >> s (the sum stays below 2^32).
struct Div31 {
  uint32_t d, m, s;
  __device__ __forceinline__ uint32_t div(uint32_t x) const { return (__umulhi(x, m) + x) >> s; }
};
inline Div31 make_div31(uint32_t d) {
  Div31 r{d, 0, 0};
  while ((uint64_t{1} << r.s) < d) ++r.s;
  r.m = static_cast<uint32_t>(((uint64_t{1} << 32) * ((uint64_t{1} << r.s) - d)) / d + 1);
  return r;
}
// The panels of a pass along an outer axis: per outer index, and per row of the field.
struct PanelDiv {
  Div31 per_outer, per_row;
  uint32_t outer;
};

template <class T>
struct PassArgs {
  const T* in0;           // input of field 0 (rung 0 when in_stride != 0)
  const T* in1;           // input of field 1 (max + min, later passes)
  const uint8_t* bits;    // box first pass: bit `bit` of this u8 field
  int32_t bit;
  T* out0;
  T* out1;
  const int32_t* win;     // [rungs * B]
  int32_t rungs;          // rungs of the launch
  int64_t in_stride;      // per-rung input offset (0: one input shared by every rung)
  int64_t out_stride;     // per-rung output offset
  int32_t op;             // CubeOp
  int32_t axis;
  BoxEpilogue<T> epi;     // box: what the last pass stores
  int32_t zr, zf;         // rungs and fields a CTA runs from one staging (1: blockIdx.z counts them)
  int32_t keys_out;       // max / min: the output holds order keys (another axis follows)
  int32_t lp;             // rows: log2 of the lines per group
  PanelDiv panels;        // the line groups of an outer axis
  unsigned long long* bytes;  // instrumentation: the pass's algorithmic bytes (nullptr: off)
};

// Where a line group lies inside its element: rows, line p at base + p pitch; column panels, line
// p at base + p (rows of the panel `inner` apart). mask: bit p set for a line of the field (rows
// inside the element, columns left of the row padding).
struct GroupPos {
  int64_t base;
  uint32_t mask;
};
template <bool ROWS>
__device__ __forceinline__ GroupPos group_at(const Geom& g, uint32_t grp, int32_t n, uint32_t inner, uint32_t P,
                                             const PanelDiv& d) {
  GroupPos s;
  if constexpr (ROWS) {
    const uint32_t c = grp * P;  // rows < 2^31
    s.base = static_cast<int64_t>(c) * static_cast<uint32_t>(g.pitch);
    const int64_t left = g.rows - c;
    s.mask = left >= P ? (1u << P) - 1u : (left > 0 ? (1u << left) - 1u : 0u);
  } else {
    const uint32_t o = d.outer > 1 ? d.per_outer.div(grp) : 0u;
    const uint32_t cg = grp - o * d.per_outer.d;
    const uint32_t col = (cg - d.per_row.div(cg) * d.per_row.d) * P;  // the panel's column in its row
    s.base = static_cast<int64_t>(o) * n * inner + cg * P;
    const int32_t room = g.n_last - static_cast<int32_t>(col);
    s.mask = room >= static_cast<int32_t>(P) ? (1u << P) - 1u : (room > 0 ? (1u << room) - 1u : 0u);
  }
  return s;
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}

// Stages the group's lines in V (row layout: sample i of line p at p LS + i; panel: at i P + p); the
// caller's stage_wait and barrier follow. 16-byte asynchronous copies where the layout allows them;
// plain loads for a bit field and for panels narrower than 16 bytes. (Every field lies on a 16-byte
// boundary with strides of whole 16-byte units: launch_pass checks it.)
template <class T, int P, bool ROWS>
__device__ __forceinline__ void stage_lines(const Geom& g, const PassArgs<T>& a, T* __restrict__ V, const T* src,
                                            const uint8_t* bits, const GroupPos& s, int32_t n, int32_t LS,
                                            uint32_t inner) {
  constexpr int VW = 16 / static_cast<int>(sizeof(T));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if constexpr (ROWS) {
    const int lp = P == 8 ? 3 : a.lp;
    const int lines = 1 << lp;
    const int per = kWarps >> lp;  // warps per line
    const int p = warp / per;
    if (p < lines && ((s.mask >> p) & 1u)) {
      const int64_t at = s.base + static_cast<int64_t>(p) * g.pitch;
      T* dst = V + p * LS;
      const int32_t i0 = lane + 32 * (warp - p * per), di = 32 * per;
      if (bits) {
        for (int32_t i = i0; i < n; i += di) dst[i] = ((bits[at + i] >> a.bit) & 1u) ? T(1) : T(0);
      } else {
        const int32_t units = (n + VW - 1) / VW;
        for (int32_t u = i0; u < units; u += di) cp_async16(dst + u * VW, src + at + u * VW);
      }
    }
  } else if (s.mask) {
    if (!bits && P >= VW) {
      constexpr int QP = P >= VW ? P / VW : 1;
      const int q = (threadIdx.x % QP) * VW;
      const T* col = src + s.base + q;
      int32_t i = threadIdx.x / QP;
      const T* from = col + static_cast<int64_t>(i) * inner;
      const int64_t step = static_cast<int64_t>(kCubeThreads / QP) * inner;
      for (; i < n; i += kCubeThreads / QP) {
        cp_async16(V + i * P + q, from);
        from += step;
      }
    } else {
      const int p = threadIdx.x % P;
      for (int32_t i = threadIdx.x / P; i < n; i += kCubeThreads / P) {
        const int64_t at = s.base + static_cast<int64_t>(i) * inner + p;
        V[i * P + p] = bits ? (((bits[at] >> a.bit) & 1u) ? T(1) : T(0)) : src[at];
      }
    }
  }
}
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// W consecutive values (16 bytes, or one) as one access.
template <class T, int W>
struct Pack {
  T v[W];
};
template <class T, int W>
__device__ __forceinline__ Pack<T, W> load_pack(const T* p) {
  Pack<T, W> r;
  if constexpr (W * sizeof(T) == 16) {
    const int4 q = *reinterpret_cast<const int4*>(p);
    memcpy(&r, &q, 16);
  } else {
#pragma unroll
    for (int k = 0; k < W; ++k) r.v[k] = p[k];
  }
  return r;
}
template <class T, int W>
__device__ __forceinline__ void store_pack(T* p, const Pack<T, W>& r) {
  if constexpr (W * sizeof(T) == 16) {
    int4 q;
    memcpy(&q, &r, 16);
    *reinterpret_cast<int4*>(p) = q;
  } else {
#pragma unroll
    for (int k = 0; k < W; ++k) p[k] = r.v[k];
  }
}

// The value that a box cube's last pass stores for the canonical sum y: the cube's scale, then the
// epilogue (its arithmetic is that of the method's pointwise steps: the threshold field
// cpp/src/method/stats_fields.cu:25-69, the raw window cpp/src/method/stats_fields.cu:340-369).
// valid: y is an output (not a pad).
template <class T, BoxEpi EPI>
struct BoxStore {
  T fac;
  double sigma_n, floor_n, f2, tol;  // kTau: the element's
  __device__ __forceinline__ void element(const PassArgs<T>& a, int64_t b, T scale) {
    fac = scale;
    if constexpr (EPI == BoxEpi::kTau) {
      sigma_n = a.epi.el[b].sigma_n;
      tol = a.epi.el[b].tol;
      const double f = __dmul_rn(a.epi.sig_noise, sigma_n);
      floor_n = f > 0.0 ? f : 0.0;
      f2 = __dmul_rn(a.epi.fine_theta, a.epi.el[b].sigma_x);
    }
  }
  __device__ __forceinline__ T operator()(const PassArgs<T>& a, int64_t b, T y, T aux, bool valid) const {
    y = mul_rn(y, fac);
    if constexpr (EPI == BoxEpi::kDetSq) {
      const T d = sub_rn(aux, y);
      return mul_rn(d, d);
    } else if constexpr (EPI == BoxEpi::kTau) {
      if (valid && !(isfinite(y) && isfinite(sigma_n))) a.epi.el[b].nonfinite = 1;
      const T lev = sqrt_rn<T>(y > T(0) ? y : T(0));
      const double ld = static_cast<double>(lev);
      double t = __dmul_rn(a.epi.sig_theta, ld > floor_n ? ld : floor_n);
      t = t > tol ? t : tol;
      if (a.epi.floor2) t = t > f2 ? t : f2;
      return static_cast<T>(t);
    } else if constexpr (EPI == BoxEpi::kRho) {
      const T sq = mul_rn(y, y);
      const T acc = a.epi.aux ? add_rn(aux, sq) : sq;
      if (!a.epi.finish) return acc;
      const T dens = sqrt_rn<T>(acc);
      return dens > T(0) ? div_rn<T>(a.epi.two_kappa, dens > a.epi.tiny ? dens : a.epi.tiny) : inf_t<T>();
    } else if constexpr (EPI == BoxEpi::kClip) {
      return clip(y, T(0), T(1));
    } else if constexpr (EPI == BoxEpi::kExp) {
      return exp_t<T>(y);
    } else {
      return y;
    }
  }
};

// Max / min passes (cube_ext.cu) and box passes (cube_box.cu): the shared memory of a CTA, and the
// launch of a pass with P lines per group.
size_t ext_smem_bytes(int32_t n, int P, bool rows, size_t es);
size_t box_smem_bytes(int32_t n, int P, bool rows, size_t es);
template <class T>
void ext_allow_smem(int bytes);
template <class T>
void box_allow_smem(int bytes);
template <class T>
void launch_ext(cudaStream_t s, const Geom& g, const PassArgs<T>& a, int P, bool rows, dim3 grid, size_t smem);
template <class T>
void launch_box(cudaStream_t s, const Geom& g, const PassArgs<T>& a, int P, bool rows, dim3 grid, size_t smem);
// The passes over 1-D lines that are not staged whole (cube_long.cu) and their scratch.
size_t long_line_part(const Geom& g, size_t es);
size_t long_totals_part(const Geom& g, size_t es);
template <class T>
void launch_long(cudaStream_t s, const Geom& g, const PassArgs<T>& a, void* lines, void* totals, int sms,
                 size_t smem_cap);

}  // namespace cubes
}  // namespace edab
