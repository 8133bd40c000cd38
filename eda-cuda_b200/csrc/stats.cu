// SPDX-License-Identifier: Apache-2.0
// The statistics of a mode: canonical energies, exact selections, the noise levels, the local
// threshold field, the significant extrema, the raw local window, the scale field with its
// face-connected components and the per-voxel floor, G2's rung test and G3's coarse median.
// Semantics of eda-cuda (cpp/src/method/stats*.cu, cpp/src/field/common.cuh:133-259); every
// decision is an integer reduction or an exact order statistic, so nothing depends on the order
// of atomics or on the launch shape.
#include "engine.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

namespace edab {
namespace {

// ---------------------------------------------------------------------------------------------
// Canonical energies. A warp per row: sum v^2 in double over each 32-sample chunk (sequential),
// the pairwise tree over the chunks padded with zeros to a power of two (32 chunks per warp step
// by shuffles, the steps' sums by a binary-counter stack), and the exact max |v|.
struct RowPartial {
  double sum_sq;
  uint64_t amax;
};

__device__ __forceinline__ double warp_tree32(double v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const double o = __shfl_down_sync(0xffffffffu, v, d);
    if ((lane & (2 * d - 1)) == 0) v = __dadd_rn(v, o);
  }
  return v;  // lane 0
}

// The sums of a binary counter over a row's steps, in order: what a tree over all of them gives.
struct StepTree {
  double stack[24];
  int level[24];
  int top = 0;
  __device__ __forceinline__ void add(double v) {
    int l = 0;
    while (top > 0 && level[top - 1] == l) {
      v = __dadd_rn(stack[top - 1], v);
      --top;
      ++l;
    }
    stack[top] = v;
    level[top] = l;
    ++top;
  }
  __device__ __forceinline__ double total() const {
    double v = stack[top - 1];
    for (int i = top - 2; i >= 0; --i) v = __dadd_rn(stack[i], v);
    return v;
  }
};

// One step of a row: the warp's tree over the chunks [32 step, 32 step + 32), staged by coalesced 16-byte loads
// and padded with zeros (+0 changes no sum of squares); the lane's max |v| (as T's bits) and whether a
// sample is not finite are added to amax and bad (counted).
template <class T>
using BitsOf = std::conditional_t<sizeof(T) == 4, uint32_t, uint64_t>;
template <class T>
__device__ __forceinline__ double row_step(const T* __restrict__ row, int32_t n, int32_t step, T* tile, BitsOf<T>& amax,
                                           unsigned& bad) {
  using U = BitsOf<T>;
  constexpr U kAbs = ~U(0) >> 1, kInf = sizeof(T) == 4 ? U(0x7f800000u) : static_cast<U>(0x7ff0000000000000ULL);
  const int lane = threadIdx.x & 31;
  const int32_t i0 = step * 1024, left = min(n - i0, 1024);
  __syncwarp();
  // 16 bytes per lane and load, eight loads in flight (rows begin on 128-byte boundaries, and their pitch is
  // a multiple of 32 samples: a load that straddles the row's end stays inside it)
  constexpr int V = 16 / static_cast<int>(sizeof(T));
  struct alignas(16) Vec {
    T e[V];
  };
  T* to = tile + 33 * ((V * lane) >> 5) + ((V * lane) & 31);
#pragma unroll 1
  for (int k0 = 0; k0 < 32 / V; k0 += 8) {
    if (32 * V * k0 >= left) break;
    Vec v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int32_t i = V * (32 * (k0 + k) + lane);
      if (i < left) v[k] = *reinterpret_cast<const Vec*>(row + i0 + i);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int32_t i = V * (32 * (k0 + k) + lane);
      if (32 * V * (k0 + k) < left) {
#pragma unroll
        for (int e = 0; e < V; ++e) to[33 * V * (k0 + k) + e] = i + e < left ? v[k].e[e] : T(0);
      }
    }
  }
  __syncwarp();
  double acc = 0.0;
  if (32 * lane < left) {
    const T* t = tile + 33 * lane;
#pragma unroll 2
    for (int32_t j = 0; j < 32; j += 8) {
      T v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = t[j + k];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const double d = static_cast<double>(v[k]);
        acc = __dadd_rn(acc, __dmul_rn(d, d));
        U u;
        memcpy(&u, &v[k], sizeof u);
        u &= kAbs;
        amax = max(amax, u);
        bad += u >= kInf ? 1u : 0u;
      }
    }
  }
  return warp_tree32(acc);
}

// Rows of one step: a warp per row. Longer rows (per_row): a CTA per row, its warps over the steps. Bound by
// the loads' latency (with scalar loads 8 % of the DRAM's rate, 13 of 15 stalled warps on a load): 64 images
// of 512 x 512 float32 63 -> 26 us, 4 volumes of 256^3 316 -> 167 us, a line of 20 011 float64 samples 45
// -> 13 us (54 us by one warp).
constexpr int kMaxSteps = 128;
template <class T>
constexpr int kRowThreads = 1024 / static_cast<int>(sizeof(T));  // (the tiles of 8 float or 4 double warps: 34 KB)
template <class T>
__global__ void __launch_bounds__(kRowThreads<T>) row_partials(const T* __restrict__ f, Geom g, RowPartial* rows,
                                                         uint64_t* nonfinite, bool per_row) {
  __shared__ T tile_s[kRowThreads<T> / 32][32 * 33];
  __shared__ double step_s[kMaxSteps];
  __shared__ BitsOf<T> amax_s[kRowThreads<T> / 32];
  __shared__ unsigned bad_s[kRowThreads<T> / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t total = g.batch * g.rows;
  T* tile = tile_s[warp];
  for (int64_t q = per_row ? blockIdx.x : blockIdx.x * static_cast<int64_t>(kRowThreads<T> / 32) + warp; q < total;
       q += static_cast<int64_t>(gridDim.x) * (per_row ? 1 : kRowThreads<T> / 32)) {
    const int32_t n = g.len ? elem_len(g, q / g.rows) : g.n_last;
    const int32_t steps = (n + 1023) >> 10;
    const T* row = f + q * g.pitch;
    BitsOf<T> amax = 0;
    unsigned bad = 0;
    double one = 0.0;
    for (int32_t k = per_row ? warp : 0; k < steps; k += kRowThreads<T> / 32) {
      one = row_step(row, n, k, tile, amax, bad);
      if (per_row && lane == 0) step_s[k] = one;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      const BitsOf<T> o = __shfl_down_sync(0xffffffffu, amax, d);
      amax = o > amax ? o : amax;
      bad += __shfl_down_sync(0xffffffffu, bad, d);
    }
    if (per_row) {
      if (lane == 0) {
        amax_s[warp] = amax;
        bad_s[warp] = bad;
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        StepTree tree;
        for (int32_t k = 0; k < steps; ++k) tree.add(step_s[k]);
        one = tree.total();
        for (int w = 1; w < kRowThreads<T> / 32; ++w) {
          amax = amax_s[w] > amax ? amax_s[w] : amax;
          bad += bad_s[w];
        }
      }
    }
    if (per_row ? threadIdx.x == 0 : lane == 0) {
      T largest;
      memcpy(&largest, &amax, sizeof largest);
      rows[q] = RowPartial{one, abs_bits(largest)};
      if (nonfinite && bad) atomicAdd(reinterpret_cast<unsigned long long*>(&nonfinite[q / g.rows]), bad);
    }
    if (per_row) __syncthreads();  // the next row rewrites the steps' sums
  }
}

// One CTA per element: the pairwise tree over the element's row sums (leaves of 1024 rows in
// shared memory, the leaves by a binary-counter stack), the max of the row maxima.
constexpr int kLeaf = 1024;
__global__ void __launch_bounds__(kThreads) element_totals(Geom g, const RowPartial* rows, double* energy,
                                                           double* amax_out) {
  __shared__ double leaf[kLeaf];
  __shared__ uint64_t am[kThreads / 32];
  const int tid = threadIdx.x;
  for (int64_t b = blockIdx.x; b < g.batch; b += gridDim.x) {
    const RowPartial* base = rows + b * g.rows;
    double stack[40];
    int level[40];
    int top = 0;
    uint64_t amax = 0;
    for (int64_t start = 0; start < g.rows; start += kLeaf) {
      for (int k = 0; k < kLeaf / kThreads; ++k) {
        const int i = tid + k * kThreads;
        double v = 0.0;
        if (start + i < g.rows) {
          const RowPartial p = base[start + i];
          v = p.sum_sq;
          amax = p.amax > amax ? p.amax : amax;
        }
        leaf[i] = v;
      }
      __syncthreads();
      for (int d = 1; d < kLeaf; d <<= 1) {
        for (int i = tid * 2 * d; i < kLeaf; i += kThreads * 2 * d) leaf[i] = __dadd_rn(leaf[i], leaf[i + d]);
        __syncthreads();
      }
      if (tid == 0) {
        double v = leaf[0];
        int l = 0;
        while (top > 0 && level[top - 1] == l) {
          v = __dadd_rn(stack[top - 1], v);
          --top;
          ++l;
        }
        stack[top] = v;
        level[top] = l;
        ++top;
      }
      __syncthreads();
    }
    for (int d = 16; d > 0; d >>= 1) {
      const uint64_t o = __shfl_down_sync(0xffffffffu, amax, d);
      amax = o > amax ? o : amax;
    }
    if ((tid & 31) == 0) am[tid >> 5] = amax;
    __syncthreads();
    if (tid == 0) {
      double v = 0.0;
      if (top > 0) {
        v = stack[top - 1];
        for (int i = top - 2; i >= 0; --i) v = __dadd_rn(stack[i], v);
      }
      uint64_t m = 0;
      for (int w = 0; w < kThreads / 32; ++w) m = am[w] > m ? am[w] : m;
      if (energy) energy[b] = v;
      if (amax_out) amax_out[b] = bits_d(m);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// Exact selections (order statistics) by most-significant-digit radix selection on order keys,
// unsigned integers that sort as the values do (-0 counts as +0). Float32 items without a centre
// select on 32-bit keys of the float values (three digits: 11, 11 and 10 bits); every other
// selection on 64-bit keys of the values as doubles (six digits: five of 11 bits, one of 9).
//
// One thread-block cluster (up to 8 CTAs) serves one element, all digits in one launch: each CTA
// counts its share of the items per digit value in shared memory; the counts are added into the
// cluster leader's shared table through distributed shared memory; the leader's threads find the
// digit value that holds the wanted rank by a block-wide prefix sum and publish the extended prefix.
// Two ranks are followed at once (a median's middle pair, a quantile's neighbours); they share one
// table while their resolved digits agree.
namespace cg = cooperative_groups;

constexpr int kDigitBits = 11;
constexpr int kDigitBins = 1 << kDigitBits;
constexpr int kSelClusterMax = 8;
// Items of an element (at least, at most) and of the batch that the split form takes: its list of 8 % is
// selected from by one CTA per element, to which batches of few elements leave the GPU. Medians of float32
// samples, us without / with it: 8 elements of 512 x 512 56 / 71, 12 64 / 72, 15 72 / 74; 8 of 1500 x 1400
// 201 / 319, 12 314 / 318, 15 354 / 333; 1 of 256^3 192 / 1708. Above the most: 16 elements of 2048 x 4096
// 1292 / 1255, 24 1895 / 1498, 16 of 256^3 2498 / 2590 and their differences along three axes 15 114 / 17 537.
// Below the total: 15 elements of 256 x 256 32 / 47, 16 60 / 48.
constexpr int64_t kSplitItems = 65536, kSplitMost = int64_t{1} << 22, kSplitTotal = int64_t{1} << 21, kSplitBatch = 16;
constexpr int kSelWide = 1024;  // threads of a cluster's CTA in a small batch
// The cluster form for batches that fill the GPU with clusters (1), or the grid-wide form always (0).
#ifndef EDAB_SEL_CLUSTERS
#define EDAB_SEL_CLUSTERS 1
#endif
constexpr bool kSelClusters = EDAB_SEL_CLUSTERS != 0;
constexpr size_t kSelSmem = 2 * kDigitBins * sizeof(unsigned long long) + 2 * kDigitBins * sizeof(uint32_t);

__device__ __forceinline__ uint32_t order_key(float v) {
  uint32_t u = __float_as_uint(v);
  if ((u & 0x7fffffffu) == 0u) u = 0u;
  return (u & 0x80000000u) ? ~u : (u ^ 0x80000000u);
}
__device__ __forceinline__ uint64_t order_key(double v) {
  uint64_t u = static_cast<uint64_t>(__double_as_longlong(v));
  if ((u & 0x7fffffffffffffffULL) == 0ULL) u = 0ULL;
  return (u >> 63) ? ~u : (u ^ 0x8000000000000000ULL);
}
__device__ __forceinline__ double key_value(uint32_t k) {
  return static_cast<double>(__uint_as_float((k & 0x80000000u) ? (k ^ 0x80000000u) : ~k));
}
__device__ __forceinline__ double key_value(uint64_t k) {
  return bits_d((k >> 63) ? (k ^ 0x8000000000000000ULL) : ~k);
}

template <class T>
struct SelView {
  Sel<T> sel;
  int32_t naxes;
  int32_t ax[kMaxDim];
  int64_t items;
};

// Item t of element b (a voxel, or a forward difference along one of the pooled axes) as a value of
// the element's dtype; false where t is a pad, masked out, or has no forward neighbour.
template <class T>
__device__ __forceinline__ bool sel_raw(const Geom& g, const SelView<T>& a, int64_t b, int64_t t, T* out) {
  if (a.sel.src == SelSrc::kField) {
    if (is_pad_b(g, b, t)) return false;
    const int64_t i = b * g.field + t;
    if (a.sel.mask != nullptr && (a.sel.mask[i] & a.sel.bits) == 0) return false;
    *out = a.sel.field[i];
    return true;
  }
  const int64_t k = static_cast<int64_t>(__umul64hi(static_cast<uint64_t>(t), g.field_inv));  // t < 3 field
  const int64_t v = t - k * g.field;
  const int axis = k == 0 ? a.ax[0] : (k == 1 ? a.ax[1] : a.ax[2]);
  if (is_pad_b(g, b, v) || coord_of(g, v, axis) >= elem_n(g, b, axis) - 1) return false;
  const int64_t i = b * g.field + v;
  const int64_t st = axis == g.dim - 1 ? 1 : geom_stride(g, axis);
  *out = sub_rn(a.sel.field[i + st], a.sel.field[i]);
  return true;
}
template <class T, class K>
__device__ __forceinline__ bool sel_key_of(const Geom& g, const SelView<T>& a, int64_t b, int64_t t, K* key) {
  T v;
  if (!sel_raw(g, a, b, t, &v)) return false;
  if constexpr (sizeof(K) == 4) {
    *key = order_key(static_cast<float>(v));
  } else {
    double d = static_cast<double>(v);
    if (a.sel.center != nullptr) d = fabs(__dsub_rn(d, a.sel.center[b]));
    *key = order_key(d);
  }
  return true;
}

// One shared-memory count per distinct digit among the warp's active lanes (the lanes holding the
// same digit add together through their lowest lane): a field's items crowd into few digit values
// (the sign and exponent bits lead every key), and per-lane atomics on one address serialize.
__device__ __forceinline__ void count_digit(uint32_t* hist, uint32_t digit, bool take) {
  const unsigned active = __ballot_sync(0xffffffffu, take);
  if (!take) return;
  const unsigned same = __match_any_sync(active, digit);
  if ((threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&hist[digit], static_cast<uint32_t>(__popc(same)));
}

// The candidates of a selection: the keys that share the digits resolved before the candidates'
// pass (64-bit keys: two digits, the items within about 2^-10 of the statistic's binade position;
// 32-bit keys: one digit), written while that pass counts, which every later pass reads instead of
// the items. cap keys per element; a selection with more candidates reads the items in every pass
// (the count n keeps growing past cap, nothing is written there).
// The digit pass that writes the candidates (the later passes read them): the third for 64-bit
// keys; the second for 32-bit keys (after one digit: sign, exponent and two mantissa bits, a quarter
// binade of the values; measured 10 % faster on the 2-D benchmark's float32 selections). Building
// with EDAB_SEL_CAND32=0 leaves 32-bit selections without candidates.
#ifndef EDAB_SEL_CAND32
#define EDAB_SEL_CAND32 1
#endif
template <class K>
constexpr int kCandPass = sizeof(K) == 8 ? 2 : 1;

template <class K>
struct SelCand {
  K* keys;               // [B][cap]; nullptr: no candidates
  unsigned long long* n;  // [B]
  int64_t cap;
};
// Appends key k of the lanes with app set (the warp's 32 lanes call it together).
template <class K>
__device__ __forceinline__ void cand_append(const SelCand<K>& c, int64_t b, bool app, K k) {
  const unsigned m = __ballot_sync(0xffffffffu, app);
  if (!m) return;
  const int lane = threadIdx.x & 31;
  const int first = __ffs(m) - 1;
  unsigned long long base = 0;
  if (lane == first) base = atomicAdd(c.n + b, static_cast<unsigned long long>(__popc(m)));
  base = __shfl_sync(0xffffffffu, base, first);
  if (app) {
    const unsigned long long pos = base + static_cast<unsigned long long>(__popc(m & ((1u << lane) - 1u)));
    if (pos < static_cast<unsigned long long>(c.cap)) c.keys[b * c.cap + static_cast<int64_t>(pos)] = k;
  }
}

template <class K>
struct SelLeader {
  K prefix[2];
  unsigned long long rank[2];
  long long count;
  double gamma;
  int32_t live, same;
};

// The digit value of table tb (nb bins) that holds rank, and the rank inside it: one block-wide
// exclusive prefix sum over the bins (nb / TH consecutive bins per thread, or one) of TH threads.
template <int TH, class C>
__device__ __forceinline__ void rank_digit(const C* tb, int nb, unsigned long long rank,
                                           unsigned long long* warp_tot, int* bin_out,
                                           unsigned long long* rest_out) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = nb >= TH ? nb / TH : 1;
  const int first = tid * per, last = first < nb ? first + per : first;
  unsigned long long mine = 0;
  for (int j = first; j < last; ++j) mine += tb[j];
  unsigned long long incl = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned long long o = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += o;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  unsigned long long before = incl - mine;
  for (int w = 0; w < warp; ++w) before += warp_tot[w];
  if (rank >= before && rank < before + mine) {
    unsigned long long acc = before;
    for (int j = first; j < last; ++j) {
      const unsigned long long c = tb[j];
      if (rank < acc + c) {
        *bin_out = j;
        *rest_out = rank - acc;
        break;
      }
      acc += c;
    }
  }
  __syncthreads();
}

// NumPy's "linear" quantile: the index (n - 1) q, clamped at the ends, and its fraction.
__device__ __forceinline__ void linear_index(long long n, double q, long long* i, long long* j, double* frac) {
  const double pos = __dmul_rn(static_cast<double>(n - 1), q);
  if (pos >= static_cast<double>(n - 1)) {
    *i = *j = n - 1;
    *frac = __dadd_rn(pos, 1.0);
  } else if (pos < 0.0) {
    *i = *j = 0;
    *frac = pos;
  } else {
    const double whole = floor(pos);
    *i = static_cast<long long>(whole);
    *j = *i + 1;
    *frac = __dsub_rn(pos, whole);
  }
}
// NumPy's interpolation between neighbours: from the nearer end.
__device__ __forceinline__ double linear_between(double lo, double hi, double frac) {
  const double span = __dsub_rn(hi, lo);
  if (frac >= 0.5) return __dsub_rn(hi, __dmul_rn(span, __dsub_rn(1.0, frac)));
  return __dadd_rn(lo, __dmul_rn(span, frac));
}

template <class T, class K, int TH>
__global__ void __launch_bounds__(TH) select_cluster(Geom g, SelView<T> a, const int32_t* run, double q,
                                                          double* out, int64_t* count_out, SelCand<K> cand) {
  constexpr int kKeyBits = 8 * static_cast<int>(sizeof(K));
  constexpr int kDigits = (kKeyBits + kDigitBits - 1) / kDigitBits;
  extern __shared__ __align__(16) unsigned char sel_smem[];
  auto* table = reinterpret_cast<unsigned long long*>(sel_smem);                                  // leader: [2][bins]
  auto* local = reinterpret_cast<uint32_t*>(sel_smem + 2 * kDigitBins * sizeof(unsigned long long));  // [2][bins]
  __shared__ SelLeader<K> lead;
  __shared__ unsigned long long warp_tot[TH / 32];
  __shared__ int hit_bin;
  __shared__ unsigned long long hit_rest;
  cg::cluster_group cl = cg::this_cluster();
  const unsigned me = cl.block_rank();
  const unsigned ctas = cl.num_blocks();
  const int64_t b = blockIdx.y;
  if (run && !run[b]) return;  // every CTA of the cluster leaves here
  const int tid = threadIdx.x;
  const bool leader = me == 0;
  SelLeader<K>* L = cl.map_shared_rank(&lead, 0);
  unsigned long long* T0 = cl.map_shared_rank(table, 0);
  if (leader) {
    for (int i = tid; i < 2 * kDigitBins; i += TH) table[i] = 0ULL;
    if (tid == 0) {
      lead.prefix[0] = lead.prefix[1] = K(0);
      lead.live = 1;
      lead.same = 1;
      if (cand.keys) cand.n[b] = 0ULL;
    }
  }
  bool from_cand = false;
  int64_t n_it = a.items;
  for (int pass = 0; pass < kDigits; ++pass) {
    const int hi = kKeyBits - kDigitBits * pass;  // key bits at and above hi are resolved
    const int shift = hi > kDigitBits ? hi - kDigitBits : 0;
    const int width = hi - shift;
    const K dmask = static_cast<K>((K(1) << width) - K(1));
    for (int i = tid; i < 2 * kDigitBins; i += TH) local[i] = 0u;
    cl.sync();  // the leader's prefixes and cleared table are visible to the cluster
    const int live = L->live;
    if (!live) break;
    const bool two = pass > 0 && !L->same;
    const K p0 = L->prefix[0], p1 = L->prefix[1];
    if (pass == kCandPass<K> + 1 && cand.keys) {  // the candidates are complete (the barrier above)
      const unsigned long long nc = *reinterpret_cast<volatile unsigned long long*>(cand.n + b);
      from_cand = nc <= static_cast<unsigned long long>(cand.cap);
      if (from_cand) n_it = static_cast<int64_t>(nc);
    }
    const int64_t stride = static_cast<int64_t>(ctas) * TH;
    // the warp steps through the items together (count_digit is warp-collective)
    const int64_t t_end = (n_it + 31) / 32 * 32;
    for (int64_t t = static_cast<int64_t>(me) * TH + tid; t < t_end + stride; t += stride) {
      if (t - tid % 32 >= n_it) break;  // the warp's first item is past the end: the whole warp leaves
      K k = K(0);
      bool have;
      if (from_cand) {
        have = t < n_it;
        if (have) k = cand.keys[b * cand.cap + t];
      } else {
        have = t < a.items && sel_key_of<T, K>(g, a, b, t, &k);
      }
      const uint32_t digit = static_cast<uint32_t>((k >> shift) & dmask);
      const K top = pass == 0 ? K(0) : (k >> hi);
      count_digit(local, digit, have && (pass == 0 || top == (p0 >> hi)));
      if (two) count_digit(local + kDigitBins, digit, have && top == (p1 >> hi));
      if (pass == kCandPass<K> && cand.keys) cand_append(cand, b, have && (top == (p0 >> hi) || (two && top == (p1 >> hi))), k);
    }
    __syncthreads();
    const int bins = 1 << width;
    for (int i = tid; i < (two ? 2 : 1) * bins; i += TH) {
      const int r = i >= bins ? 1 : 0;
      const uint32_t c = local[r * kDigitBins + (i - r * bins)];
      if (c) atomicAdd(&T0[r * kDigitBins + (i - r * bins)], static_cast<unsigned long long>(c));
    }
    cl.sync();  // the cluster's counts are complete in the leader's table
    if (!leader) continue;
    if (pass == 0) {
      // the item count and the ranks of the statistic
      unsigned long long n = 0;
      for (int i = tid; i < bins; i += TH) n += table[i];
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) n += __shfl_xor_sync(0xffffffffu, n, d);
      if ((tid & 31) == 0) warp_tot[tid >> 5] = n;
      __syncthreads();
      if (tid == 0) {
        unsigned long long total = 0;
        for (int w = 0; w < TH / 32; ++w) total += warp_tot[w];
        lead.count = static_cast<long long>(total);
        lead.live = total > 0;
        if (total > 0) {
          if (q < 0) {
            lead.rank[0] = (total - 1) / 2;
            lead.rank[1] = total / 2;
          } else {
            long long i = 0, j = 0;
            linear_index(static_cast<long long>(total), q, &i, &j, &lead.gamma);
            lead.rank[0] = static_cast<unsigned long long>(i);
            lead.rank[1] = static_cast<unsigned long long>(j);
          }
        }
      }
      __syncthreads();
    }
    if (lead.live) {
      for (int r = 0; r < 2; ++r) {
        rank_digit<TH>(table + (two ? r : 0) * kDigitBins, bins, lead.rank[r], warp_tot, &hit_bin, &hit_rest);
        if (tid == 0) {
          lead.prefix[r] |= static_cast<K>(hit_bin) << shift;
          lead.rank[r] = hit_rest;
        }
        __syncthreads();
      }
      if (tid == 0) lead.same = lead.prefix[0] == lead.prefix[1];
    }
    for (int i = tid; i < 2 * kDigitBins; i += TH) table[i] = 0ULL;
  }
  cl.sync();  // no CTA reads the leader's shared memory after this
  if (leader && tid == 0) {
    if (!lead.live) {
      out[b] = d_nan();
      if (count_out) count_out[b] = 0;
    } else {
      const double v0 = key_value(lead.prefix[0]), v1 = key_value(lead.prefix[1]);
      out[b] = q < 0 ? ((lead.count & 1) ? v0 : __dmul_rn(__dadd_rn(v0, v1), 0.5)) : linear_between(v0, v1, lead.gamma);
      if (count_out) count_out[b] = lead.count;
    }
  }
}

// The small form: one CTA per element whose keys fit its shared memory. The keys are gathered densely with
// their smallest and largest; a histogram of 2048 bins over the range that is left finds the bin of both
// ranks (neighbours or the same), until few keys are left (ranked by comparing them all), the ranks part
// (the lower bin's largest key, the upper one's smallest) or a bin is one key. Bound by the gather's loads
// and the barriers: no digit of the keys is fixed, so one histogram mostly does. (In clusters a median of
// 4096 samples took three passes of 11 fixed digits, 25 us at 64 signals; 7 us here.)
constexpr int kSmallBins = 2048, kSmallList = 128, kSmallThreads = 1024;
constexpr int64_t kSmallItems = 32768;
constexpr size_t kSmallBytes = 216 * 1024;  // (the state takes 3 KB more)
template <class K>
struct SmallState {
  K lo, hi, v0, v1;
  unsigned n, r0, r1, d0, d1, listed;
  unsigned warp_tot[kSmallThreads / 32];
  K list[kSmallList];
};
__device__ __forceinline__ int bit_length(uint32_t v) { return 32 - __clz(static_cast<int>(v)); }
__device__ __forceinline__ int bit_length(uint64_t v) { return 64 - __clzll(static_cast<long long>(v)); }
template <class K>
__device__ __forceinline__ K warp_max_key(K v) {
  if constexpr (sizeof(K) == 4) return __reduce_max_sync(0xffffffffu, v);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    const K o = __shfl_xor_sync(0xffffffffu, v, d);
    v = o > v ? o : v;
  }
  return v;
}
__device__ __forceinline__ void shared_max(uint32_t* at, uint32_t v) { atomicMax(at, v); }
__device__ __forceinline__ void shared_max(uint64_t* at, uint64_t v) {
  atomicMax(reinterpret_cast<unsigned long long*>(at), static_cast<unsigned long long>(v));
}
// The element's largest of v over the CTA goes to *at (set before the last barrier).
template <class K>
__device__ __forceinline__ void block_max(K* at, K v) {
  v = warp_max_key(v);
  if ((threadIdx.x & 31) == 0) shared_max(at, v);
}

// dynamic shared memory: the keys [items], the bins
template <class T, class K>
__global__ void __launch_bounds__(kSmallThreads) select_small(Geom g, SelView<T> a, const int32_t* run, double q, double* out,
                                                     int64_t* count_out) {
  extern __shared__ __align__(16) unsigned char sel_smem[];
  __shared__ SmallState<K> st;
  const int64_t b = blockIdx.x;
  if (run && !run[b]) return;
  auto* bins = reinterpret_cast<uint32_t*>(sel_smem);
  K* keys = reinterpret_cast<K*>(bins + kSmallBins);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, TH = blockDim.x;
  if (tid == 0) {
    st.lo = st.hi = K(0);  // lo: the complements' largest, for now
    st.n = 0;
  }
  __syncthreads();
  {
    K top = K(0), bottom = K(0);
    const int32_t items = static_cast<int32_t>(a.items);
    for (int32_t t0 = 0; t0 < items; t0 += 4 * TH) {
      K k[4];
      bool have[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int32_t t = t0 + u * TH + tid;
        k[u] = K(0);
        have[u] = t < items && sel_key_of<T, K>(g, a, b, t, &k[u]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const unsigned m = __ballot_sync(0xffffffffu, have[u]);
        if (!m) continue;
        unsigned base = 0;
        if (lane == 0) base = atomicAdd(&st.n, static_cast<unsigned>(__popc(m)));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (have[u]) {
          keys[base + __popc(m & ((1u << lane) - 1u))] = k[u];
          top = k[u] > top ? k[u] : top;
          const K c = static_cast<K>(~k[u]);
          bottom = c > bottom ? c : bottom;
        }
      }
    }
    block_max(&st.hi, top);
    block_max(&st.lo, bottom);
  }
  __syncthreads();
  const int32_t n = static_cast<int32_t>(st.n);
  if (n == 0) {
    if (tid == 0) {
      out[b] = d_nan();
      if (count_out) count_out[b] = 0;
    }
    return;
  }
  K lo = static_cast<K>(~st.lo), hi = st.hi;
  unsigned r0, r1;
  double gamma = 0.0;
  if (q < 0) {
    r0 = static_cast<unsigned>((n - 1) / 2);
    r1 = static_cast<unsigned>(n / 2);
  } else {
    long long i = 0, j = 0;
    linear_index(n, q, &i, &j, &gamma);
    r0 = static_cast<unsigned>(i);
    r1 = static_cast<unsigned>(j);
  }
  unsigned left = static_cast<unsigned>(n);  // keys in [lo, hi]; the ranks count from lo's
  K v0 = K(0), v1 = K(0);
  for (;;) {  // (the range shrinks to a bin, 2^-10 of it or less, each time)
    if (lo == hi) {
      v0 = v1 = lo;
      break;
    }
    if (left <= kSmallList) {
      if (tid == 0) st.listed = 0;
      __syncthreads();
      for (int32_t i = tid; i < n; i += TH) {
        const K k = keys[i];
        if (k >= lo && k <= hi) st.list[atomicAdd(&st.listed, 1u)] = k;
      }
      __syncthreads();
      if (tid < static_cast<int>(left)) {
        const K mine = st.list[tid];
        unsigned rank = 0;
        for (int i = 0; i < static_cast<int>(left); ++i) {
          const K k = st.list[i];
          rank += (k < mine || (k == mine && i < tid)) ? 1u : 0u;
        }
        if (rank == r0) st.v0 = mine;
        if (rank == r1) st.v1 = mine;
      }
      __syncthreads();
      v0 = st.v0;
      v1 = st.v1;
      break;
    }
    const int shift = max(bit_length(static_cast<K>(hi - lo)) - 11, 0);
    for (int i = tid; i < kSmallBins; i += TH) bins[i] = 0u;
    if (tid == 0) st.v0 = st.v1 = K(0);
    __syncthreads();
    const int32_t end = (n + 31) / 32 * 32;
    for (int32_t i = tid; i < end; i += TH) {
      const K k = i < n ? keys[i] : K(0);
      count_digit(bins, static_cast<uint32_t>((k - lo) >> shift), i < n && k >= lo && k <= hi);
    }
    __syncthreads();
    // the bins of the ranks: exclusive prefix sums over kSmallBins / TH consecutive bins per thread
    const int per = kSmallBins / TH;
    unsigned mine = 0;
    for (int i = 0; i < per; ++i) mine += bins[tid * per + i];
    unsigned incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned o = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += o;
    }
    if (lane == 31) st.warp_tot[warp] = incl;
    __syncthreads();
    unsigned before = incl - mine;
    for (int w = 0; w < warp; ++w) before += st.warp_tot[w];
    for (int i = 0; i < per; ++i) {
      const unsigned c = bins[tid * per + i];
      if (r0 >= before && r0 < before + c) {
        st.d0 = static_cast<unsigned>(tid * per + i);
        st.r0 = r0 - before;
        st.listed = c;
      }
      if (r1 >= before && r1 < before + c) {
        st.d1 = static_cast<unsigned>(tid * per + i);
        st.r1 = r1 - before;
      }
      before += c;
    }
    __syncthreads();
    const K d0 = st.d0, d1 = st.d1;
    if (shift == 0) {
      v0 = lo + d0;
      v1 = lo + d1;
      break;
    }
    if (d0 != d1) {  // neighbours in rank: the lower bin's largest key and the upper one's smallest
      K low = K(0), up = K(0);
      for (int32_t i = tid; i < n; i += TH) {
        const K k = keys[i];
        if (k < lo || k > hi) continue;
        const K d = (k - lo) >> shift;
        if (d == d0) low = k > low ? k : low;
        if (d == d1) up = static_cast<K>(~k) > up ? static_cast<K>(~k) : up;
      }
      __syncwarp();
      block_max(&st.v0, low);
      block_max(&st.v1, up);
      __syncthreads();
      v0 = st.v0;
      v1 = static_cast<K>(~st.v1);
      break;
    }
    r0 = st.r0;
    r1 = st.r1;
    left = st.listed;
    lo = lo + (d0 << shift);
    if (hi - lo >= (K(1) << shift)) hi = lo + ((K(1) << shift) - 1);
    __syncthreads();  // the state is read before the next round writes it
  }
  if (tid == 0) {
    const double x0 = key_value(v0), x1 = key_value(v1);
    out[b] = q < 0 ? ((n & 1) ? x0 : __dmul_rn(__dadd_rn(x0, x1), 0.5)) : linear_between(x0, x1, gamma);
    if (count_out) count_out[b] = n;
  }
}

// The grid-wide form for batches of few, large elements (select):
// per digit, a launch over many CTAs per element (warp-aggregated shared-memory counts, flushed with
// one global atomic per digit value and CTA) whose last CTA finds the digit by the same block-wide
// prefix sum, the element's state in global memory between launches. (The pick was a launch of its
// own: 6 and 12 launches per selection instead of 3 and 6, and two memsets instead of one.)
template <class K>
struct SelGridState {
  K prefix[2];
  unsigned long long rank[2];
  long long count;
  double gamma;
  int16_t live, same;
  int32_t done;  // CTAs of the digit's launch that have added their counts
};

template <int KeyBits>
__device__ __forceinline__ void digit_of_pass(int pass, int* hi, int* shift, int* width) {
  *hi = KeyBits - kDigitBits * pass;
  *shift = *hi > kDigitBits ? *hi - kDigitBits : 0;
  *width = *hi - *shift;
}

// The digit of element b's ranks from its complete table tb (left zeroed), by one CTA.
template <class K>
__device__ __forceinline__ void grid_pick(int64_t b, SelGridState<K>* st, unsigned long long* tb, int32_t pass, double q,
                                          double* out, int64_t* count_out) {
  constexpr int kKeyBits = 8 * static_cast<int>(sizeof(K));
  constexpr int kDigits = (kKeyBits + kDigitBits - 1) / kDigitBits;
  __shared__ SelGridState<K> S;
  __shared__ unsigned long long warp_tot[kThreads / 32];
  __shared__ int hit_bin;
  __shared__ unsigned long long hit_rest;
  const int tid = threadIdx.x;
  int hi, shift, width;
  digit_of_pass<kKeyBits>(pass, &hi, &shift, &width);
  const int bins = 1 << width;
  if (pass == 0) {
    unsigned long long n = 0;
    for (int i = tid; i < bins; i += kThreads) n += tb[i];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) n += __shfl_xor_sync(0xffffffffu, n, d);
    if ((tid & 31) == 0) warp_tot[tid >> 5] = n;
    __syncthreads();
    if (tid == 0) {
      unsigned long long total = 0;
      for (int w = 0; w < kThreads / 32; ++w) total += warp_tot[w];
      S.prefix[0] = S.prefix[1] = K(0);
      S.same = 1;
      S.count = static_cast<long long>(total);
      S.live = total > 0;
      S.gamma = 0.0;
      if (q < 0) {
        S.rank[0] = total ? (total - 1) / 2 : 0;
        S.rank[1] = total / 2;
      } else if (total) {
        long long i = 0, j = 0;
        linear_index(static_cast<long long>(total), q, &i, &j, &S.gamma);
        S.rank[0] = static_cast<unsigned long long>(i);
        S.rank[1] = static_cast<unsigned long long>(j);
      }
    }
  } else if (tid == 0) {
    S = st[b];
  }
  __syncthreads();
  const bool two = pass > 0 && !S.same;
  if (S.live) {
    for (int r = 0; r < 2; ++r) {
      rank_digit<kThreads>(tb + (two ? r : 0) * kDigitBins, bins, S.rank[r], warp_tot, &hit_bin, &hit_rest);
      if (tid == 0) {
        S.prefix[r] |= static_cast<K>(hit_bin) << shift;
        S.rank[r] = hit_rest;
      }
      __syncthreads();
    }
  }
  for (int i = tid; i < 2 * kDigitBins; i += kThreads) tb[i] = 0ULL;  // clean for the next digit
  if (tid == 0) {
    S.same = S.prefix[0] == S.prefix[1];
    S.done = 0;
    st[b] = S;
    if (!S.live) {  // no item: no later digit either
      out[b] = d_nan();
      if (count_out) count_out[b] = 0;
    } else {
      if (pass == kDigits - 1) {
        const double v0 = key_value(S.prefix[0]), v1 = key_value(S.prefix[1]);
        out[b] = q < 0 ? ((S.count & 1) ? v0 : __dmul_rn(__dadd_rn(v0, v1), 0.5)) : linear_between(v0, v1, S.gamma);
        if (count_out) count_out[b] = S.count;
      }
    }
  }
}

template <class T, class K>
__global__ void __launch_bounds__(kThreads) select_grid_count(Geom g, SelView<T> a, const int32_t* run,
                                                             SelGridState<K>* st,
                                                             unsigned long long* table, int32_t pass,
                                                             SelCand<K> cand, double q, double* out, int64_t* count_out) {
  __shared__ uint32_t local[2 * kDigitBins];
  __shared__ int32_t last_s;
  const int64_t b = blockIdx.y;
  if (run && !run[b]) return;
  bool two = false;
  K p0 = K(0), p1 = K(0);
  if (pass > 0) {
    if (!st[b].live) return;
    two = !st[b].same;
    p0 = st[b].prefix[0];
    p1 = st[b].prefix[1];
  }
  int hi, shift, width;
  digit_of_pass<8 * static_cast<int>(sizeof(K))>(pass, &hi, &shift, &width);
  const K dmask = static_cast<K>((K(1) << width) - K(1));
  const int tid = threadIdx.x;
  for (int i = tid; i < 2 * kDigitBins; i += kThreads) local[i] = 0u;
  __syncthreads();
  // after the candidates pass, its candidates (when they fit) instead of the items
  bool from_cand = false;
  int64_t n_it = a.items;
  if (pass > kCandPass<K> && cand.keys) {
    const unsigned long long nc = cand.n[b];
    from_cand = nc <= static_cast<unsigned long long>(cand.cap);
    if (from_cand) n_it = static_cast<int64_t>(nc);
  }
  const int64_t stride = static_cast<int64_t>(gridDim.x) * kThreads;
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * kThreads + tid;; t += stride) {
    if (t - tid % 32 >= n_it) break;  // the warp's first item is past the end
    K k = K(0);
    bool have;
    if (from_cand) {
      have = t < n_it;
      if (have) k = cand.keys[b * cand.cap + t];
    } else {
      have = t < a.items && sel_key_of<T, K>(g, a, b, t, &k);
    }
    const uint32_t digit = static_cast<uint32_t>((k >> shift) & dmask);
    const K top = pass == 0 ? K(0) : (k >> hi);
    count_digit(local, digit, have && (pass == 0 || top == (p0 >> hi)));
    if (two) count_digit(local + kDigitBins, digit, have && top == (p1 >> hi));
    if (pass == kCandPass<K> && cand.keys) cand_append(cand, b, have && (top == (p0 >> hi) || (two && top == (p1 >> hi))), k);
  }
  __syncthreads();
  const int bins = 1 << width;
  unsigned long long* tb = table + static_cast<int64_t>(b) * 2 * kDigitBins;
  for (int i = tid; i < (two ? 2 : 1) * bins; i += kThreads) {
    const int r = i >= bins ? 1 : 0;
    const uint32_t c = local[r * kDigitBins + (i - r * bins)];
    if (c) atomicAdd(&tb[r * kDigitBins + (i - r * bins)], static_cast<unsigned long long>(c));
  }
  // the element's last CTA to get here has the whole table: it picks the digit
  __threadfence();
  __syncthreads();
  if (tid == 0) last_s = atomicAdd(&st[b].done, 1) == static_cast<int32_t>(gridDim.x) - 1;
  __syncthreads();
  if (!last_s) return;
  __threadfence();
  grid_pick<K>(b, st, tb, pass, q, out, count_out);
}

// The split form for many items (select): one pass over the items instead of one per digit. A sample of
// the items brackets the statistic: the keys lo and hi of the sample about 5 standard deviations of
// its rank to either side. The pass counts the items below lo and lists those in [lo, hi] (about 8 %);
// when the wanted ranks lie in the list and it fits, a radix selection of the list is the answer, else
// (a bracket that missed, or more ties than the list holds) the element is handed to the other forms.
// Exact whatever the sample: the ranks are counted, not estimated. Bound by reading the items once
// (a 512 x 512 element's median of differences: 230 us per 64 images before, the digit passes' counting).
template <class K>
struct SplitState {
  K lo, hi;
  unsigned long long less, total, listed;
};
static_assert(sizeof(SplitState<uint64_t>) <= sizeof(SelGridState<uint64_t>), "the split's states lie in the grid form's");

constexpr int kSplitSample = 4096, kSplitThreads = 1024;

template <class T, class K>
__global__ void __launch_bounds__(kSplitThreads) split_pivots(Geom g, SelView<T> a, const int32_t* run, double q,
                                                             SplitState<K>* st) {
  __shared__ K keys[kSplitSample];
  __shared__ int32_t found_s;
  const int64_t b = blockIdx.x;
  if (run && !run[b]) return;
  if (threadIdx.x == 0) found_s = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < kSplitSample; i += kSplitThreads) {
    // pseudo-random items (splitmix64 of the draw): a regular stride could fall in step with the field
    uint64_t z = 0x9e3779b97f4a7c15ULL * static_cast<uint64_t>(i + 1);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    z ^= z >> 31;
    const int64_t t = static_cast<int64_t>(__umul64hi(z, static_cast<uint64_t>(a.items)));
    K k = K(0);
    const bool have = sel_key_of<T, K>(g, a, b, t, &k);
    keys[i] = have ? k : ~K(0);
    const unsigned m = __ballot_sync(0xffffffffu, have);
    if ((threadIdx.x & 31) == 0) atomicAdd(&found_s, __popc(m));
  }
  for (int size = 2; size <= kSplitSample; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      __syncthreads();
      for (int t = threadIdx.x; t < kSplitSample / 2; t += kSplitThreads) {
        const int i = 2 * t - (t & (stride - 1)), j = i + stride;
        const K x = keys[i], y = keys[j];
        if ((x > y) == ((i & size) == 0)) {
          keys[i] = y;
          keys[j] = x;
        }
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int m = found_s;
    const double rho = q < 0 ? 0.5 : q, at = rho * (m - 1);
    const double spread = 5.0 * sqrt(rho * (1.0 - rho) * m) + 2.0;
    const int lo = static_cast<int>(floor(at - spread)), hi = static_cast<int>(ceil(at + spread));
    SplitState<K> s;
    s.lo = lo < 0 ? K(0) : keys[lo];
    s.hi = hi >= m ? ~K(0) : keys[hi];
    s.less = s.total = s.listed = 0ULL;
    st[b] = s;
  }
}

// A warp's keys for the list, written 32 at a time.
template <class K>
__device__ __forceinline__ void list_keys(K* queue, int& held, bool listed, K key, const SelCand<K>& cand,
                                          SplitState<K>* st, int64_t b) {
  const int lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(0xffffffffu, listed);
  if (m == 0u) return;
  if (listed) queue[held + __popc(m & ((1u << lane) - 1u))] = key;
  held += __popc(m);
  __syncwarp();
  if (held >= 32) {
    held -= 32;
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(&st[b].listed, 32ULL);
    at = __shfl_sync(0xffffffffu, at, 0) + lane;
    if (at < static_cast<unsigned long long>(cand.cap)) cand.keys[b * cand.cap + static_cast<int64_t>(at)] = queue[held + lane];
    __syncwarp();
  }
}

template <class T, class K>
__global__ void __launch_bounds__(kThreads) split_count(Geom g, SelView<T> a, const int32_t* run, SplitState<K>* st,
                                                       SelCand<K> cand) {
  constexpr int W = 16 / static_cast<int>(sizeof(T));  // samples of a step of a thread: of one row
  __shared__ K queue_s[kThreads / 32][64];
  __shared__ unsigned long long less_s, total_s;
  const int64_t b = blockIdx.y;
  if (run && !run[b]) return;
  if (threadIdx.x == 0) less_s = total_s = 0ULL;
  __syncthreads();
  const K lo = st[b].lo, hi = st[b].hi;
  const bool diff = a.sel.src == SelSrc::kDiff;
  const T* f = a.sel.field + b * g.field;
  const uint8_t* mask = !diff && a.sel.mask ? a.sel.mask + b * g.field : nullptr;
  const double center = a.sel.center ? a.sel.center[b] : 0.0;
  const int32_t nl = elem_len(g, b);
  const uint32_t units = static_cast<uint32_t>(g.field / W);  // per axis
  K* queue = queue_s[threadIdx.x >> 5];
  int held = 0;
  uint32_t less = 0, total = 0;
  const uint32_t step = gridDim.x * kThreads;
  for (int ax = 0; ax < (diff ? a.naxes : 1); ++ax) {
    const int axis = ax == 0 ? a.ax[0] : (ax == 1 ? a.ax[1] : a.ax[2]);
    const bool last = axis == g.dim - 1;
    const int64_t st_ax = last ? 1 : geom_stride(g, axis);
    const int32_t n_ax = elem_n(g, b, axis);
    for (uint32_t u = blockIdx.x * kThreads + threadIdx.x; u - (threadIdx.x & 31) < units; u += step) {
      const int64_t v = static_cast<int64_t>(u) * W;
      int32_t room = 0;  // samples of the step that are items
      T x[W];
      if (u < units) {
        const int32_t col = static_cast<int32_t>(pitch_col(g, v));
        room = min(W, nl - (diff && last ? 1 : 0) - col);
        if (diff && !last && room > 0 && coord_of(g, v, axis) >= n_ax - 1) room = 0;
        if (room > 0) {
          const int4 p = *reinterpret_cast<const int4*>(f + v);
          memcpy(x, &p, 16);
          if (diff) {
            T y[W];
            if (last) {
#pragma unroll
              for (int k = 0; k + 1 < W; ++k) y[k] = x[k + 1];
              y[W - 1] = room == W ? f[v + W] : T(0);
            } else {
              const int4 r = *reinterpret_cast<const int4*>(f + v + st_ax);
              memcpy(y, &r, 16);
            }
#pragma unroll
            for (int k = 0; k < W; ++k) x[k] = sub_rn(y[k], x[k]);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < W; ++k) {
        bool have = k < room;
        if (have && mask) have = (mask[v + k] & a.sel.bits) != 0;
        K key = K(0);
        if constexpr (sizeof(K) == 4) {
          key = order_key(static_cast<float>(x[k]));
        } else {
          double d = static_cast<double>(x[k]);
          if (a.sel.center) d = fabs(__dsub_rn(d, center));
          key = order_key(d);
        }
        total += have;
        less += have && key < lo;
        list_keys(queue, held, have && key >= lo && key <= hi, key, cand, st, b);
      }
    }
  }
  const int lane = threadIdx.x & 31;
  if (held > 0) {
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(&st[b].listed, static_cast<unsigned long long>(held));
    at = __shfl_sync(0xffffffffu, at, 0) + lane;
    if (lane < held && at < static_cast<unsigned long long>(cand.cap)) cand.keys[b * cand.cap + static_cast<int64_t>(at)] = queue[lane];
  }
  less = __reduce_add_sync(0xffffffffu, less);
  total = __reduce_add_sync(0xffffffffu, total);
  if (lane == 0) {
    atomicAdd(&less_s, static_cast<unsigned long long>(less));
    atomicAdd(&total_s, static_cast<unsigned long long>(total));
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (less_s) atomicAdd(&st[b].less, less_s);
    if (total_s) atomicAdd(&st[b].total, total_s);
  }
}

template <class K>
__global__ void __launch_bounds__(kSplitThreads) split_finish(const int32_t* run, const SplitState<K>* st, SelCand<K> cand,
                                                             double q, double* out, int64_t* count_out, int32_t* mask) {
  constexpr int kKeyBits = 8 * static_cast<int>(sizeof(K));
  constexpr int kDigits = (kKeyBits + kDigitBits - 1) / kDigitBits;
  __shared__ uint32_t local[2 * kDigitBins];
  __shared__ unsigned long long warp_tot[kSplitThreads / 32];
  __shared__ int hit_bin;
  __shared__ unsigned long long hit_rest;
  const int64_t b = blockIdx.x;
  const int tid = threadIdx.x;
  if (run && !run[b]) {
    if (tid == 0) mask[b] = 0;
    return;
  }
  const SplitState<K> s = st[b];
  unsigned long long rank[2] = {0, 0};
  double gamma = 0.0;
  if (s.total > 0) {
    if (q < 0) {
      rank[0] = (s.total - 1) / 2;
      rank[1] = s.total / 2;
    } else {
      long long i = 0, j = 0;
      linear_index(static_cast<long long>(s.total), q, &i, &j, &gamma);
      rank[0] = static_cast<unsigned long long>(i);
      rank[1] = static_cast<unsigned long long>(j);
    }
  }
  const bool tie = s.lo == s.hi;  // every listed key is the same
  const bool ok = s.total == 0 || (rank[0] >= s.less && rank[1] < s.less + s.listed &&
                                   (tie || s.listed <= static_cast<unsigned long long>(cand.cap)));
  if (tid == 0) mask[b] = ok ? 0 : 1;
  if (!ok) return;
  if (s.total == 0) {
    if (tid == 0) {
      out[b] = d_nan();
      if (count_out) count_out[b] = 0;
    }
    return;
  }
  K prefix[2] = {K(0), K(0)};
  if (tie) {
    prefix[0] = prefix[1] = s.lo;
  } else {
    rank[0] -= s.less;
    rank[1] -= s.less;
    const K* keys = cand.keys + b * cand.cap;
    const int64_t n = static_cast<int64_t>(s.listed);
    for (int pass = 0; pass < kDigits; ++pass) {
      int hi, shift, width;
      digit_of_pass<kKeyBits>(pass, &hi, &shift, &width);
      const K dmask = static_cast<K>((K(1) << width) - K(1));
      const bool two = pass > 0 && prefix[0] != prefix[1];
      for (int i = tid; i < 2 * kDigitBins; i += kSplitThreads) local[i] = 0u;
      __syncthreads();
      for (int64_t t = tid; t - (tid & 31) < n; t += kSplitThreads) {
        const bool have = t < n;
        const K k = have ? keys[t] : K(0);
        const uint32_t digit = static_cast<uint32_t>((k >> shift) & dmask);
        const K top = pass == 0 ? K(0) : (k >> hi);
        count_digit(local, digit, have && (pass == 0 || top == (prefix[0] >> hi)));
        if (two) count_digit(local + kDigitBins, digit, have && top == (prefix[1] >> hi));
      }
      __syncthreads();
      const int bins = 1 << width;
      for (int r = 0; r < 2; ++r) {
        rank_digit<kSplitThreads>(local + (two ? r : 0) * kDigitBins, bins, rank[r], warp_tot, &hit_bin, &hit_rest);
        prefix[r] |= static_cast<K>(hit_bin) << shift;
        rank[r] = hit_rest;
        __syncthreads();
      }
    }
  }
  if (tid == 0) {
    const double v0 = key_value(prefix[0]), v1 = key_value(prefix[1]);
    out[b] = q < 0 ? ((s.total & 1) ? v0 : __dmul_rn(__dadd_rn(v0, v1), 0.5)) : linear_between(v0, v1, gamma);
    if (count_out) count_out[b] = static_cast<int64_t>(s.total);
  }
}

size_t align256(size_t v) { return (v + 255) / 256 * 256; }

}  // namespace

size_t totals_scratch_bytes(const Geom& g) {
  return align256(static_cast<size_t>(g.batch * g.rows) * sizeof(RowPartial));
}

template <class T>
void field_totals(cudaStream_t s, const Geom& g, const T* f, double* energy, double* amax, uint64_t* nonfinite,
                  void* scratch) {
  auto* rows = static_cast<RowPartial*>(scratch);
  const int64_t total = g.batch * g.rows;
  if (g.n_last > kMaxSteps * 1024) throw std::invalid_argument("edab: a row is too long for the energy sums");
  const bool per_row = g.n_last > 1024;
  const int64_t blocks = std::clamp<int64_t>(per_row ? total : (total + (kRowThreads<T> / 32) - 1) / (kRowThreads<T> / 32), 1, int64_t{1} << 20);
  enqueue(row_partials<T>, static_cast<unsigned>(blocks), kRowThreads<T>, 0, s, f, g, rows, nonfinite, per_row);
  const unsigned eb = static_cast<unsigned>(std::clamp<int64_t>(g.batch, 1, 65535));
  enqueue(element_totals, eb, kThreads, 0, s, g, rows, energy, amax);
}

constexpr int64_t kMaskKeys = 32;
// Candidate keys per element: a quarter of the largest selection's items (the differences along
// every axis), at least 64.
int64_t cand_cap(const Geom& g) { return std::max<int64_t>(64, static_cast<int64_t>(g.dim) * g.field / 4 / 32 * 32); }

// scratch: the grid form's states and count tables, then the candidates' counts and keys
size_t select_scratch_bytes(const Geom& g) {
  const size_t B = static_cast<size_t>(g.batch);
  return align256(B * sizeof(SelGridState<uint64_t>)) + align256(B * 2 * kDigitBins * sizeof(unsigned long long)) +
         align256(B * sizeof(unsigned long long)) + align256(B * static_cast<size_t>(cand_cap(g)) * sizeof(uint64_t));
}

template <class K>
SelCand<K> cand_of(const Geom& g, void* scratch) {
  const size_t B = static_cast<size_t>(g.batch);
  char* p = static_cast<char*>(scratch) + align256(B * sizeof(SelGridState<uint64_t>)) +
            align256(B * 2 * kDigitBins * sizeof(unsigned long long));
  SelCand<K> c;
  c.n = reinterpret_cast<unsigned long long*>(p);
  c.keys = reinterpret_cast<K*>(p + align256(B * sizeof(unsigned long long)));
  c.cap = cand_cap(g) - kMaskKeys;
  return c;
}
// The split selection's run mask of the elements that it hands on, behind the candidate lists (each of
// which is kMaskKeys shorter than its share of the scratch).
template <class K>
int32_t* split_mask(const Geom& g, const SelCand<K>& c) {
  return reinterpret_cast<int32_t*>(c.keys + static_cast<size_t>(g.batch) * c.cap);
}

// The grid-wide form: a launch per digit (scratch: the states, then the [B][2][bins] count tables,
// zeroed here and left zeroed by every pick).
template <class T, class K>
void select_grid(cudaStream_t s, const Geom& g, const SelView<T>& a, double q, const int32_t* run, double* out,
                 int64_t* count, void* scratch, int sms) {
  constexpr int kDigits = (8 * static_cast<int>(sizeof(K)) + kDigitBits - 1) / kDigitBits;
  auto* st = static_cast<SelGridState<K>*>(scratch);
  auto* table = reinterpret_cast<unsigned long long*>(static_cast<char*>(scratch) +
                                                       align256(static_cast<size_t>(g.batch) * sizeof(SelGridState<uint64_t>)));
  // the states, the tables and the candidates' counts lie one after the other
  const SelCand<K> cand = (sizeof(K) == 8 || EDAB_SEL_CAND32) ? cand_of<K>(g, scratch) : SelCand<K>{};
  const size_t clear = static_cast<size_t>(reinterpret_cast<char*>(cand_of<K>(g, scratch).n) - static_cast<char*>(scratch)) +
                       static_cast<size_t>(g.batch) * sizeof(unsigned long long);
  enqueue_zero(scratch, clear, s);
  // CTAs per element: 64 items per thread, and for small batches enough CTAs for 8 per SM (at
  // least 4 items per thread)
  const int64_t by_items = (a.items + int64_t{kThreads} * 64 - 1) / (int64_t{kThreads} * 64);
  const int64_t fill = std::min<int64_t>((int64_t{8} * sms + g.batch - 1) / g.batch,
                                         std::max<int64_t>(1, a.items / (int64_t{kThreads} * 4)));
  const unsigned ctas = static_cast<unsigned>(std::clamp<int64_t>(std::max(by_items, fill), 1, 1024));
  for (int pass = 0; pass < kDigits; ++pass) {
    enqueue(select_grid_count<T, K>, dim3(ctas, static_cast<unsigned>(g.batch)), kThreads, 0, s, g, a, run, st, table, pass,
                                                                                          cand, q, out, count);
  }
}

// The split form of a selection; returns the run mask of the elements that it hands on.
template <class T, class K>
const int32_t* select_split(cudaStream_t s, const Geom& g, const SelView<T>& a, double q, const int32_t* run, double* out,
                            int64_t* count, void* scratch, int sms) {
  const SelCand<K> cand = cand_of<K>(g, scratch);
  auto* st = static_cast<SplitState<K>*>(scratch);
  int32_t* mask = split_mask(g, cand);
  const unsigned B = static_cast<unsigned>(g.batch);
  enqueue(split_pivots<T, K>, B, kSplitThreads, 0, s, g, a, run, q, st);
  // 8 CTAs per SM in all, at least 16 items per thread
  const int64_t fill = (int64_t{8} * sms + g.batch - 1) / g.batch;
  const unsigned ctas = static_cast<unsigned>(std::clamp<int64_t>(fill, 1, std::max<int64_t>(1, a.items / (int64_t{kThreads} * 16))));
  enqueue(split_count<T, K>, dim3(ctas, B), kThreads, 0, s, g, a, run, st, cand);
  enqueue(split_finish<K>, B, kSplitThreads, 0, s, run, st, cand, q, out, count, mask);
  return mask;
}

template <class T>
void select(cudaStream_t s, const Geom& g, const Sel<T>& sel, double q, const int32_t* run, double* out,
            int64_t* count, void* scratch) {
  SelView<T> a{};
  a.sel = sel;
  if (sel.src == SelSrc::kField) {
    a.naxes = 1;
    a.items = g.field;
  } else {
    for (int ax = 0; ax < g.dim; ++ax) {
      if (sel.axes & (1u << ax)) a.ax[a.naxes++] = ax;
    }
    a.items = static_cast<int64_t>(a.naxes) * g.field;
  }
  if (g.batch > 65535) throw std::invalid_argument("edab: select batch too large");
  int sms = 148;
  {
    int dev = 0;
    EDAB_CUDA(cudaGetDevice(&dev));
    EDAB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  }
  // Many items: the split form first, then the others for the elements that it hands on.
  if (scratch && a.items >= kSplitItems && a.items <= kSplitMost && g.batch >= kSplitBatch &&
      a.items * g.batch >= kSplitTotal) {
    bool done = false;
    if constexpr (std::is_same_v<T, float>) {
      if (sel.center == nullptr) {
        run = select_split<T, uint32_t>(s, g, a, q, run, out, count, scratch, sms);
        done = true;
      }
    }
    if (!done) run = select_split<T, uint64_t>(s, g, a, q, run, out, count, scratch, sms);
  }
  // Elements whose keys fit one CTA's shared memory: the small form (medians of 2048 samples 5.8 us, of up to
  // 8192 in batches 7 to 12 us, of 20 011 float64 samples 21 us; as clusters 12.5, 25 to 33 and 30 us).
  const bool narrow = std::is_same_v<T, float> && sel.center == nullptr;  // 32-bit keys
  const size_t small = static_cast<size_t>(a.items) * (narrow ? 4 : 8) + kSmallBins * sizeof(uint32_t);
  if (a.items <= kSmallItems && small <= kSmallBytes) {
    const unsigned th = a.items > 4096 ? 1024u : a.items > 2048 ? 512u : a.items > 512 ? 256u : 128u;
    const auto go = [&](auto kernel) {
      once_on_device(reinterpret_cast<const void*>(kernel), [&] {
        EDAB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmallBytes)));
      });
      enqueue(kernel, static_cast<unsigned>(g.batch), th, small, s, g, a, run, q, out, count);
    };
    if constexpr (std::is_same_v<T, float>) {
      if (narrow) {
        go(select_small<T, uint32_t>);
        return;
      }
    }
    go(select_small<T, uint64_t>);
    return;
  }
  // Otherwise clusters (one launch): of 256-thread CTAs when the batch fills the GPU with them, else of
  // 1024-thread CTAs while an element has at most 8 items for each of their threads; larger elements of
  // small batches take the grid-wide form, a launch per digit over many CTAs (133 000 items: 26 us for
  // 32-bit keys, against 54 us in one cluster).
  const bool many = g.batch * kSelClusterMax >= 2 * static_cast<int64_t>(sms);
  if (!kSelClusters || (!many && a.items > int64_t{kSelClusterMax} * kSelWide * 8)) {
    if (!scratch) throw std::logic_error("edab: the grid-wide selection needs its scratch");
    if constexpr (std::is_same_v<T, float>) {
      if (sel.center == nullptr) {
        select_grid<T, uint32_t>(s, g, a, q, run, out, count, scratch, sms);
        return;
      }
    }
    select_grid<T, uint64_t>(s, g, a, q, run, out, count, scratch, sms);
    return;
  }
  // CTAs per element: about 16 items per thread (4 in a small batch), up to a cluster of 8
  const int64_t per_cta = many ? int64_t{kThreads} * 16 : int64_t{kSelWide} * 4;
  const unsigned ctas = static_cast<unsigned>(std::clamp<int64_t>((a.items + per_cta - 1) / per_cta, 1, kSelClusterMax));
  const auto launch = [&](auto kernel, auto cand) {
    once_on_device(reinterpret_cast<const void*>(kernel), [&] {
      EDAB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSelSmem)));
    });
    enqueue_clusters(ctas, kernel, dim3(ctas, static_cast<unsigned>(g.batch)), many ? kThreads : kSelWide, kSelSmem, s, g, a, run,
                     q, out, count, cand);
  };
  if constexpr (std::is_same_v<T, float>) {
    if (sel.center == nullptr) {
      const SelCand<uint32_t> cand = (EDAB_SEL_CAND32 && scratch) ? cand_of<uint32_t>(g, scratch) : SelCand<uint32_t>{};
      if (many) launch(select_cluster<T, uint32_t, kThreads>, cand);
      else launch(select_cluster<T, uint32_t, kSelWide>, cand);
      return;
    }
  }
  const SelCand<uint64_t> cand = scratch ? cand_of<uint64_t>(g, scratch) : SelCand<uint64_t>{};
  if (many) launch(select_cluster<T, uint64_t, kThreads>, cand);
  else launch(select_cluster<T, uint64_t, kSelWide>, cand);
}

// ---------------------------------------------------------------------------------------------
// Significant extrema (cpp/src/method/stats_fields.cu:1-14, 182-331 of eda-cuda): the peaks of r
// and -r along every line as scipy.signal.find_peaks defines them, with topographic prominence
// >= tau at the peak. A CTA stages P lines in shared memory with their 32-sample block minima and
// maxima; the thread of a run start owns a peak and walks each side over samples, then whole
// blocks (entering a block only where it holds the side's end).
namespace {

constexpr int kBlk = 32;

// A drop from hi to lo is significant when fl64(hi - lo) >= tau: the difference of the two samples
// in double, rounded once. (For float32 samples the float difference decides the same way except on
// an exact tie with tau; the double difference settles every case with one rule.)
template <class T>
__device__ __forceinline__ bool drops(T hi, T lo, T tau) {
  return __dsub_rn(static_cast<double>(hi), static_cast<double>(lo)) >= static_cast<double>(tau);
}

// Sample k of a staged line: one pad word after every 32 samples (the lanes of a warp scanning
// consecutive blocks hit distinct banks).
template <class T>
__device__ __forceinline__ T xs(const T* x, int32_t k) {
  return x[k + (k >> 5)];
}

// Samples k = from, from + Dir, .. to of a staged line against the peak value v: 1 when a sample
// lies a significant drop away from v before any sample lies beyond v (above a maximum, below a
// minimum, or NaN), 0 when a sample beyond v comes first, -1 when the range holds neither.
template <bool Max, int Dir, class T, class X>
__device__ __forceinline__ int walk_samples(const X& x, int32_t from, int32_t to, T v, T tau) {
  for (int32_t k = from; (to - k) * Dir >= 0; k += Dir) {
    const T u = x(k);
    if (Max ? !(u <= v) : !(u >= v)) return 0;
    if (Max ? drops(v, u, tau) : drops(u, v, tau)) return 1;
  }
  return -1;
}

// Whether the side of the peak at p (value v) in direction Dir falls by tau before it rises beyond
// v (the line end counts as no fall): SciPy's prominence base on that side is at least tau below
// the peak. The rest of the peak's 32-sample block is walked sample by sample; then every block is
// judged by its extremes (bext: the extreme towards "beyond", bnear: the other one): a block with
// nothing beyond v either holds a significant drop or is passed over; the first block with a sample
// beyond v is walked and decides.
template <bool Max, int Dir, class T, class X>
__device__ bool side_falls(const X& x, int32_t n, int32_t p, T v, T tau, const T* bext, const T* bnear) {
  const int32_t blocks = (n + kBlk - 1) / kBlk;
  int32_t c = p / kBlk;
  const int32_t edge = Dir > 0 ? min(c * kBlk + kBlk - 1, n - 1) : c * kBlk;
  if ((edge - p) * Dir > 0) {
    const int verdict = walk_samples<Max, Dir, T>(x, p + Dir, edge, v, tau);
    if (verdict >= 0) return verdict == 1;
  }
  for (c += Dir; c >= 0 && c < blocks; c += Dir) {
    const T e = bext[c];
    if (Max ? !(e <= v) : !(e >= v)) {
      const int32_t first = c * kBlk, last = min(first + kBlk - 1, n - 1);
      return walk_samples<Max, Dir, T>(x, Dir > 0 ? first : last, Dir > 0 ? last : first, v, tau) == 1;
    }
    if (Max ? drops(v, bnear[c], tau) : drops(bnear[c], v, tau)) return true;
  }
  return false;
}

// The run of samples equal to x(s) from s, when s starts one (x(s - 1) differs): its middle sample as
// the peak pk, and 1 for a maximum, 2 for a minimum, 0 for neither.
template <class T, class X>
__device__ __forceinline__ int peak_at(const X& x, int32_t n, int32_t nb, int32_t s, const T* bmin, const T* bmax,
                                       int32_t* pk) {
  const T cur = x(s), prev = x(s - 1);
  if (!(prev < cur || prev > cur)) return 0;
  int32_t e;
  const int32_t lim = min((s / kBlk) * kBlk + kBlk - 1, n - 1);
  int32_t k = s + 1;
  while (k <= lim && x(k) == cur) ++k;
  if (k <= lim || k >= n) {
    e = k - 1;
  } else {
    e = n - 1;
    for (int32_t c = k / kBlk; c < nb; ++c) {
      if (bmin[c] == cur && bmax[c] == cur) continue;
      k = c * kBlk;
      while (x(k) == cur) ++k;
      e = k - 1;
      break;
    }
  }
  if (e > n - 2) return 0;
  const T nxt = x(e + 1);
  *pk = (s + e) / 2;
  return prev < cur && nxt < cur ? 1 : (prev > cur && nxt > cur ? 2 : 0);
}

// Whether the peak pk (kind 1: maximum, 2: minimum) falls by tau on both sides.
template <class T, class X>
__device__ __forceinline__ bool peak_counts(const X& x, int32_t n, int32_t pk, int kind, T tau, const T* bmin,
                                            const T* bmax) {
  const T v = x(pk);
  return kind == 1 ? side_falls<true, -1>(x, n, pk, v, tau, bmax, bmin) && side_falls<true, 1>(x, n, pk, v, tau, bmax, bmin)
                   : side_falls<false, -1>(x, n, pk, v, tau, bmin, bmax) && side_falls<false, 1>(x, n, pk, v, tau, bmin, bmax);
}

// A warp's peaks waiting to be judged. Testing a sample for a peak is short and the same for every
// lane; walking a peak's sides is long, and only a third of the samples of a noisy line are peaks.
// So the lanes that find peaks push them here, and the warp judges 32 at a time, every lane one.
constexpr int kPeakQueue = 64;
template <class Judge>
__device__ __forceinline__ void push_peaks(uint32_t* queue, int& held, bool found, uint32_t entry, const Judge& judge) {
  const int lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(0xffffffffu, found);
  if (found) queue[held + __popc(m & ((1u << lane) - 1u))] = entry;
  held += __popc(m);
  __syncwarp();
  if (held >= 32) {
    held -= 32;
    judge(queue[held + lane]);
    __syncwarp();
  }
}
template <class Judge>
__device__ __forceinline__ void drain_peaks(const uint32_t* queue, int held, const Judge& judge) {
  if (static_cast<int>(threadIdx.x & 31) < held) judge(queue[threadIdx.x & 31]);
}

__device__ __forceinline__ void copy_async(float* smem, const float* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(smem))),
               "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void copy_async(double* smem, const double* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(smem))),
               "l"(gmem)
               : "memory");
}

// The inner samples [first, end) of a line of n that part blockIdx.x % parts of it takes.
__device__ __forceinline__ void part_of_line(int32_t n, int32_t* first, int32_t* end, int32_t parts, int32_t part) {
  const int32_t per = ((n - 2 + parts - 1) / parts + 31) & ~31;
  *first = 1 + part * per;
  *end = min(*first + per, n - 1);
}

// Staged lines: P lines of LX words (sample k at k + k / 32; LX odd, so lanes on consecutive lines
// hit distinct banks), then the block minima and maxima. Rows: a warp takes 32 consecutive samples of
// a line; column panels: its lanes cover the panel's columns (whole sectors of flags and tau). What
// bounds it: the walks of the peaks' sides (shared-memory latency, lanes with walks of different
// lengths); staging is asynchronous, all of a thread's samples in flight at once.
template <class T>
__global__ void __launch_bounds__(kThreads) flags_pass(Geom g, int axis, const T* __restrict__ r,
                                                       const T* __restrict__ tau, uint8_t* __restrict__ flags,
                                                       Elem* el, const int32_t* run, int P, int32_t LX,
                                                       int32_t parts) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int64_t b = blockIdx.y;
  if (run && !run[b]) return;
  const int32_t n = elem_n(g, b, axis);
  const bool contig = axis == g.dim - 1;
  const int32_t nb = (n + kBlk - 1) / kBlk;
  T* X = reinterpret_cast<T*>(smem_raw);
  T* bmin = X + static_cast<int64_t>(P) * LX;
  T* bmax = bmin + static_cast<int64_t>(P) * nb;
  __shared__ int64_t base_s[64];
  __shared__ int32_t ok_s[64];
  __shared__ int32_t count_s;
  __shared__ uint32_t queue_s[kThreads / 32][kPeakQueue];
  const int64_t grp = parts > 1 ? blockIdx.x / parts : blockIdx.x;
  int32_t s_first = 1, s_end = n - 1;
  if (parts > 1) {
    part_of_line(n, &s_first, &s_end, parts, static_cast<int32_t>(blockIdx.x % parts));
    if (s_first >= s_end) return;
  }
  if (threadIdx.x < P) {
    const int p = threadIdx.x;
    bool ok;
    int64_t base;
    if (contig) {
      const int64_t row = grp * P + p;
      ok = row < g.rows;
      base = row * g.pitch;
    } else {
      // 32-bit divisions (an element holds fewer than 2^31 samples)
      const uint32_t inner = static_cast<uint32_t>(geom_stride(g, axis));
      const uint32_t gpo = (inner + P - 1) / P;
      const uint32_t o = static_cast<uint32_t>(grp) / gpo;
      const uint32_t c = (static_cast<uint32_t>(grp) - o * gpo) * P + p;
      ok = c < inner && static_cast<int32_t>(c % static_cast<uint32_t>(g.pitch)) < g.n_last;
      base = static_cast<int64_t>(o) * n * inner + c;
    }
    base_s[p] = base;
    ok_s[p] = ok ? 1 : 0;
  }
  if (threadIdx.x == 0) count_s = 0;
  const int64_t step = contig ? 1 : geom_stride(g, axis);
  const int64_t eoff = b * g.field;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (contig) {
    // a warp stages 1 / share of a line
    const int share = P >= kThreads / 32 ? 1 : kThreads / 32 / P;
    for (int q = warp; q < P * share; q += kThreads / 32) {
      const int p = q / share;
      if (!ok_s[p]) continue;
      const T* src = r + eoff + base_s[p];
      T* x = X + p * LX;
      for (int32_t i = lane + 32 * (q - p * share); i < n; i += 32 * share) copy_async(x + i + (i >> 5), src + i);
    }
  } else {
    // the P columns of a row over consecutive threads (whole sectors); one division per thread
    const int32_t rows_per = static_cast<int32_t>(blockDim.x) / P;
    const int p = static_cast<int>(threadIdx.x % P);
    const int32_t i0 = static_cast<int32_t>(threadIdx.x / P);
    if (i0 < rows_per && ok_s[p]) {
      const T* src = r + eoff + base_s[p];
      T* x = X + p * LX;
      for (int32_t i = i0; i < n; i += rows_per) copy_async(x + i + (i >> 5), src + static_cast<int64_t>(i) * step);
    }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  for (int32_t t = threadIdx.x; t < P * nb; t += blockDim.x) {
    const int p = t / nb;
    const int32_t c = t - p * nb;
    if (!ok_s[p]) continue;
    const T* xb = X + p * LX + c * (kBlk + 1);  // block c, stored contiguously
    const int32_t len = min(kBlk, n - c * kBlk);
    T mn = xb[0], mx = mn;
    for (int32_t i = 1; i < len; ++i) {
      const T v = xb[i];
      mn = (v < mn || v != v) ? v : mn;
      mx = (v > mx || v != v) ? v : mx;
    }
    bmin[p * nb + c] = mn;
    bmax[p * nb + c] = mx;
  }
  __syncthreads();
  int mine = 0, held = 0;
  uint32_t* queue = queue_s[warp];
  // a queued peak: its sample (below 2^24), line (6 bits) and kind
  const auto judge = [&](uint32_t entry) {
    const int32_t pk = static_cast<int32_t>(entry & 0xffffffu);
    const int p = static_cast<int>(entry >> 24) & 63;
    const int64_t at = eoff + base_s[p] + pk * step;
    const T tp = tau[at];
    const T* x = X + p * LX;
    const auto at_k = [x](int32_t k) { return xs(x, k); };
    if (peak_counts<T>(at_k, n, pk, static_cast<int>(entry >> 30), tp, bmin + p * nb, bmax + p * nb)) {
      flags[at] |= static_cast<uint8_t>(1u << axis);
      ++mine;
    }
  };
  // the warp's lanes together: lane's sample s of line p (valid: inside the line)
  const auto visit = [&](int p, int32_t s, bool valid) {
    int kind = 0;
    int32_t pk = 0;
    if (valid) {
      const T* x = X + p * LX;
      const auto at_k = [x](int32_t k) { return xs(x, k); };
      kind = peak_at<T>(at_k, n, nb, s, bmin + p * nb, bmax + p * nb, &pk);
    }
    push_peaks(queue, held, kind != 0,
               static_cast<uint32_t>(pk) | static_cast<uint32_t>(p) << 24 | static_cast<uint32_t>(kind) << 30, judge);
  };
  if (contig) {
    const int32_t runs = (s_end - s_first + 31) / 32;  // 32-sample runs of a line's inner samples
    for (int32_t q = warp; q < P * runs; q += kThreads / 32) {
      const int p = q / runs;
      if (!ok_s[p]) continue;
      const int32_t s = s_first + 32 * (q - p * runs) + lane;
      visit(p, s, s < s_end);
    }
  } else {
    // lanes over the panel's columns; a warp covers 32 / P rows (P a power of two <= 32)
    const int p = threadIdx.x & (P - 1);
    const int32_t rpw = 32 / P;
    const int32_t nrows = static_cast<int32_t>(blockDim.x >> 5) * rpw;
    const bool ok = ok_s[p] != 0;
    for (int32_t s0 = 1 + warp * rpw; s0 <= n - 2; s0 += nrows) {
      const int32_t s = s0 + lane / P;
      visit(p, s, ok && s <= n - 2);
    }
  }
  drain_peaks(queue, held, judge);
  for (int d = 16; d > 0; d >>= 1) mine += __shfl_down_sync(0xffffffffu, mine, d);
  if (lane == 0 && mine) atomicAdd(&count_s, mine);
  __syncthreads();
  if (threadIdx.x == 0 && count_s) {
    atomicAdd(reinterpret_cast<unsigned long long*>(&el[b].ext[axis]), static_cast<unsigned long long>(count_s));
  }
}

// Lines too long to stage (1-D signals beyond the staged capacity): a CTA takes one of gridDim.x parts
// of a line's samples, reads samples from global memory (L1 / L2) and keeps the whole line's 32-sample
// block extremes in shared memory (a warp per block); the peaks and their walks are those of the
// staged kernel.
template <class T>
__global__ void __launch_bounds__(kThreads) flags_long(Geom g, const T* __restrict__ r, const T* __restrict__ tau,
                                                       uint8_t* __restrict__ flags, Elem* el, const int32_t* run) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int32_t count_s;
  __shared__ uint32_t queue_s[kThreads / 32][kPeakQueue];
  const int64_t b = blockIdx.y;
  if (run && !run[b]) return;
  const int32_t n = elem_len(g, b);
  int32_t s_first, s_end;
  part_of_line(n, &s_first, &s_end, static_cast<int32_t>(gridDim.x), static_cast<int32_t>(blockIdx.x));
  if (s_first >= s_end) return;
  const int32_t nb = (n + kBlk - 1) / kBlk;
  T* bmin = reinterpret_cast<T*>(smem_raw);
  T* bmax = bmin + nb;
  const int64_t base = b * g.field;
  const T* line = r + base;
  if (threadIdx.x == 0) count_s = 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int32_t c = warp; c < nb; c += kThreads / 32) {
    const T v = line[min(c * kBlk + lane, n - 1)];
    T mn = v, mx = v;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      const T a = __shfl_xor_sync(0xffffffffu, mn, d), z = __shfl_xor_sync(0xffffffffu, mx, d);
      mn = (a < mn || a != a) ? a : mn;
      mx = (z > mx || z != z) ? z : mx;
    }
    if (lane == 0) {
      bmin[c] = mn;
      bmax[c] = mx;
    }
  }
  __syncthreads();
  const auto at_k = [line](int32_t k) { return line[k]; };
  int mine = 0, held = 0;
  uint32_t* queue = queue_s[warp];
  const auto judge = [&](uint32_t entry) {
    const int32_t pk = static_cast<int32_t>(entry & 0xffffffu);
    if (peak_counts<T>(at_k, n, pk, static_cast<int>(entry >> 30), tau[base + pk], bmin, bmax)) {
      flags[base + pk] |= static_cast<uint8_t>(1u);
      ++mine;
    }
  };
  for (int32_t s0 = s_first + 32 * warp; s0 < s_end; s0 += kThreads) {
    int kind = 0;
    int32_t pk = 0;
    if (s0 + lane < s_end) kind = peak_at<T>(at_k, n, nb, s0 + lane, bmin, bmax, &pk);
    push_peaks(queue, held, kind != 0, static_cast<uint32_t>(pk) | static_cast<uint32_t>(kind) << 30, judge);
  }
  drain_peaks(queue, held, judge);
  for (int d = 16; d > 0; d >>= 1) mine += __shfl_down_sync(0xffffffffu, mine, d);
  if (lane == 0 && mine) atomicAdd(&count_s, mine);
  __syncthreads();
  if (threadIdx.x == 0 && count_s) {
    atomicAdd(reinterpret_cast<unsigned long long*>(&el[b].ext[0]), static_cast<unsigned long long>(count_s));
  }
}

// ---------------------------------------------------------------------------------------------
// Face-connected components, labelled by the smallest padded index of the component. Parent links
// always point to a smaller index and a root is linked only by a compare-and-swap that finds it
// still a root, so every tree's root is its smallest member whatever the order of the threads.
// Phase 1 labels the components of every tile (consecutive rows of an element) in shared memory;
// phase 2 joins the trees across the tile borders in global memory; phase 3 points every voxel at
// its root.

// Root of x; parent reads bypass L1 (another SM may have relinked a root), shared memory is
// coherent inside the CTA and read volatile.
template <bool Global>
__device__ __forceinline__ int32_t uf_root(int32_t* P, int32_t x) {
  for (;;) {
    const int32_t up = Global ? __ldcg(P + x) : *reinterpret_cast<volatile int32_t*>(P + x);
    if (up == x) return x;
    if constexpr (Global) {
      x = up;
    } else {
      // (shared memory) the walked nodes skip to their grandparents, ancestors at any time: later
      // walks halve. A plain store loses no join: a node that has a parent is never linked again.
      const int32_t above = *reinterpret_cast<volatile int32_t*>(P + up);
      if (above != up) *reinterpret_cast<volatile int32_t*>(P + x) = above;
      x = above;
    }
  }
}
template <bool Global>
__device__ __forceinline__ void uf_join(int32_t* P, int32_t x, int32_t y) {
  for (;;) {
    x = uf_root<Global>(P, x);
    y = uf_root<Global>(P, y);
    if (x == y) return;
    const int32_t big = x > y ? x : y, small = x > y ? y : x;
    if (atomicCAS(P + big, big, small) == big) return;  // big was still a root: now under small
    x = big;
    y = small;
  }
}

constexpr int32_t kTileWords = 8192;  // int32 parents per tile (32 KiB of shared memory)

__device__ __forceinline__ int64_t rows_between(const Geom& g, int a) { return geom_stride(g, a) / g.pitch; }

// Bound by the joins' chains in shared memory: with runs labelled by a ballot and joined at their heads
// only, and walks that shorten their paths, one image of 301 x 443 takes 41 us (225 us when every set
// sample was joined to its neighbours) and 64 of 512 x 512 160 us (413 us).
// A tile is tile_rows consecutive rows of an element, whole (tile_cols = pitch), or for rows longer
// than a tile (1-D lines beyond kTileWords samples) a run of tile_cols columns of one row.
__global__ void __launch_bounds__(kThreads) ccl_tiles(Geom g, const uint8_t* __restrict__ mask, uint8_t bits,
                                                     int32_t* __restrict__ labels, const int32_t* run, int32_t tile_rows,
                                                     int32_t tile_cols) {
  __shared__ int32_t P[kTileWords];
  const int64_t b = blockIdx.y;
  if (run && !run[b]) return;
  const int32_t pitch = static_cast<int32_t>(g.pitch), nl = elem_len(g, b);
  const int32_t col_tiles = (pitch + tile_cols - 1) / tile_cols;
  const int64_t row0 = static_cast<int64_t>(blockIdx.x / col_tiles) * tile_rows;
  const int32_t c0 = static_cast<int32_t>(blockIdx.x % col_tiles) * tile_cols;
  if (row0 >= g.rows) return;
  const int32_t rows = static_cast<int32_t>(min(static_cast<int64_t>(tile_rows), g.rows - row0));
  const int32_t cols = min(tile_cols, pitch - c0);
  const int32_t words = rows * cols;
  const int64_t v0 = row0 * g.pitch + c0;  // the tile's first padded offset in the element
  const int64_t eb = b * g.field;
  // local index k = r cols + c <-> padded offset v0 + r pitch + c. A warp's 32 consecutive samples lie in
  // one row (cols is a multiple of 32): each set sample starts under the first sample of its run
  // among them, by a ballot, so only the runs' heads are joined
  const int lane = threadIdx.x & 31;
  for (int32_t k = threadIdx.x; k < words; k += blockDim.x) {
    const int32_t r = k / cols, c = k - r * cols;
    const bool set = c0 + c < nl && (mask[eb + v0 + static_cast<int64_t>(r) * pitch + c] & bits) != 0;
    const unsigned m = __ballot_sync(0xffffffffu, set);
    const unsigned gaps = ~m & ((1u << lane) - 1u);  // unset samples before this lane
    P[k] = set ? k - lane + (gaps ? 32 - __clz(gaps) : 0) : -1;
  }
  __syncthreads();
  for (int32_t k = threadIdx.x; k < words; k += blockDim.x) {
    if (P[k] < 0) continue;
    const int32_t r = k / cols, c = k - r * cols;
    const bool left = c > 0 && P[k - 1] >= 0;
    if (lane == 0 && left) uf_join<false>(P, k - 1, k);
    for (int a = 0; a + 1 < g.dim; ++a) {
      const int64_t rs = rows_between(g, a);
      if (r + rs >= rows || coord_of(g, v0 + static_cast<int64_t>(r) * pitch + c, a) + 1 >= geom_n(g, a)) continue;
      const int32_t u = k + static_cast<int32_t>(rs) * cols;
      // (where the samples to the left are set in both rows, they join the same two runs)
      if (P[u] >= 0 && !(left && P[u - 1] >= 0)) uf_join<false>(P, k, u);
    }
  }
  __syncthreads();
  for (int32_t k = threadIdx.x; k < words; k += blockDim.x) {
    const int32_t r = k / cols, c = k - r * cols;
    int32_t lab = -1;
    if (P[k] >= 0) {
      const int32_t root = uf_root<false>(P, k);  // the local root: the smallest local index, so the
      const int32_t rr = root / cols;             // smallest padded offset of the tile's component
      lab = static_cast<int32_t>(v0 + static_cast<int64_t>(rr) * pitch + (root - rr * cols));
    }
    labels[eb + v0 + static_cast<int64_t>(r) * pitch + c] = lab;
  }
}

}  // namespace

// ---------------------------------------------------------------------------------------------
template <class T>
void sig_flags(cudaStream_t s, const Geom& g, const T* r, const T* tau, uint8_t* flags, Elem* el, const int32_t* run) {
  for_samples(s, g.batch * g.field, [=] __device__(int64_t i) {
    if (run == nullptr || run[elem_of(g, i)]) flags[i] = 0;
  });
  int optin = 0, dev = 0;
  EDAB_CUDA(cudaGetDevice(&dev));
  EDAB_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const size_t cap = static_cast<size_t>(optin) - 4096;  // (the kernels' static shared memory)
  once_on_device(reinterpret_cast<const void*>(flags_pass<T>), [&] {  // the limit is per device
    EDAB_CUDA(cudaFuncSetAttribute(flags_pass<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(cap)));
  });
  int sms = 148;
  EDAB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  for (int a = 0; a < g.dim; ++a) {
    const int32_t n = g.n[a];
    if (n < 3) continue;
    const bool rows = a == g.dim - 1;
    const int32_t nb = (n + kBlk - 1) / kBlk;
    int64_t outer = 1;
    for (int ax = 0; ax < a; ++ax) outer *= g.n[ax];
    const auto groups_of = [&](int p) { return rows ? (g.rows + p - 1) / p : outer * ((g.stride[a] + p - 1) / p); };
    int P;
    if (rows) P = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>({static_cast<int64_t>(8192 / n), g.rows, 64})));
    else P = static_cast<int>(std::min<int64_t>(16, g.stride[a]));  // a power of two (stride: a multiple of 32)
    // fewer lines per CTA while the launch would leave SMs without one (a column panel keeps whole
    // sectors)
    while (P > (rows ? 1 : 8) && groups_of(P) * g.batch < 2 * sms) P /= 2;
    const int32_t LX = (n + ((n - 1) >> 5) + 1) | 1;  // padded line words, odd
    const auto bytes = [&](int p) { return static_cast<size_t>(p) * (LX + 2 * nb) * sizeof(T); };
    while (P > 1 && bytes(P) > cap) P = rows ? P - 1 : P / 2;
    // a 1-D line's parts: at least 512 samples each, about one CTA per SM in all
    const int32_t parts = g.dim == 1 ? static_cast<int32_t>(std::clamp<int64_t>(
                                           std::min<int64_t>(n / 512, sms / std::max<int64_t>(1, g.batch)), 1, 64))
                                     : 1;
    if (bytes(P) > cap) {
      // a 1-D line beyond the staged capacity: samples from global memory, block extremes staged
      const size_t ext_bytes = static_cast<size_t>(2) * nb * sizeof(T);
      if (g.dim != 1 || ext_bytes > cap) throw std::invalid_argument("edab: a line exceeds the shared memory of the extrema pass");
      once_on_device(reinterpret_cast<const void*>(flags_long<T>), [&] {
        EDAB_CUDA(cudaFuncSetAttribute(flags_long<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(cap)));
      });
      const int64_t fill = std::clamp<int64_t>((8 * static_cast<int64_t>(sms) + g.batch - 1) / g.batch, 1, 16);
      enqueue(flags_long<T>, dim3(static_cast<unsigned>(fill), static_cast<unsigned>(g.batch)), kThreads, ext_bytes, s, 
          g, r, tau, flags, el, run);
      continue;
    }
    enqueue(flags_pass<T>, dim3(static_cast<unsigned>(groups_of(P) * parts), static_cast<unsigned>(g.batch)), kThreads, bytes(P), s, 
        g, a, r, tau, flags, el, run, P, LX, parts);
  }
}

void ccl(cudaStream_t s, const Geom& g, const uint8_t* mask, uint8_t bits, int32_t* labels, const int32_t* run) {
  const bool wide = g.pitch > kTileWords;
  const int32_t tile_rows = wide ? 1 : static_cast<int32_t>(kTileWords / g.pitch);
  const int32_t tile_cols = wide ? kTileWords : static_cast<int32_t>(g.pitch);
  const int64_t col_tiles = (g.pitch + tile_cols - 1) / tile_cols;
  const int64_t tiles = (g.rows + tile_rows - 1) / tile_rows * col_tiles;
  if (tiles > 0x7fffffffLL || g.batch > 65535) throw std::invalid_argument("edab: components: grid too large");
  enqueue(ccl_tiles, dim3(static_cast<unsigned>(tiles), static_cast<unsigned>(g.batch)), kThreads, 0, s, 
      g, mask, bits, labels, run, tile_rows, tile_cols);
  // the edges between tiles
  for_voxels(s, g, [=] __device__(int64_t b) { return run == nullptr || run[b] != 0; },
             [=] __device__(int64_t b, int64_t v, int64_t i) {
               int32_t* L = labels + b * g.field;
               if (L[v] < 0) return;
               const int64_t row = pitch_row(g, v);
               const int64_t col = v - row * g.pitch;
               if (wide && (col + 1) % tile_cols == 0 && col + 1 < elem_len(g, b) && L[v + 1] >= 0) {
                 uf_join<true>(L, static_cast<int32_t>(v), static_cast<int32_t>(v + 1));
               }
               const int64_t tile = row / tile_rows;
               for (int a = 0; a + 1 < g.dim; ++a) {
                 const int64_t rs = geom_stride(g, a) / g.pitch;
                 if ((row + rs) / tile_rows == tile || coord_of(g, v, a) + 1 >= geom_n(g, a)) continue;
                 const int64_t u = v + geom_stride(g, a);
                 if (L[u] >= 0) uf_join<true>(L, static_cast<int32_t>(v), static_cast<int32_t>(u));
               }
             });
  // every voxel to its root
  for_voxels(s, g, [=] __device__(int64_t b) { return run == nullptr || run[b] != 0; },
             [=] __device__(int64_t b, int64_t v, int64_t i) {
               int32_t* L = labels + b * g.field;
               if (L[v] < 0) return;
               L[v] = uf_root<true>(L, static_cast<int32_t>(v));
             });
}

template void field_totals<float>(cudaStream_t, const Geom&, const float*, double*, double*, uint64_t*, void*);
template void field_totals<double>(cudaStream_t, const Geom&, const double*, double*, double*, uint64_t*, void*);
template void select<float>(cudaStream_t, const Geom&, const Sel<float>&, double, const int32_t*, double*, int64_t*, void*);
template void select<double>(cudaStream_t, const Geom&, const Sel<double>&, double, const int32_t*, double*, int64_t*, void*);
template void sig_flags<float>(cudaStream_t, const Geom&, const float*, const float*, uint8_t*, Elem*, const int32_t*);
template void sig_flags<double>(cudaStream_t, const Geom&, const double*, const double*, uint8_t*, Elem*, const int32_t*);

}  // namespace edab
