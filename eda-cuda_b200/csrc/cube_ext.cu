// SPDX-License-Identifier: Apache-2.0
// The running max / min passes of the cube filter. Max and min of order keys have no rounding, so
// any cover of the window gives the reference's bits (cpp/src/field/vhgw.cu:1-36 of eda-cuda folds
// segments of the window's own length instead), and the half-sample reflection only repeats
// samples of the window: y(x) is the extreme of the samples [max(0, x - r), min(n - 1, x + r)].
//
// A line is cut into blocks of B samples (B <= 2r, at most block_cap), independent of the window:
// H, the extreme of a block from a sample to its end, G, of a block up to a sample, and a table of
// the extremes of 2^k consecutive blocks. An output takes H of its window's first sample, G of its
// last, and two table entries that cover the blocks between: four reads whatever the window. H, G
// and the table are built once per staging for every rung with the same B (a ladder shares one B
// but for its smallest windows), by threads that each run a block forward and backward, so a pass
// has two barriers and chains of at most B steps.
//
// What bounds it: issue slots (48 warp instructions per 32 samples and pass, 60 while the choice of what
// is stored stood inside the loops) and the barrier between build and output. A pass of 64 fields of
// 512 x 512 float32: rows 40 us, panels 46 us for every window up to 127 (62 to 108 us and 67 to
// 104 us with segments of the window's own length); a ladder of 7 rungs in one staging 155 us (339);
// 134 MB move per single pass, 21 us at the copy rate. Running several line groups per CTA with the
// next group's copies under way during the output was slower (55 us): fewer CTAs to overlap.
// B is odd (column panels) or, with fewer than 8 lines, four times an odd number (rows) so that the
// lanes of a warp, working on consecutive blocks, lie in distinct banks.
#include "cube.cuh"

#include <algorithm>
#include <type_traits>

namespace edab {
namespace cubes {
namespace {

__device__ __forceinline__ int32_t bits_of(float v) { return __float_as_int(v); }
__device__ __forceinline__ long long bits_of(double v) { return __double_as_longlong(v); }
__device__ __forceinline__ float value_bits(int32_t k) { return __int_as_float(k); }
__device__ __forceinline__ double value_bits(long long k) { return __longlong_as_double(k); }

// The longest blocks: short ones keep the CTA's threads busy on short lines (512 samples of 8 lines
// are 256 blocks of 16 in rows for 256 threads), long ones keep the table small on long lines. The line at 640
// is not a sharp one. Short / long blocks, us at a window of 127: panels of 64 x 512^2 46.3 / 43.6, of 40 x
// 640^2 45.5 / 43.8, of 28 x 768^2 54.6 / 52.3; single rows, 1024 of 512 samples 7.9 / 8.3, of 640 8.4 / 8.9,
// of 1024 9.7 / 10.3, of 4096 18.5 / 18.7 (a ladder of 7 rungs 70.4 / 68.9).
__host__ __device__ constexpr int32_t block_cap(int32_t n, int P, bool rows) {
  return rows ? (P == 8 ? 16 : (n <= 640 ? 20 : 28)) : (n <= 640 ? 15 : 31);
}
// The block length of half width r >= 2 (B <= 2r; below the cap a window holds at most two whole
// blocks, which are read from H instead of the table).
template <int P, bool ROWS>
__device__ __forceinline__ int32_t block_len(int32_t r, int32_t cap) {
  if (2 * r >= cap) return cap;
  if constexpr (ROWS && P != 8) return r < 6 ? 4 : 12;
  const int32_t two = 2 << (31 - __clz(r));
  return ROWS ? two : two - 1;
}
// (at most nb - 1 whole blocks lie beside the block of a window's end)
__host__ __device__ constexpr int32_t table_levels(int32_t nb) {
  int32_t k = 1;
  while ((2 << (k - 1)) <= nb - 1) ++k;
  return k;
}
__host__ __device__ constexpr int32_t table_elems(int32_t n, int P, bool rows) {
  const int32_t nb = (n + block_cap(n, P, rows) - 1) / block_cap(n, P, rows);
  return nb * table_levels(nb);
}

// H and G of a whole block of BT samples held in registers (rows; left: the samples up to the line's
// end, at most BT of which count); returns the block's extreme.
template <class T, class K, int BT>
__device__ __forceinline__ K build_block(const T* v, K* h, K* g, int32_t left, K nm) {
  constexpr int VW = 16 / static_cast<int>(sizeof(T));
  K key[BT];
#pragma unroll
  for (int i = 0; i < BT; i += VW) {
    const Pack<T, VW> x = load_pack<T, VW>(v + i);
#pragma unroll
    for (int k = 0; k < VW; ++k) key[i + k] = okey_i(x.v[k]) ^ nm;
  }
  if (left < BT) {
#pragma unroll
    for (int i = 0; i < BT; ++i) key[i] = i < left ? key[i] : key_min<K>();
  }
  K run = key[BT - 1];
#pragma unroll
  for (int i = BT - VW; i >= 0; i -= VW) {
    Pack<K, VW> o;
#pragma unroll
    for (int k = VW - 1; k >= 0; --k) {
      run = max(run, key[i + k]);
      o.v[k] = run;
    }
    store_pack<K, VW>(h + i, o);
  }
  run = key[0];
#pragma unroll
  for (int i = 0; i < BT; i += VW) {
    Pack<K, VW> o;
#pragma unroll
    for (int k = 0; k < VW; ++k) {
      run = max(run, key[i + k]);
      o.v[k] = run;
    }
    store_pack<K, VW>(g + i, o);
  }
  return run;
}

template <class T, int P, bool ROWS>
__global__ void __launch_bounds__(kCubeThreads, kCubeCtas) ext_pass(Geom g, PassArgs<T> a) {
  using K = typename KeyType<T>::type;
  constexpr int VW = 16 / static_cast<int>(sizeof(T));
  constexpr int W = !ROWS && P >= VW ? VW : 1;  // columns of one access
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int64_t b = blockIdx.y;
  const int32_t n = elem_n(g, b, a.axis);
  const uint32_t inner = ROWS ? 1u : static_cast<uint32_t>(geom_stride(g, a.axis));
  const int lp = ROWS && P != 8 ? a.lp : 3;
  const int lines = ROWS && P != 8 ? 1 << a.lp : P;
  const int32_t LS = ROWS ? row_stride<T>(n) : 1;
  const int32_t gel = ROWS ? lines * LS : ((n * P + 3) & ~3);
  // (blockIdx.z counts the rungs, and the fields of a max + min cube, that a CTA does not loop over)
  const bool fields_z = a.op == static_cast<int>(CubeOp::kMaxMin) && a.zf == 1;
  const int32_t j_begin = static_cast<int32_t>(fields_z ? blockIdx.z >> 1 : blockIdx.z) * a.zr;
  const int f_begin = fields_z ? static_cast<int>(blockIdx.z & 1) : 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // every warp looks its rungs' windows up (no barrier before the staging starts): lane j holds the
  // clamped half width of rung j, or -1
  const int32_t w = lane < a.zr ? a.win[static_cast<int64_t>(j_begin + lane) * g.batch + b] : 0;
  if (__ballot_sync(0xffffffffu, w >= 1) == 0u) return;
  const int32_t r_lane = w >= 1 ? min((w - 1) >> 1, n - 1) : -1;
  const GroupPos pos = group_at<ROWS>(g, blockIdx.x, n, inner, static_cast<uint32_t>(lines), a.panels);
  if (!pos.mask) return;
  const int64_t eoff = b * g.field;
  // long lines, one rung and field per CTA: G over the samples (each read by its block's thread only,
  // before it writes there), so that longer lines fit
  const bool over = ROWS && P != 8 && a.zr == 1 && a.zf == 1;
  T* V = reinterpret_cast<T*>(smem_raw);
  K* H = reinterpret_cast<K*>(smem_raw) + gel;
  K* G = over ? reinterpret_cast<K*>(smem_raw) : H + gel;
  K* tab = (over ? H : G) + gel;
  stage_lines<T, P, ROWS>(g, a, V, (f_begin == 0 || !a.in1 ? a.in0 : a.in1) + j_begin * a.in_stride + eoff, nullptr, pos,
                          n, LS, inner);
  stage_wait();
  __syncthreads();
  const int32_t cap = block_cap(geom_n(g, a.axis), P, ROWS);  // (the table is sized for the longest element)
  const K idn = key_min<K>();
  constexpr int QP = P / W;
  unsigned long long outputs = 0;
  for (int f = f_begin; f < f_begin + a.zf; ++f) {
    const bool is_min = a.op == static_cast<int>(CubeOp::kMin) || f == 1;
    const K nm = is_min ? static_cast<K>(-1) : static_cast<K>(0);  // min: the complement's max
    int32_t B = 0, nb = 0, levels = 0;
    uint32_t inv = 0;
    // the samples of the first axis (rows) are values, those of the others (panels) already keys
    const auto key_of = [&](T v) {
      if constexpr (ROWS) return static_cast<K>(okey_i(v) ^ nm);
      else return bits_of(v);
    };
    for (int32_t jj = 0; jj < a.zr; ++jj) {
      const int32_t r = __shfl_sync(0xffffffffu, r_lane, jj);
      if (r < 0) continue;
      if (r >= 2 && block_len<P, ROWS>(r, cap) != B) {
        if (B) __syncthreads();  // the last rung's outputs are taken
        B = block_len<P, ROWS>(r, cap);
        inv = 0xffffffffu / static_cast<uint32_t>(B) + 1u;  // i / B = umulhi(i, inv) for i < 2^32 / B
        nb = static_cast<int32_t>(__umulhi(n + B - 1, inv));
        levels = 1;
        if constexpr (ROWS && P == 8) {
          for (int32_t t = threadIdx.x; t < nb * 8; t += kCubeThreads) {
            const int p = t & 7;
            const int32_t blk = t >> 3;
            const int32_t s0 = p * LS + blk * B, left = n - blk * B;
            if (B == 16) tab[t] = build_block<T, K, 16>(V + s0, H + s0, G + s0, left, nm);
            else if (B == 8) build_block<T, K, 8>(V + s0, H + s0, G + s0, left, nm);
            else build_block<T, K, 4>(V + s0, H + s0, G + s0, left, nm);
          }
        } else if constexpr (ROWS) {
          for (int32_t t = threadIdx.x; t < nb << lp; t += kCubeThreads) {
            const int p = t & (lines - 1);
            const int32_t blk = t >> lp;
            const int32_t s0 = p * LS + blk * B, left = n - blk * B;  // samples from the block's start
            K run = idn;
#pragma unroll 2
            for (int32_t i = B - VW; i >= 0; i -= VW) {
              const Pack<T, VW> v = load_pack<T, VW>(V + s0 + i);
              Pack<K, VW> o;
#pragma unroll
              for (int k = VW - 1; k >= 0; --k) {
                const K key = i + k < left ? key_of(v.v[k]) : idn;
                run = max(run, key);
                o.v[k] = run;
              }
              if (i < left) store_pack<K, VW>(H + s0 + i, o);
            }
            run = idn;
#pragma unroll 2
            for (int32_t i = 0; i < B; i += VW) {
              const Pack<T, VW> v = load_pack<T, VW>(V + s0 + i);
              Pack<K, VW> o;
#pragma unroll
              for (int k = 0; k < VW; ++k) {
                const K key = i + k < left ? key_of(v.v[k]) : idn;
                run = max(run, key);
                o.v[k] = run;
              }
              if (i < left) store_pack<K, VW>(G + s0 + i, o);
            }
            if (B == cap) tab[blk * lines + p] = run;
          }
        } else {
          // a thread runs one block of W columns forward (G) or backward (H)
          for (int32_t t = threadIdx.x; t < 2 * nb * QP; t += kCubeThreads) {
            const bool back = t >= nb * QP;
            const int32_t u = back ? t - nb * QP : t;
            const int q = (u % QP) * W;
            const int32_t blk = u / QP;
            const int32_t i0 = blk * B, len = min(B, n - i0);
            const T* v = V + (back ? i0 + len - 1 : i0) * P + q;
            K* o = (back ? H : G) + (back ? i0 + len - 1 : i0) * P + q;
            const int32_t step = back ? -P : P;
            Pack<K, W> run;
#pragma unroll
            for (int k = 0; k < W; ++k) run.v[k] = idn;
            int32_t i = 0;
            for (; i + 5 <= len; i += 5) {
              Pack<T, W> x[5];
#pragma unroll
              for (int m = 0; m < 5; ++m) x[m] = load_pack<T, W>(v + m * step);
#pragma unroll
              for (int m = 0; m < 5; ++m) {
#pragma unroll
                for (int k = 0; k < W; ++k) run.v[k] = max(run.v[k], key_of(x[m].v[k]));
                store_pack<K, W>(o + m * step, run);
              }
              v += 5 * step;
              o += 5 * step;
            }
            for (; i < len; ++i) {
              const Pack<T, W> x = load_pack<T, W>(v);
#pragma unroll
              for (int k = 0; k < W; ++k) run.v[k] = max(run.v[k], key_of(x.v[k]));
              store_pack<K, W>(o, run);
              v += step;
              o += step;
            }
            if (B == cap && !back) store_pack<K, W>(tab + blk * P + q, run);
          }
        }
        __syncthreads();
      }
      if (r >= 2 && B == cap) {
        // levels up to the most whole blocks that a window holds
        const int32_t most = min(nb - 1, static_cast<int32_t>(__umulhi(2 * r, inv)));
        while ((2 << (levels - 1)) <= most) {
          const int32_t half = 1 << (levels - 1);
          const K* from = tab + (levels - 1) * nb * lines;
          K* to = tab + levels * nb * lines;
          for (int32_t t = threadIdx.x; t < nb * lines; t += kCubeThreads) {
            const int32_t j = ROWS ? t >> lp : t / P;
            const int p = ROWS ? t & (lines - 1) : t % P;
            to[t] = max(from[t], from[min(j + half, nb - 1) * lines + p]);
          }
          __syncthreads();
          ++levels;
        }
      }
      T* out = (f == 0 ? a.out0 : a.out1) + static_cast<int64_t>(j_begin + jj) * a.out_stride + eoff + pos.base;
      const auto line_out = [&](auto keys) {  // (what is stored is chosen outside the loops)
        const auto value_of = [&](K k) {
          if constexpr (decltype(keys)::value) return value_bits(k);
          else return key_back(static_cast<K>(k ^ nm));
        };
        if constexpr (ROWS) {
          const int per = kWarps >> lp;
          const int p = P == 8 ? warp : warp / per;
          if (p >= lines || !((pos.mask >> p) & 1u)) return;
          T* o = out + static_cast<int64_t>(p) * g.pitch;
          const K* Hp = H + p * LS;
          const K* Gp = G + p * LS;
          const T* Vp = V + p * LS;
          const K* tp = tab + p;
          const int32_t dx = 32 * per;
          int32_t x = lane + 32 * (P == 8 ? 0 : warp - p * per);
          if (r == 0) {
            for (; x < n; x += dx) o[x] = value_of(key_of(Vp[x]));
          } else if (r == 1) {
            for (; x < n; x += dx) {
              o[x] = value_of(max(max(key_of(Vp[max(x - 1, 0)]), key_of(Vp[x])), key_of(Vp[min(x + 1, n - 1)])));
            }
          } else {
            const auto edge_out = [&](int32_t x) {
              const int32_t lo = x - r, hi = min(x + r, n - 1);
              const int32_t b0 = lo >= 0 ? static_cast<int32_t>(__umulhi(lo, inv)) : -1;
              const int32_t b1 = static_cast<int32_t>(__umulhi(hi, inv));
              K y = lo >= 0 ? Hp[lo] : idn;
              if (b1 > b0) y = max(y, Gp[hi]);
              const int32_t L = b1 - b0 - 1;  // whole blocks between
              if (L > 0) {
                if (B == cap) {
                  const int32_t k = 31 - __clz(L);
                  const K* lv = tp + (k * nb) * lines;
                  y = max(y, max(lv[(b0 + 1) * lines], lv[(b1 - (1 << k)) * lines]));
                } else {
                  y = max(y, max(Hp[(b0 + 1) * B], Hp[(b1 - 1) * B]));
                }
              }
              o[x] = value_of(y);
            };
            if constexpr (P == 8) {
              // outputs whose window lies inside the line, 32 consecutive per warp step: a step is a whole
              // number of blocks, so a lane's blocks between keep their number and its reads advance
              // by constants (a lane with none reads its H again)
              const int32_t first = (r + 31) >> 5, steps = max(((n - r) >> 5) - first, 0);
              const int32_t edge = min(32 * first, n);
              for (; x < edge; x += 32) edge_out(x);
              if (steps > 0) {
                x = lane + 32 * first;
                const int32_t b0 = static_cast<int32_t>(__umulhi(x - r, inv)), b1 = static_cast<int32_t>(__umulhi(x + r, inv));
                const int32_t L = b1 - b0 - 1;
                const K* h = Hp + (x - r);
                const K* e = Gp + (x + r);
                const K *t0 = h, *t1 = h;
                int32_t ts = 32;
                if (L > 0 && B < cap) {
                  t0 = t1 = Hp + (b0 + 1) * B;
                } else if (L > 0) {
                  const int32_t k = 31 - __clz(L);
                  t0 = tp + (k * nb + b0 + 1) * 8;
                  t1 = tp + (k * nb + b1 - (1 << k)) * 8;
                  ts = 32 / 16 * 8;  // (the cap is 16)
                }
                T* ox = o + x;
                int32_t i = 0;
                for (; i + 4 <= steps; i += 4) {
#pragma unroll
                  for (int u = 0; u < 4; ++u) {
                    ox[32 * u] = value_of(max(max(h[32 * u], e[32 * u]), max(*t0, *t1)));
                    t0 += ts;
                    t1 += ts;
                  }
                  h += 128;
                  e += 128;
                  ox += 128;
                }
                for (; i < steps; ++i) {
                  *ox = value_of(max(max(*h, *e), max(*t0, *t1)));
                  t0 += ts;
                  t1 += ts;
                  h += 32;
                  e += 32;
                  ox += 32;
                }
                x = lane + 32 * (first + steps);
              }
            }
            for (; x < n; x += dx) edge_out(x);
          }
          for (; x < static_cast<int32_t>(g.pitch); x += dx) o[x] = T(0);
        } else {
          const int q = (threadIdx.x % QP) * W;
          T* o = out + static_cast<int64_t>(threadIdx.x / QP) * inner + q;
          const int64_t step = static_cast<int64_t>(kCubeThreads / QP) * inner;
          const uint32_t live = pos.mask >> q;  // columns left of the row padding
          const auto put = [&](const Pack<K, W>& y) {
            Pack<T, W> res;
#pragma unroll
            for (int k = 0; k < W; ++k) res.v[k] = ((live >> k) & 1u) ? value_of(y.v[k]) : T(0);
            store_pack<T, W>(o, res);
            o += step;
          };
          if (r < 2) {
            for (int32_t x = threadIdx.x / QP; x < n; x += kCubeThreads / QP) {
              const Pack<T, W> v0 = load_pack<T, W>(V + max(x - r, 0) * P + q), v1 = load_pack<T, W>(V + x * P + q),
                               v2 = load_pack<T, W>(V + min(x + r, n - 1) * P + q);
              Pack<K, W> y;
#pragma unroll
              for (int k = 0; k < W; ++k) y.v[k] = max(max(key_of(v0.v[k]), key_of(v1.v[k])), key_of(v2.v[k]));
              put(y);
            }
            return;
          }
          for (int32_t x = threadIdx.x / QP; x < n; x += kCubeThreads / QP) {
            const int32_t lo = x - r, hi = min(x + r, n - 1);
            const int32_t b0 = lo >= 0 ? static_cast<int32_t>(__umulhi(lo, inv)) : -1;
            const int32_t b1 = static_cast<int32_t>(__umulhi(hi, inv));
            Pack<K, W> y = load_pack<K, W>(lo >= 0 ? H + lo * P + q : G + hi * P + q);
            if (b1 > b0 && lo >= 0) {
              const Pack<K, W> v = load_pack<K, W>(G + hi * P + q);
#pragma unroll
              for (int k = 0; k < W; ++k) y.v[k] = max(y.v[k], v.v[k]);
            }
            const int32_t L = b1 - b0 - 1;
            if (L > 0) {
              const K *p0, *p1;
              if (B == cap) {
                const int32_t k = 31 - __clz(L);
                const K* lv = tab + (k * nb) * P + q;
                p0 = lv + (b0 + 1) * P;
                p1 = lv + (b1 - (1 << k)) * P;
              } else {
                p0 = H + (b0 + 1) * B * P + q;
                p1 = H + (b1 - 1) * B * P + q;
              }
              const Pack<K, W> v0 = load_pack<K, W>(p0), v1 = load_pack<K, W>(p1);
#pragma unroll
              for (int k = 0; k < W; ++k) y.v[k] = max(y.v[k], max(v0.v[k], v1.v[k]));
            }
            put(y);
          }
        }
      };
      if (a.keys_out) line_out(std::true_type{});
      else line_out(std::false_type{});
      ++outputs;
    }
    if (f + 1 < f_begin + a.zf) __syncthreads();  // the next field rewrites H, G and the table
  }
  if (a.bytes && threadIdx.x == 0) {
    atomicAdd(a.bytes, (1 + outputs) * static_cast<unsigned long long>(__popc(pos.mask)) * n * sizeof(T));
  }
}

}  // namespace

size_t ext_smem_bytes(int32_t n, int P, bool rows, size_t es) {
  const int32_t gel = es == 4 ? group_elems<float>(n, P, rows) : group_elems<double>(n, P, rows);
  return (static_cast<size_t>(3) * gel + static_cast<size_t>(table_elems(n, P, rows)) * P) * es;
}

template <class T>
void ext_allow_smem(int bytes) {
  EDAB_CUDA(cudaFuncSetAttribute(ext_pass<T, 8, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  EDAB_CUDA(cudaFuncSetAttribute(ext_pass<T, 1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  EDAB_CUDA(cudaFuncSetAttribute(ext_pass<T, 1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  EDAB_CUDA(cudaFuncSetAttribute(ext_pass<T, 2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  EDAB_CUDA(cudaFuncSetAttribute(ext_pass<T, 4, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  EDAB_CUDA(cudaFuncSetAttribute(ext_pass<T, 8, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}

template <class T>
void launch_ext(cudaStream_t s, const Geom& g, const PassArgs<T>& a, int P, bool rows, dim3 grid, size_t smem) {
  if (rows && P != 8 && a.zr == 1 && a.zf == 1) smem -= static_cast<size_t>(group_elems<T>(geom_n(g, a.axis), P, rows)) * sizeof(T);
  if (rows && P == 8) enqueue(ext_pass<T, 8, true>, grid, kCubeThreads, smem, s, g, a);
  else if (rows) enqueue(ext_pass<T, 1, true>, grid, kCubeThreads, smem, s, g, a);
  else if (P == 1) enqueue(ext_pass<T, 1, false>, grid, kCubeThreads, smem, s, g, a);
  else if (P == 2) enqueue(ext_pass<T, 2, false>, grid, kCubeThreads, smem, s, g, a);
  else if (P == 4) enqueue(ext_pass<T, 4, false>, grid, kCubeThreads, smem, s, g, a);
  else enqueue(ext_pass<T, 8, false>, grid, kCubeThreads, smem, s, g, a);
}

template void ext_allow_smem<float>(int);
template void ext_allow_smem<double>(int);
template void launch_ext<float>(cudaStream_t, const Geom&, const PassArgs<float>&, int, bool, dim3, size_t);
template void launch_ext<double>(cudaStream_t, const Geom&, const PassArgs<double>&, int, bool, dim3, size_t);

}  // namespace cubes
}  // namespace edab
