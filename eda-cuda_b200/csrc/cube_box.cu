// SPDX-License-Identifier: Apache-2.0
// The box passes of the cube filter: running sums in the reference's canonical order
// (cpp/src/field/vhgw.cu:1-36 of eda-cuda). The extended line is cut into segments of wa = 2r + 1
// samples; a segment's prefix sum G is folded in 32-sample chunks, sequentially inside a chunk and
// over the chunk totals, H is G of the reversed line, and y(x) = H(x - r) + G(x + r) (an output
// whose window is a whole segment takes (H + G) * 0.5).
//
// Every chunk of both directions is folded on its own (the prefix sums of its samples into the
// output slots of H and of G, its total into a table); segments of several chunks then sum their
// carries in chunk order, added to the slots (rows) or by the store (panels, whose outputs share a
// segment over a row); the store takes H + G, the cube's scale and epilogue. So both directions fold
// at once, each sample once per direction, in chains of at most 32 additions, and a pass has two
// barriers (three or four with carries).
// What bounds it: the fold phase's shared-memory round trips (one read and one write per sample and
// direction), issue slots (50 to 60 warp instructions per 32 samples, 80 to 120 with carries) and the
// barriers between the phases. A pass of 64 fields of 512 x 512 float32, panels / rows: 49 / 44 us at
// windows of 15, 59 / 60 us at 63, 71 / 80 us at 255 (74 / 63, 83 / 76 and 124 / 122 us when H and G
// were folded one after the other and the totals in a pass of their own); 134 MB move, 21 us at the
// copy rate. Segments are an odd number of samples long, so the lanes of a warp, on the same chunk of
// consecutive segments, lie in distinct banks.
#include "cube.cuh"

#include <algorithm>
#include <type_traits>

namespace edab {
namespace cubes {
namespace {

// The fold tasks (segment k, chunk c) of one worker, chunk-major (u = c nseg + k, u = first,
// first + stride, ..): the workers of a warp take the same chunk of consecutive segments (wa
// samples apart, spreading their shared-memory banks). Advanced without divisions.
struct Tasks {
  int32_t k, c, dk, dc;
  __device__ __forceinline__ Tasks(int32_t first, int32_t stride, int32_t nseg) {
    if (nseg > stride) {  // first < stride: no division
      k = first;
      c = 0;
      dk = stride;
      dc = 0;
    } else {
      k = first % nseg;
      c = first / nseg;
      dk = stride % nseg;
      dc = stride / nseg;
    }
  }
  __device__ __forceinline__ void next(int32_t nseg) {
    k += dk;
    c += dc;
    if (k >= nseg) {
      k -= nseg;
      ++c;
    }
  }
};

// The prefix sums of len <= 32 samples v[0], v[STEP], .. into o (the same steps), samples before
// `skip` without an output; returns the total.
template <class T, int STEP>
__device__ __forceinline__ T fold_line(const T* v, T* o, int32_t len, int32_t skip) {
  if (len == 32 && skip == 0) {
    T loc = v[0];
    o[0] = loc;
    T x[8];
#pragma unroll
    for (int u = 0; u < 7; ++u) x[u] = v[(u + 1) * STEP];
#pragma unroll
    for (int s = 1; s < 32; ++s) {
      const T cur = x[(s - 1) & 7];
      if (s + 7 < 32) x[(s + 6) & 7] = v[(s + 7) * STEP];
      loc = add_rn(loc, cur);
      o[s * STEP] = loc;
    }
    return loc;
  }
  T loc = v[0];
  if (skip == 0) o[0] = loc;
  int32_t i = 1;
  const int32_t pre = min(skip, len);
  for (; i < pre; ++i) loc = add_rn(loc, v[i * STEP]);
  for (; i + 3 < len; i += 4) {
    T x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) x[u] = v[(i + u) * STEP];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      loc = add_rn(loc, x[u]);
      o[(i + u) * STEP] = loc;
    }
  }
  for (; i < len; ++i) {
    loc = add_rn(loc, v[i * STEP]);
    o[i * STEP] = loc;
  }
  return loc;
}

// The same for positions c0 .. c1 of the extended line in direction dir that reach beyond the line.
template <class T>
__device__ __forceinline__ T fold_reflected(const T* V, T* L, int32_t PP, int32_t n, int32_t r, int32_t c0, int32_t c1,
                                            int dir) {
  T loc = T(-0.0);  // -0 + x == x
  for (int32_t e = c0; e <= c1; ++e) {
    const int32_t i = reflect_index(e, n);
    loc = add_rn(loc, V[(dir ? n - 1 - i : i) * PP]);
    if (e >= r) L[(dir ? n - 1 + r - e : e - r) * PP] = loc;
  }
  return loc;
}

// o[i] = carry + o[i] for the samples skip <= i < len <= 32.
template <class T, int STEP>
__device__ __forceinline__ void add_carry(T* o, int32_t len, int32_t skip, T carry) {
  int32_t i = skip;
  for (; i + 8 <= len; i += 8) {
    T x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = o[(i + u) * STEP];
#pragma unroll
    for (int u = 0; u < 8; ++u) o[(i + u) * STEP] = add_rn(carry, x[u]);
  }
  for (; i < len; ++i) o[i * STEP] = add_rn(carry, o[i * STEP]);
}

// Box cubes run the outer axes first: a panel pass stores the sums, a row pass is the cube's last and
// applies its scale and epilogue.
template <class T, int P, bool ROWS>
__global__ void __launch_bounds__(kCubeThreads, kCubeCtas) box_pass(Geom g, PassArgs<T> a) {
  constexpr int VW = 16 / static_cast<int>(sizeof(T));
  constexpr int PP = ROWS ? 1 : P;                // sample stride in shared memory
  constexpr int W = !ROWS && P >= VW ? VW : 1;  // columns of one access
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ Win win_s[kMaxRungs];
  __shared__ uint32_t inv_s[kMaxRungs];
  __shared__ T fac_s[kMaxRungs];
  const int64_t b = blockIdx.y;
  const int32_t n = elem_n(g, b, a.axis);
  const uint32_t inner = ROWS ? 1u : static_cast<uint32_t>(geom_stride(g, a.axis));
  const int lp = ROWS && P != 8 ? a.lp : (P == 8 ? 3 : (P == 4 ? 2 : (P == 2 ? 1 : 0)));
  const int lines = 1 << lp;
  const int32_t LS = ROWS ? row_stride<T>(n) : 1;
  const int32_t gel = ROWS ? lines * LS : ((n * P + 3) & ~3);
  const int32_t TS = tot_slots(n);
  const int32_t j_begin = static_cast<int32_t>(blockIdx.z) * a.zr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // every warp looks its rungs' windows up (no barrier before the staging starts)
  const int32_t w = lane < a.zr ? a.win[static_cast<int64_t>(j_begin + lane) * g.batch + b] : 0;
  if (__ballot_sync(0xffffffffu, w >= 1) == 0u || (a.epi.run && !a.epi.run[b])) return;
  const GroupPos pos = group_at<ROWS>(g, blockIdx.x, n, inner, static_cast<uint32_t>(lines), a.panels);
  if (!pos.mask) return;
  const int64_t eoff = b * g.field;
  T* V = reinterpret_cast<T*>(smem_raw);
  T* LH = V + gel;
  T* LG = LH + gel;
  T* tot = LG + gel;  // [2][TS][lines]
  stage_lines<T, P, ROWS>(g, a, V, a.bits ? nullptr : a.in0 + j_begin * a.in_stride + eoff,
                          a.bits ? a.bits + eoff : nullptr, pos, n, LS, inner);
  if (warp == 0 && lane < a.zr) {  // the window set-up, while the copies are under way
    Win q{};
    if (w >= 1) {
      q = make_win(n, w);
      inv_s[lane] = 0xffffffffu / static_cast<uint32_t>(q.wa) + 1u;
      if (ROWS) {
        double prod = 1.0;
#pragma unroll
        for (int ax = 0; ax < kMaxDim; ++ax) {
          if (ax < g.dim) prod *= static_cast<double>(2 * min((w - 1) / 2, (g.len ? n : g.n[ax]) - 1) + 1);
        }
        fac_s[lane] = static_cast<T>(1.0 / prod);
      }
    }
    win_s[lane] = q;  // wa == 0: the rung skips this element
  }
  stage_wait();
  __syncthreads();
  const int p = lane & (lines - 1);
  const int workers = kCubeThreads >> lp;
  const int worker = static_cast<int>(threadIdx.x) >> lp;
  const T* Vp = V + (ROWS ? p * LS : p);
  unsigned long long outputs = 0;
  for (int32_t jj = 0; jj < a.zr; ++jj) {
    const Win q = win_s[jj];
    if (q.wa == 0) continue;
    const int32_t e_max = n - 1 + q.r;
    if (q.wa > 1) {
      // chunks of both directions: half of the workers take the line, half the reversed line
      const int half = workers >> 1;
      const int dir = worker >= half;
      T* Lp = (dir ? LH : LG) + (ROWS ? p * LS : p);
      if (q.cps == 1) {
        int32_t s = q.o + (q.k_lo + worker - dir * half) * q.wa;
        const int32_t ds = half * q.wa;
        for (int32_t k = worker - dir * half; k < q.nseg; k += half, s += ds) {
          const int32_t c1 = min(s + q.wa - 1, e_max);
          if (s < 0 || c1 > n - 1) fold_reflected<T>(Vp, Lp, PP, n, q.r, s, c1, dir);
          else if (dir) fold_line<T, -PP>(Vp + (n - 1 - s) * PP, Lp + (n - 1 + q.r - s) * PP, c1 - s + 1, max(0, q.r - s));
          else fold_line<T, PP>(Vp + s * PP, Lp + (s - q.r) * PP, c1 - s + 1, max(0, q.r - s));
        }
      } else {
        for (Tasks t(worker - dir * half, half, q.nseg); t.c < q.cps; t.next(q.nseg)) {
          const int32_t s = q.o + (q.k_lo + t.k) * q.wa;
          const int32_t e_last = min(s + q.wa - 1, e_max);
          const int32_t c0 = s + 32 * t.c;
          if (c0 > e_last) continue;
          const int32_t c1 = min(c0 + 31, e_last);
          T total;
          if (c0 < 0 || c1 > n - 1) total = fold_reflected<T>(Vp, Lp, PP, n, q.r, c0, c1, dir);
          else if (dir) total = fold_line<T, -PP>(Vp + (n - 1 - c0) * PP, Lp + (n - 1 + q.r - c0) * PP, c1 - c0 + 1, max(0, q.r - c0));
          else total = fold_line<T, PP>(Vp + c0 * PP, Lp + (c0 - q.r) * PP, c1 - c0 + 1, max(0, q.r - c0));
          tot[((dir ? TS : 0) + t.k * q.cps + t.c) * lines + p] = total;
        }
      }
      __syncthreads();
      if (q.cps > 1) {
        // exclusive carries per segment, in place (the first chunk's is the identity)
        for (int32_t t = worker; t < 2 * q.nseg; t += workers) {
          const int cd = t >= q.nseg;
          const int32_t k = t - cd * q.nseg;
          const int32_t s = q.o + (q.k_lo + k) * q.wa;
          const int32_t nch = (min(s + q.wa - 1, e_max) - s) / 32 + 1;
          T* tl = tot + ((cd ? TS : 0) + k * q.cps) * lines + p;
          T run = T(-0.0);
          int32_t c = 0;
          for (; c + 8 <= nch; c += 8) {
            T x[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) x[u] = tl[(c + u) * lines];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              tl[(c + u) * lines] = run;
              run = add_rn(run, x[u]);
            }
          }
          for (; c < nch; ++c) {
            const T x = tl[c * lines];
            tl[c * lines] = run;
            run = add_rn(run, x);
          }
        }
        __syncthreads();
        if constexpr (ROWS) {
          // carry + local of every chunk but the segments' first, in place
          for (Tasks t(worker - dir * half, half, q.nseg); t.c + 1 < q.cps; t.next(q.nseg)) {
            const int32_t s = q.o + (q.k_lo + t.k) * q.wa;
            const int32_t e_last = min(s + q.wa - 1, e_max);
            const int32_t c0 = s + 32 * (t.c + 1);
            if (c0 > e_last) continue;
            const int32_t len = min(32, e_last - c0 + 1);
            const T cv = tot[((dir ? TS : 0) + t.k * q.cps + t.c + 1) * lines + p];
            if (dir) add_carry<T, -PP>(Lp + (n - 1 + q.r - c0) * PP, len, max(0, q.r - c0), cv);
            else add_carry<T, PP>(Lp + (c0 - q.r) * PP, len, max(0, q.r - c0), cv);
          }
          __syncthreads();
        }
      }
    }
    // the outputs H + G; an output whose window is a whole segment (x + r is a segment's last sample:
    // u mod wa = wa - 1 for its position u from the first segment's start) takes half of it
    T* out = a.out0 + static_cast<int64_t>(j_begin + jj) * a.out_stride + eoff + pos.base;
    const uint32_t inv = inv_s[jj];
    const int32_t ug = q.r - q.o - q.k_lo * q.wa;
    if constexpr (ROWS) {
      const T* aux = a.epi.aux ? a.epi.aux + eoff + pos.base : nullptr;
      const T fac = fac_s[jj];
      const int per = kWarps >> lp;
      const int pl = warp / per;
      if (pl < lines && ((pos.mask >> pl) & 1u)) {
        const auto line_out = [&](auto kind) {  // (the epilogue is chosen outside the loop)
          constexpr BoxEpi EPI = decltype(kind)::value;
          BoxStore<T, EPI> fin;
          fin.element(a, b, fac);
          T* o = out + static_cast<int64_t>(pl) * g.pitch;
          const T* ax = aux ? aux + static_cast<int64_t>(pl) * g.pitch : nullptr;
          const T* Hr = (q.wa == 1 ? V : LH) + pl * LS;
          const T* Gr = (q.wa == 1 ? V : LG) + pl * LS;
          const int32_t pitch = static_cast<int32_t>(g.pitch), dx = 32 * per * VW;
          // the distance to the next whole segment's output, advanced without divisions (one sample
          // windows: every output is one)
          int32_t x = (lane + 32 * (warp - pl * per)) * VW;
          const int32_t skip = q.wa == 1 ? 0 : dx - static_cast<int32_t>(__umulhi(dx, inv)) * q.wa;
          int32_t whole = q.wa == 1 ? 0 : q.wa - 1 - (x + ug - static_cast<int32_t>(__umulhi(x + ug, inv)) * q.wa);
          for (; x < pitch; x += dx) {
            Pack<T, VW> y;
            if (x < n) {
              const Pack<T, VW> h = load_pack<T, VW>(Hr + x), l = load_pack<T, VW>(Gr + x);
              Pack<T, VW> av{};
              if constexpr (EPI == BoxEpi::kDetSq) av = load_pack<T, VW>(ax + x);
              else if constexpr (EPI == BoxEpi::kRho) {
                if (ax) av = load_pack<T, VW>(ax + x);
              }
#pragma unroll
              for (int k = 0; k < VW; ++k) y.v[k] = add_rn(h.v[k], l.v[k]);
              if (whole < VW) {  // (a second one in the same access: wa == 1, or wa == 3 at 0 and 3)
#pragma unroll
                for (int k = 0; k < VW; ++k) {
                  if (k == whole || q.wa == 1 || (k == 3 && whole == 0 && q.wa == 3)) y.v[k] = mul_rn(y.v[k], T(0.5));
                }
              }
#pragma unroll
              for (int k = 0; k < VW; ++k) y.v[k] = fin(a, b, y.v[k], av.v[k], x + k < n);
            }
            if (x + VW > n) {
#pragma unroll
              for (int k = 0; k < VW; ++k) y.v[k] = x + k < n ? y.v[k] : T(0);
            }
            store_pack<T, VW>(o + x, y);
            whole -= skip;
            if (whole < 0) whole += q.wa;
          }
        };
        switch (a.epi.kind) {
          case BoxEpi::kDetSq: line_out(std::integral_constant<BoxEpi, BoxEpi::kDetSq>{}); break;
          case BoxEpi::kTau: line_out(std::integral_constant<BoxEpi, BoxEpi::kTau>{}); break;
          case BoxEpi::kRho: line_out(std::integral_constant<BoxEpi, BoxEpi::kRho>{}); break;
          case BoxEpi::kClip: line_out(std::integral_constant<BoxEpi, BoxEpi::kClip>{}); break;
          case BoxEpi::kExp: line_out(std::integral_constant<BoxEpi, BoxEpi::kExp>{}); break;
          default: line_out(std::integral_constant<BoxEpi, BoxEpi::kStore>{}); break;
        }
      }
    } else {
      constexpr int QP = P / W;
      const int c = (threadIdx.x % QP) * W;
      T* o = out + static_cast<int64_t>(threadIdx.x / QP) * inner + c;
      const int64_t step = static_cast<int64_t>(kCubeThreads / QP) * inner;
      const uint32_t live = pos.mask >> c;  // columns left of the row padding
      const auto panel_out = [&](auto form) {  // 0: one-sample windows, 1: one chunk a segment, 2: carries
        constexpr int FORM = decltype(form)::value;
        const int32_t uh = n - 1 + ug;
        for (int32_t x = threadIdx.x / QP; x < n; x += kCubeThreads / QP, o += step) {
          Pack<T, W> y;
          if constexpr (FORM == 0) {
            const Pack<T, W> v = load_pack<T, W>(V + x * P + c);
#pragma unroll
            for (int k = 0; k < W; ++k) y.v[k] = mul_rn(add_rn(v.v[k], v.v[k]), T(0.5));
          } else {
            Pack<T, W> h = load_pack<T, W>(LH + x * P + c), l = load_pack<T, W>(LG + x * P + c);
            const int32_t kg = static_cast<int32_t>(__umulhi(x + ug, inv));
            const int32_t mg = x + ug - kg * q.wa;
            if constexpr (FORM == 2) {
              const int32_t kh = static_cast<int32_t>(__umulhi(uh - x, inv));
              const int32_t mh = uh - x - kh * q.wa;
              const Pack<T, W> cg = load_pack<T, W>(tot + (kg * q.cps + (mg >> 5)) * P + c);
              const Pack<T, W> ch = load_pack<T, W>(tot + (TS + kh * q.cps + (mh >> 5)) * P + c);
#pragma unroll
              for (int k = 0; k < W; ++k) {
                h.v[k] = add_rn(ch.v[k], h.v[k]);
                l.v[k] = add_rn(cg.v[k], l.v[k]);
              }
            }
#pragma unroll
            for (int k = 0; k < W; ++k) y.v[k] = add_rn(h.v[k], l.v[k]);
            if (mg == q.wa - 1) {
#pragma unroll
              for (int k = 0; k < W; ++k) y.v[k] = mul_rn(y.v[k], T(0.5));
            }
          }
#pragma unroll
          for (int k = 0; k < W; ++k) y.v[k] = ((live >> k) & 1u) ? y.v[k] : T(0);
          store_pack<T, W>(o, y);
        }
      };
      if (q.wa == 1) panel_out(std::integral_constant<int, 0>{});
      else if (q.cps == 1) panel_out(std::integral_constant<int, 1>{});
      else panel_out(std::integral_constant<int, 2>{});
    }
    ++outputs;
    if (jj + 1 < a.zr) __syncthreads();  // the next rung rewrites the slots and totals
  }
  if (a.bytes && threadIdx.x == 0) {
    const unsigned long long samples = static_cast<unsigned long long>(__popc(pos.mask)) * n;
    atomicAdd(a.bytes, samples * (a.bits ? 1u : sizeof(T)) + outputs * samples * sizeof(T));
  }
}

}  // namespace

size_t box_smem_bytes(int32_t n, int P, bool rows, size_t es) {
  const int32_t gel = es == 4 ? group_elems<float>(n, P, rows) : group_elems<double>(n, P, rows);
  return (static_cast<size_t>(3) * gel + static_cast<size_t>(2) * tot_slots(n) * P) * es;
}

template <class T>
void box_allow_smem(int bytes) {
  EDAB_CUDA(cudaFuncSetAttribute(box_pass<T, 8, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  EDAB_CUDA(cudaFuncSetAttribute(box_pass<T, 1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  EDAB_CUDA(cudaFuncSetAttribute(box_pass<T, 1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  EDAB_CUDA(cudaFuncSetAttribute(box_pass<T, 2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  EDAB_CUDA(cudaFuncSetAttribute(box_pass<T, 4, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  EDAB_CUDA(cudaFuncSetAttribute(box_pass<T, 8, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}

template <class T>
void launch_box(cudaStream_t s, const Geom& g, const PassArgs<T>& a, int P, bool rows, dim3 grid, size_t smem) {
  if (rows && P == 8) enqueue(box_pass<T, 8, true>, grid, kCubeThreads, smem, s, g, a);
  else if (rows) enqueue(box_pass<T, 1, true>, grid, kCubeThreads, smem, s, g, a);
  else if (P == 1) enqueue(box_pass<T, 1, false>, grid, kCubeThreads, smem, s, g, a);
  else if (P == 2) enqueue(box_pass<T, 2, false>, grid, kCubeThreads, smem, s, g, a);
  else if (P == 4) enqueue(box_pass<T, 4, false>, grid, kCubeThreads, smem, s, g, a);
  else enqueue(box_pass<T, 8, false>, grid, kCubeThreads, smem, s, g, a);
}

template void box_allow_smem<float>(int);
template void box_allow_smem<double>(int);
template void launch_box<float>(cudaStream_t, const Geom&, const PassArgs<float>&, int, bool, dim3, size_t);
template void launch_box<double>(cudaStream_t, const Geom&, const PassArgs<double>&, int, bool, dim3, size_t);

}  // namespace cubes
}  // namespace edab
