// SPDX-License-Identifier: Apache-2.0
// The cube filter's passes over 1-D lines too long for one CTA: the line's samples (order keys for
// max / min) are written once per call into a scratch, with what a tile needs of the rest of the
// line, and the outputs are cut into tiles, one CTA per tile, rung and field. Every bit is that of
// the staged passes (cube_ext.cu, cube_box.cu).
//
// Max / min: the scratch holds the extreme of every 32-sample block. A tile computes the block
// suffixes H where its windows begin and the block prefixes G where they end (a lane per block, in shared
// memory: three instructions per sample of 32 lanes; by warp shuffles they were twenty), doubles the
// extremes of the blocks that its windows reach to runs of 2^k blocks, two of which cover the blocks
// between, and takes four reads per output whatever the window. Two launches.
// Box sums: a tile folds the 32-sample chunks where its windows begin (H, the reversed line) and end
// (G). Short segments (at most a quarter tile) are folded from their start inside the tile; the
// carries of longer ones come from a table of the line's chunk totals, summed per segment in chunk
// order by the last CTA of the totals' launch. Two launches, three where the samples have to be copied
// (bit fields, outputs over the input).
// What bounds them: at small batches the launches themselves, else the output loops' issue slots and
// the folds' shared-memory round trips; the samples lie in L2 after the first launch. A batch of 1024
// signals of 256 to 65 536 float32 samples: max and min 147 -> 89 us per launch, the copies 25.6 -> 15.2 ms
// in all, box sums 88 -> 80 us (tiles of 2048 outputs: 76 us, but the totals 29 -> 37 us). Totals from
// coalesced tiles instead of a lane per chunk: 31 us either way, float64 6.4 -> 9.2 us; not kept.
#include "cube.cuh"

#include <algorithm>
#include <type_traits>

namespace edab {
namespace cubes {
namespace {

// The scratch: the lines' samples or keys [B][pitch] and per field (max; min as the complements' max)
// the blocks' extremes [2][B][pitch / 32]; apart from them the chunk totals [rungs][B][2][TSL] and the
// counts of the totals' CTAs that are done [rungs][B].
template <class T>
struct LongScratch {
  T* line;
  typename KeyType<T>::type* blocks;
  T* tot;
  int32_t* done;
  int32_t TSL;
};

// Every sample of every line; a warp takes 32 consecutive samples.
template <class T>
__global__ void __launch_bounds__(kThreads) long_input(Geom g, PassArgs<T> a, LongScratch<T> L, int32_t counters) {
  using K = typename KeyType<T>::type;
  const bool box = a.op == static_cast<int>(CubeOp::kBox);
  const int64_t b = blockIdx.y;
  const int32_t n = elem_len(g, b);
  const int32_t nbp = static_cast<int32_t>(g.pitch >> 5);
  if (blockIdx.x == 0 && b == 0) {
    for (int32_t i = threadIdx.x; i < counters; i += kThreads) L.done[i] = 0;
  }
  for (int32_t i = static_cast<int32_t>(blockIdx.x * kThreads + threadIdx.x); i < g.pitch;
       i += static_cast<int32_t>(gridDim.x) * kThreads) {
    const int64_t at = b * g.field + i;
    T v;
    if (a.bits) v = ((a.bits[at] >> a.bit) & 1u) ? T(1) : T(0);
    else v = a.in0[at];
    if (box) {
      L.line[at] = v;
      continue;
    }
    const K key = okey_i(v);
    reinterpret_cast<K*>(L.line)[at] = key;
    K hi = i < n ? key : key_min<K>(), lo = i < n ? ~key : key_min<K>();
    if constexpr (sizeof(K) == 4) {
      hi = __reduce_max_sync(0xffffffffu, hi);
      lo = __reduce_max_sync(0xffffffffu, lo);
    } else {
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) {
        hi = max(hi, static_cast<K>(__shfl_xor_sync(0xffffffffu, hi, d)));
        lo = max(lo, static_cast<K>(__shfl_xor_sync(0xffffffffu, lo, d)));
      }
    }
    if ((threadIdx.x & 31) == 0) {
      L.blocks[b * nbp + (i >> 5)] = hi;
      L.blocks[(g.batch + b) * nbp + (i >> 5)] = lo;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// max / min

// The block length of half width r: B <= 2r, at most 32.
__device__ __forceinline__ int32_t long_block(int32_t r) { return r >= 16 ? 32 : 2 << (31 - __clz(max(r, 1))); }

// A staged sample's word: a lane's 32 samples lie one word further than its neighbour's.
__host__ __device__ constexpr int32_t padded(int32_t i) { return i + (i >> 5); }
// Words of the samples that a tile stages where its windows begin, or end.
__host__ __device__ constexpr int32_t ext_words(int32_t tile) { return padded(tile + 128); }

// The extremes of the 32 staged samples at x (32 words) from each to its block's end (DOWN) or from its
// block's start on, in place.
template <bool DOWN, class K>
__device__ __forceinline__ void scan_blocks(K* x, int32_t B) {
  K v = key_min<K>();
#pragma unroll
  for (int u = 0; u < 32; ++u) {
    const int i = DOWN ? 31 - u : u;
    if (B < 32 && (u & (B - 1)) == 0) v = key_min<K>();
    v = max(v, x[i]);
    x[i] = v;
  }
}

// dynamic shared memory: H, G [ext_words], S0, S1, PB [nbp]
template <class T>
__global__ void __launch_bounds__(kThreads) long_ext(Geom g, PassArgs<T> a, LongScratch<T> L, int32_t tile) {
  using K = typename KeyType<T>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ K warp_max[kThreads / 32];
  const int64_t b = blockIdx.y;
  const int nf = a.op == static_cast<int>(CubeOp::kMaxMin) ? 2 : 1;
  const int32_t j = static_cast<int32_t>(blockIdx.z) / nf;
  const int f = static_cast<int>(blockIdx.z) % nf;
  const int32_t n = elem_len(g, b);
  const int32_t X0 = static_cast<int32_t>(blockIdx.x) * tile;
  if (X0 >= n) return;
  const int32_t w = a.win[static_cast<int64_t>(j) * g.batch + b];
  if (w < 1) return;
  const int32_t X1 = min(X0 + tile, n);
  const int32_t r = min((w - 1) >> 1, n - 1);
  const bool is_min = a.op == static_cast<int>(CubeOp::kMin) || f == 1;
  const K nm = is_min ? static_cast<K>(-1) : static_cast<K>(0);
  const K idn = key_min<K>();
  const K* line = reinterpret_cast<const K*>(L.line) + b * g.field;
  T* out = (f == 0 ? a.out0 : a.out1) + static_cast<int64_t>(j) * a.out_stride + b * g.field;
  const int32_t end = X1 == n ? static_cast<int32_t>(g.pitch) : X1;  // the last tile writes the pads
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (r == 0) {
    for (int32_t x = X0 + threadIdx.x; x < end; x += kThreads) out[x] = x < n ? key_back(line[x]) : T(0);
    return;
  }
  const int32_t span = ext_words(tile), nbp = static_cast<int32_t>(g.pitch >> 5);
  K* H = reinterpret_cast<K*>(smem_raw);
  K* G = H + span;
  K* S = G + span;
  K* S2 = S + nbp;
  K* PB = S2 + nbp;
  const int32_t B = long_block(r), sh = 31 - __clz(B);
  // H from the block of the first window's start to two blocks past the last window's (short blocks: the
  // block between is read from H), G over the blocks of the windows' ends
  const int32_t h0 = max(X0 - r, 0) >> 5 << 5, h1 = min(n, ((max(X1 - 1 - r, 0) + 2 * B) >> 5) * 32 + 32);
  const int32_t g0 = min(X0 + r, n - 1) >> 5 << 5, g1 = min(n, (min(X1 - 1 + r, n - 1) >> 5) * 32 + 32);
  for (int32_t i = h0 + threadIdx.x; i < h1; i += kThreads) H[padded(i - h0)] = line[i] ^ nm;
  for (int32_t i = g0 + threadIdx.x; i < g1; i += kThreads) G[padded(i - g0)] = line[i] ^ nm;
  const int32_t hb = (h1 - h0 + 31) >> 5, gb = (g1 - g0 + 31) >> 5;
  for (int32_t i = h1 + threadIdx.x; i < h0 + 32 * hb; i += kThreads) H[padded(i - h0)] = idn;
  for (int32_t i = g1 + threadIdx.x; i < g0 + 32 * gb; i += kThreads) G[padded(i - g0)] = idn;
  // the blocks that the tile's windows reach, and their extremes (B == 32)
  const int32_t bs = max(X0 - r, 0) >> 5, be = (min(X1 - 1 + r, n - 1) >> 5) + 1;
  if (B == 32) {
    const K* from = L.blocks + (is_min ? g.batch + b : b) * nbp;
    for (int32_t i = bs + threadIdx.x; i < be; i += kThreads) S[i] = from[i];
  }
  __syncthreads();
  for (int32_t t = threadIdx.x; t < hb + gb; t += kThreads) {
    if (t < hb) scan_blocks<true>(H + 33 * t, B);
    else scan_blocks<false>(G + 33 * (t - hb), B);
  }
  int32_t run = 0;  // B == 32: S holds the extremes of runs of 2^run blocks
  if (B == 32) {
    if (X0 < r) {  // some windows begin before the line: the extremes of the blocks up to each
      const int32_t per = (be + kThreads - 1) / kThreads;
      const int32_t c0 = min(static_cast<int32_t>(threadIdx.x) * per, be), c1 = min(c0 + per, be);
      K run_max = idn;
      for (int32_t i = c0; i < c1; ++i) run_max = max(run_max, S[i]);
      K scan = run_max;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const K o = __shfl_up_sync(0xffffffffu, scan, d);
        if (lane >= d) scan = max(scan, o);
      }
      if (lane == 31) warp_max[warp] = scan;
      __syncthreads();
      K before = __shfl_up_sync(0xffffffffu, scan, 1);
      if (lane == 0) before = idn;
      for (int u = 0; u < warp; ++u) before = max(before, warp_max[u]);
      for (int32_t i = c0; i < c1; ++i) {
        before = max(before, S[i]);
        PB[i] = before;
      }
    }
    const int32_t least = (r >> 4) - 1;  // whole blocks that every window inside the line holds
    while ((2 << run) <= least) {
      const int32_t half = 1 << run;
      for (int32_t i = bs + threadIdx.x; i < be; i += kThreads) S2[i] = max(S[i], S[min(i + half, be - 1)]);
      __syncthreads();
      K* t = S;
      S = S2;
      S2 = t;
      ++run;
    }
  }
  __syncthreads();
  for (int32_t x = X0 + threadIdx.x; x < end; x += kThreads) {
    T res = T(0);
    if (x < n) {
      const int32_t lo = x - r, hi = min(x + r, n - 1);
      const int32_t b0 = lo >= 0 ? lo >> sh : -1, b1 = hi >> sh;
      K y = lo >= 0 ? H[padded(lo - h0)] : idn;
      if (b1 > b0) y = max(y, G[padded(hi - g0)]);
      if (b1 - b0 > 1) {
        if (B < 32) y = max(y, H[padded(((b0 + 1) << sh) - h0)]);
        else if (lo < 0) y = max(y, PB[b1 - 1]);
        else y = max(y, max(S[b0 + 1], S[max(b0 + 1, b1 - (1 << run))]));
      }
      res = key_back(static_cast<K>(y ^ nm));
    }
    out[x] = res;
  }
  if (a.bytes && threadIdx.x == 0) {
    atomicAdd(a.bytes, static_cast<unsigned long long>(X1 - X0) * sizeof(T) * (f == 0 ? 2 : 1));
  }
}

// ---------------------------------------------------------------------------------------------
// box sums

// Whether window q takes its carries from the table of chunk totals.
__device__ __forceinline__ bool long_wide(const Win& q, int32_t tile) { return q.wa > tile / 4; }

// The prefix sums of the chunk's samples in place (at i + i / 32: the lanes of a warp, on consecutive
// chunks, lie in distinct banks); returns the total.
template <class T>
__device__ __forceinline__ T fold_padded(T* R, int32_t i0, int32_t len) {
  T loc = T(-0.0);  // -0 + x == x
  int32_t i = i0;
  const int32_t end = i0 + len;
  for (; i + 4 <= end; i += 4) {
    T x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) x[u] = R[i + u + ((i + u) >> 5)];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      loc = add_rn(loc, x[u]);
      R[i + u + ((i + u) >> 5)] = loc;
    }
  }
  for (; i < end; ++i) {
    loc = add_rn(loc, R[i + (i >> 5)]);
    R[i + (i >> 5)] = loc;
  }
  return loc;
}

// The chunk totals of the wide windows, task t < 2 nseg cps = (direction, segment, chunk); the last CTA
// of a rung and element then sums the exclusive carries of every segment, in chunk order, in place.
// dynamic shared memory: the carries' staging [2 TSL]
template <class T>
__global__ void __launch_bounds__(kThreads) long_totals(Geom g, PassArgs<T> a, LongScratch<T> L, int32_t tile) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int32_t last_s;
  const int64_t b = blockIdx.y;
  const int32_t j = static_cast<int32_t>(blockIdx.z);
  const int32_t w = a.win[static_cast<int64_t>(j) * g.batch + b];
  if (w < 1 || (a.epi.run && !a.epi.run[b])) return;
  const int32_t n = elem_len(g, b);
  const Win q = make_win(n, w);
  if (!long_wide(q, tile)) return;
  const int32_t per_dir = q.nseg * q.cps, e_max = n - 1 + q.r;
  if (per_dir > L.TSL) return;  // (never: nseg cps <= tot_slots(n) for windows of several chunks)
  const T* V = L.line + b * g.field;
  T* tot = L.tot + ((static_cast<int64_t>(j) * g.batch + b) * 2) * L.TSL;
  for (int32_t t = static_cast<int32_t>(blockIdx.x * kThreads + threadIdx.x); t < 2 * per_dir;
       t += static_cast<int32_t>(gridDim.x) * kThreads) {
    const int dir = t >= per_dir;
    const int32_t kc = t - dir * per_dir;
    const int32_t k = kc / q.cps, c = kc - k * q.cps;
    const int32_t s = q.o + (q.k_lo + k) * q.wa;
    const int32_t c0 = s + 32 * c, c1 = min(min(c0 + 31, s + q.wa - 1), e_max);
    if (c0 > c1) continue;
    T loc = T(-0.0);
    if (c0 >= 0 && c1 == c0 + 31 && c1 < n) {
      const T* v = V + (dir ? n - 1 - c0 : c0);
      T x[32];
#pragma unroll
      for (int u = 0; u < 32; ++u) x[u] = dir ? v[-u] : v[u];
#pragma unroll
      for (int u = 0; u < 32; ++u) loc = add_rn(loc, x[u]);
    } else {
      for (int32_t e = c0; e <= c1; ++e) {
        const int32_t i = reflect_index(e, n);
        loc = add_rn(loc, V[dir ? n - 1 - i : i]);
      }
    }
    tot[dir * L.TSL + kc] = loc;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last_s = atomicAdd(&L.done[static_cast<int64_t>(j) * g.batch + b], 1) == static_cast<int32_t>(gridDim.x) - 1;
  }
  __syncthreads();
  if (!last_s) return;
  __threadfence();
  T* st = reinterpret_cast<T*>(smem_raw);
  for (int32_t i = threadIdx.x; i < 2 * per_dir; i += kThreads) {
    const int dir = i >= per_dir;
    st[i] = __ldcg(tot + dir * L.TSL + (i - dir * per_dir));
  }
  __syncthreads();
  for (int32_t t = threadIdx.x; t < 2 * q.nseg; t += kThreads) {
    const int dir = t >= q.nseg;
    const int32_t k = t - dir * q.nseg;
    const int32_t s = q.o + (q.k_lo + k) * q.wa;
    const int32_t nch = (min(s + q.wa - 1, e_max) - s) / 32 + 1;
    T* tl = st + dir * per_dir + k * q.cps;
    T run = T(-0.0);
    int32_t c = 0;
    for (; c + 8 <= nch; c += 8) {
      T x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = tl[c + u];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        tl[c + u] = run;
        run = add_rn(run, x[u]);
      }
    }
    for (; c < nch; ++c) {
      const T x = tl[c];
      tl[c] = run;
      run = add_rn(run, x);
    }
  }
  __syncthreads();
  for (int32_t i = threadIdx.x; i < 2 * per_dir; i += kThreads) {
    const int dir = i >= per_dir;
    tot[dir * L.TSL + (i - dir * per_dir)] = st[i];
  }
}

// One direction of a tile: the extended positions [p0, p1] that its outputs read, from the segment or
// chunk start e0 on.
struct LongSide {
  int32_t k0;      // the first segment (relative to k_lo)
  int32_t c_skip;  // its chunks before e0 (wide windows)
  int32_t e0, len, chunks;
};
__host__ __device__ inline LongSide long_side(int32_t wa, int32_t cps, int32_t first, int32_t p0, int32_t p1,
                                              bool wide) {
  LongSide s;
  s.k0 = (p0 - first) / wa;
  const int32_t in0 = p0 - first - s.k0 * wa;
  s.c_skip = wide ? in0 >> 5 : 0;
  s.e0 = first + s.k0 * wa + 32 * s.c_skip;
  s.len = p1 - s.e0 + 1;
  const int32_t k1 = (p1 - first) / wa;
  s.chunks = (k1 - s.k0) * cps + ((p1 - first - k1 * wa) >> 5) - s.c_skip + 1;
  return s;
}

// Samples a side of a tile stages, and its chunks, at most: from a segment's start (short segments, at
// most tile / 4 samples) or a chunk's.
__host__ __device__ constexpr int32_t side_samples(int32_t tile) { return tile + tile / 4 + 32; }
__host__ __device__ constexpr int32_t side_chunks(int32_t tile) { return side_samples(tile) / 2 + 8; }
__host__ __device__ constexpr int32_t side_words(int32_t tile) { return side_samples(tile) + side_samples(tile) / 32 + 4; }

// dynamic shared memory: G, H samples (side_words each), then their chunks' totals (side_chunks each)
template <class T>
__global__ void __launch_bounds__(kThreads) long_box(Geom g, PassArgs<T> a, LongScratch<T> L, int32_t tile) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int64_t b = blockIdx.y;
  const int32_t j = static_cast<int32_t>(blockIdx.z);
  const int32_t n = elem_len(g, b);
  const int32_t X0 = static_cast<int32_t>(blockIdx.x) * tile;
  if (X0 >= n) return;
  const int32_t w = a.win[static_cast<int64_t>(j) * g.batch + b];
  if (w < 1 || (a.epi.run && !a.epi.run[b])) return;
  const int32_t X1 = min(X0 + tile, n);
  const Win q = make_win(n, w);
  const T* line = L.line + b * g.field;
  const T* aux = a.epi.aux ? a.epi.aux + b * g.field : nullptr;
  T* out = a.out0 + static_cast<int64_t>(j) * a.out_stride + b * g.field;
  const T fac = static_cast<T>(1.0 / static_cast<double>(q.wa));
  const int32_t end = X1 == n ? static_cast<int32_t>(g.pitch) : X1;  // the last tile writes the pads
  // the sums y(x), each stored with the cube's scale and epilogue (chosen outside the loop)
  const auto tile_out = [&](const auto& sum) {
    const auto with = [&](auto kind) {
      constexpr BoxEpi EPI = decltype(kind)::value;
      BoxStore<T, EPI> fin;
      fin.element(a, b, fac);
      for (int32_t x = X0 + threadIdx.x; x < end; x += kThreads) {
        out[x] = x < n ? fin(a, b, sum(x), aux ? aux[x] : T(0), true) : T(0);
      }
    };
    switch (a.epi.kind) {
      case BoxEpi::kDetSq: with(std::integral_constant<BoxEpi, BoxEpi::kDetSq>{}); break;
      case BoxEpi::kTau: with(std::integral_constant<BoxEpi, BoxEpi::kTau>{}); break;
      case BoxEpi::kRho: with(std::integral_constant<BoxEpi, BoxEpi::kRho>{}); break;
      case BoxEpi::kClip: with(std::integral_constant<BoxEpi, BoxEpi::kClip>{}); break;
      case BoxEpi::kExp: with(std::integral_constant<BoxEpi, BoxEpi::kExp>{}); break;
      default: with(std::integral_constant<BoxEpi, BoxEpi::kStore>{}); break;
    }
  };
  if (q.wa == 1) {
    tile_out([&](int32_t x) { return mul_rn(add_rn(line[x], line[x]), T(0.5)); });
    return;
  }
  const bool wide = long_wide(q, tile);
  const int32_t first = q.o + q.k_lo * q.wa, e_max = n - 1 + q.r;
  // G at x + r of the line, H at n - 1 - (x - r) of the reversed line
  const LongSide sg = long_side(q.wa, q.cps, first, X0 + q.r, X1 - 1 + q.r, wide);
  const LongSide sh = long_side(q.wa, q.cps, first, n - X1 + q.r, n - 1 - X0 + q.r, wide);
  T* RG = reinterpret_cast<T*>(smem_raw);
  T* RH = RG + side_words(tile);
  T* TG = RH + side_words(tile);
  T* TH = TG + side_chunks(tile);
  // (within the bounds for every length, window and tile, checked on the CPU)
  if (max(sg.len, sh.len) > side_samples(tile) || max(sg.chunks, sh.chunks) > side_chunks(tile)) return;
  if (min(sg.e0, sh.e0) >= 0 && max(sg.e0 + sg.len, sh.e0 + sh.len) <= n) {  // no sample is a reflected one
    const T* from = line + sg.e0;
    for (int32_t i = threadIdx.x; i < sg.len; i += kThreads) RG[padded(i)] = from[i];
    from = line + (n - 1 - sh.e0);
    for (int32_t i = threadIdx.x; i < sh.len; i += kThreads) RH[padded(i)] = from[-i];
  } else {
    for (int32_t i = threadIdx.x; i < sg.len; i += kThreads) RG[padded(i)] = line[reflect_index(sg.e0 + i, n)];
    for (int32_t i = threadIdx.x; i < sh.len; i += kThreads) RH[padded(i)] = line[n - 1 - reflect_index(sh.e0 + i, n)];
  }
  __syncthreads();
  const int32_t all = sg.chunks + sh.chunks;
  for (int32_t t = threadIdx.x; t < all; t += kThreads) {
    const bool rev = t >= sg.chunks;
    const LongSide& s = rev ? sh : sg;
    const int32_t u = (rev ? t - sg.chunks : t) + s.c_skip;
    const int32_t k = u / q.cps, c = u - k * q.cps;
    const int32_t s0 = first + (s.k0 + k) * q.wa;
    const int32_t c0 = s0 + 32 * c, c1 = min(min(c0 + 31, s0 + q.wa - 1), min(e_max, s.e0 + s.len - 1));
    const T total = c1 >= c0 ? fold_padded(rev ? RH : RG, c0 - s.e0, c1 - c0 + 1) : T(-0.0);
    (rev ? TH : TG)[t - (rev ? sg.chunks : 0)] = total;
  }
  __syncthreads();
  if (q.cps > 1 && !wide) {
    // exclusive carries of the tile's segments, in chunk order
    const int32_t ng = (sg.chunks + q.cps - 1) / q.cps, nh = (sh.chunks + q.cps - 1) / q.cps;
    for (int32_t t = threadIdx.x; t < ng + nh; t += kThreads) {
      const bool rev = t >= ng;
      const int32_t k = rev ? t - ng : t;
      T* tl = (rev ? TH : TG) + k * q.cps;
      const int32_t nch = min(q.cps, (rev ? sh.chunks : sg.chunks) - k * q.cps);
      T run = T(-0.0);
      for (int32_t c = 0; c < nch; ++c) {
        const T x = tl[c];
        tl[c] = run;
        run = add_rn(run, x);
      }
    }
    __syncthreads();
  }
  const T* gt = L.tot + ((static_cast<int64_t>(j) * g.batch + b) * 2) * L.TSL;
  const uint32_t inv = 0xffffffffu / static_cast<uint32_t>(q.wa) + 1u;  // exact below tile + tile / 4 for short segments
  // carry + local at extended position e of a side; *at_end: e is its segment's last sample
  const auto side_value = [&](const LongSide& s, const T* R, const T* tl, const T* table, int32_t e, bool* at_end) {
    int32_t m = e - (first + s.k0 * q.wa), k = 0;
    if (wide) {
      while (m >= q.wa) {
        m -= q.wa;
        ++k;
      }
    } else {
      k = static_cast<int32_t>(__umulhi(m, inv));
      m -= k * q.wa;
    }
    *at_end = m == q.wa - 1;
    const int32_t i = e - s.e0;
    const T loc = R[i + (i >> 5)];
    const int32_t c = m >> 5;
    if (c == 0) return loc;
    return add_rn(wide ? table[(s.k0 + k) * q.cps + c] : tl[k * q.cps + c], loc);
  };
  tile_out([&](int32_t x) {
    bool whole, unused;
    const T gv = side_value(sg, RG, TG, gt, x + q.r, &whole);
    const T hv = side_value(sh, RH, TH, gt + L.TSL, n - 1 - x + q.r, &unused);
    const T y = add_rn(hv, gv);
    return whole ? mul_rn(y, T(0.5)) : y;
  });
  if (a.bytes && threadIdx.x == 0) atomicAdd(a.bytes, static_cast<unsigned long long>(X1 - X0) * sizeof(T) * 2);
}

size_t up256(size_t v) { return (v + 255) / 256 * 256; }
size_t line_bytes(const Geom& g, size_t es) { return up256(static_cast<size_t>(g.batch * g.pitch) * es); }

}  // namespace

size_t long_line_part(const Geom& g, size_t es) {
  return line_bytes(g, es) + up256(2 * static_cast<size_t>(g.batch) * static_cast<size_t>(g.pitch / 32) * es);
}
size_t long_totals_part(const Geom& g, size_t es) {
  const size_t B = static_cast<size_t>(g.batch);
  return kMaxRungs * B * 2 * static_cast<size_t>(tot_slots(g.n_last)) * es + kMaxRungs * B * sizeof(int32_t);
}

// Outputs per tile: 4096, or 1024 while those would leave SMs without a CTA.
int32_t long_tile(const Geom& g, int64_t others, int sms) {
  return (g.n_last + 4095) / 4096 * g.batch * others < 2 * sms ? 1024 : 4096;
}

template <class T>
void launch_long(cudaStream_t s, const Geom& g, const PassArgs<T>& a, void* lines, void* totals, int sms, size_t smem_cap) {
  const bool box = a.op == static_cast<int>(CubeOp::kBox);
  const int nf = a.op == static_cast<int>(CubeOp::kMaxMin) ? 2 : 1;
  if (g.batch > 65535) throw std::invalid_argument("edab: cube launch too large");
  LongScratch<T> L;
  L.line = static_cast<T*>(lines);
  L.blocks = reinterpret_cast<typename KeyType<T>::type*>(static_cast<char*>(lines) + line_bytes(g, sizeof(T)));
  L.TSL = tot_slots(g.n_last);
  L.tot = static_cast<T*>(totals);
  L.done = reinterpret_cast<int32_t*>(static_cast<char*>(totals) + static_cast<size_t>(kMaxRungs) * g.batch * 2 * L.TSL * sizeof(T));
  const unsigned B = static_cast<unsigned>(g.batch);
  const unsigned in_x = static_cast<unsigned>(std::clamp<int64_t>((g.pitch + 4 * kThreads - 1) / (4 * kThreads), 1, 64));
  // box sums read their input where it lies, unless it is a bit field or an output overwrites it
  const T* out_end = a.out0 + (a.rungs - 1) * a.out_stride + g.batch * g.field;
  if (box && !a.bits && (a.in0 >= out_end || a.in0 + g.batch * g.field <= a.out0)) {
    L.line = const_cast<T*>(a.in0);
    enqueue_zero(L.done, static_cast<size_t>(a.rungs) * B * sizeof(int32_t), s);
  } else {
    enqueue(long_input<T>, dim3(in_x, B), kThreads, 0, s, g, a, L, box ? a.rungs * static_cast<int32_t>(g.batch) : 0);
  }
  const int32_t tile = long_tile(g, static_cast<int64_t>(a.rungs) * nf, sms);
  const unsigned tiles = static_cast<unsigned>((g.n_last + tile - 1) / tile);
  if (!box) {
    const size_t smem = (static_cast<size_t>(2) * ext_words(tile) + 3 * static_cast<size_t>(g.pitch / 32)) * sizeof(T);
    if (smem > smem_cap) throw std::invalid_argument("edab: a line is too long for the long-line cube pass");
    once_on_device(reinterpret_cast<const void*>(long_ext<T>), [&] {
      EDAB_CUDA(cudaFuncSetAttribute(long_ext<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem_cap)));
    });
    enqueue(long_ext<T>, dim3(tiles, B, static_cast<unsigned>(a.rungs * nf)), kThreads, smem, s, g, a, L, tile);
    return;
  }
  const size_t carries = static_cast<size_t>(2) * L.TSL * sizeof(T);
  const size_t smem = (static_cast<size_t>(2) * side_words(tile) + 2 * side_chunks(tile)) * sizeof(T);
  if (carries > smem_cap || smem > smem_cap) throw std::invalid_argument("edab: a line is too long for the long-line cube pass");
  once_on_device(reinterpret_cast<const void*>(long_box<T>), [&] {
    EDAB_CUDA(cudaFuncSetAttribute(long_totals<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem_cap)));
    EDAB_CUDA(cudaFuncSetAttribute(long_box<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem_cap)));
  });
  const unsigned tx = static_cast<unsigned>(std::clamp<int64_t>((2 * L.TSL / 4 + kThreads - 1) / kThreads, 1, 16));
  enqueue(long_totals<T>, dim3(tx, B, static_cast<unsigned>(a.rungs)), kThreads, carries, s, g, a, L, tile);
  enqueue(long_box<T>, dim3(tiles, B, static_cast<unsigned>(a.rungs)), kThreads, smem, s, g, a, L, tile);
}

template void launch_long<float>(cudaStream_t, const Geom&, const PassArgs<float>&, void*, void*, int, size_t);
template void launch_long<double>(cudaStream_t, const Geom&, const PassArgs<double>&, void*, void*, int, size_t);

}  // namespace cubes
}  // namespace edab
