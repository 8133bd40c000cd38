// SPDX-License-Identifier: Apache-2.0
// The float32 axis transforms of the orientation on the 5th-generation tensor cores (sm_100a):
// out = A B^T per element rows, A the field's rows along its contiguous axis (K = that axis),
// B the n x n basis (forward DCT-II, inverse cosine or inverse sine) of that axis.
//
// Precision: split products with float32 accumulation in tensor memory, the float32 operand x split
// into hi + lo and the product taken as hi_a hi_b + hi_a lo_b + lo_a hi_b (three MMAs; the dropped
// lo_a lo_b term is below 2^-2p of the product). 3xTF32 (kind::tf32): hi = tf32(x), lo =
// tf32(x - hi), about 22 bits of every operand; BF16x3 (kind::f16 on bfloat16): hi = bf16(x), lo =
// bf16(x - hi), about 16 bits, at twice the MMA rate. (The reference runs these transforms with
// cuFFT in float32, cpp/src/method/orientation.cu:674-767 of eda-cuda.) The basis is split once on
// the host; the field tile is split in shared memory after its TMA load.
//
// Kernel (persistent: one CTA of 320 threads per SM runs tiles of 128 rows and 128 or 256 columns in turn):
//   warp 4      TMA producer: A tile (128 rows) and the hi and lo basis tiles per k-block into a ring of
//               3 or 4 stages (full / empty mbarriers);
//   warps 0-3   split the A tile into hi and lo tiles (3xTF32: hi in place; BF16x3: two bfloat16 tiles),
//               fence the async proxy, arrive on the stage's split barrier;
//   warp 5      allocates two accumulators in TMEM; one thread issues the split MMAs of every k-block
//               (kind::tf32 with K = 8, or kind::f16 with K = 16), commits each stage back to the producer
//               and each tile to the epilogue;
//   warps 6-9   the epilogue: tcgen05.ld of their TMEM lane quarter and the transposed store, while
//               the next tile's products go to the other accumulator.
// Bound by the MMAs' and the k-blocks' fixed costs (tensor pipe 40 % active at N = 128, L2 15 %): the split
// A in tensor memory with four stages (129 us against 138 for 16 fields of 1000 x 768), 256 rows per tile
// (139), descriptors stepped by additions (135), the rounding by integer operations (no change) and
// k-blocks of 16 in six stages (154) were tried at N = 128; N = 256 takes 101.
// The store writes the tile transposed: the transformed axis becomes the slowest axis of the
// element and the next axis the contiguous one (a rotation of the layout), so every transform of
// the orientation reads K-major rows, and D passes bring a field back to its layout.
// Every wait is bounded (about 2 s): on expiry the kernel sets *err, waits (bounded) for its own
// TMA copies, frees its tensor memory and returns.
#include "orient.cuh"

#include <cuda.h>

#include <algorithm>
#include <cstring>
#include <mutex>

namespace edab {
namespace tc {

constexpr int kBM = 128;
constexpr int kThreadsTc = 320;
constexpr unsigned long long kWaitNs = 2000000000ull;

// The stage layout of a split mode and tiles of BN columns. 3xTF32: [A hi (TMA, then split in place) | A lo |
// B hi | B lo], rows of 32 floats (BN = 128) or 16 (BN = 256: two stages of 32 were too few); BF16x3:
// [A float32 (TMA), rows of 128 bytes | A hi | A lo | B hi | B lo], rows of 32 bfloat16. Every tile starts
// on a 1024-byte boundary; its swizzle spans a row.
template <bool BF16, int BN>
struct Stage {
  static_assert(!BF16 || BN == 128);
  static constexpr int kBK = BN == 256 ? 16 : 32;
  static constexpr int kStages = BN == 256 ? 4 : 3;
  static constexpr int kRowBytes = kBK * (BF16 ? 2 : 4);  // of an operand tile
  static constexpr int kTileF32 = kBM * kBK * 4;  // the float32 A tile
  static constexpr int kTileA = kBM * kRowBytes, kTileB = BN * kRowBytes;
  static constexpr int kAhi = BF16 ? kTileF32 : 0;
  static constexpr int kAlo = kAhi + kTileA;
  static constexpr int kBhi = kAlo + kTileA;
  static constexpr int kBlo = kBhi + kTileB;
  static constexpr int kBytes = kBlo + kTileB;
  static constexpr int kTmaBytes = kTileF32 + 2 * kTileB;  // A float32, B hi, B lo
  static constexpr int kSmem = kStages * kBytes + 1024 + 256;
};

// Instruction descriptors (D float32, both operands K-major, N, M): kind::tf32 with tf32 A and B;
// kind::f16 with bfloat16 A and B.
template <int BN>
constexpr uint32_t kIdescTf32 = (1u << 4) | (2u << 7) | (2u << 10) | (static_cast<uint32_t>(BN >> 3) << 17) |
                                (static_cast<uint32_t>(kBM >> 4) << 24);
template <int BN>
constexpr uint32_t kIdescBf16 = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(BN >> 3) << 17) |
                                (static_cast<uint32_t>(kBM >> 4) << 24);

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// Shared-memory matrix descriptor of a K-major tile with rows of 128 or 64 bytes and the swizzle of that
// span: 8-row groups 1024 or 512 bytes apart (SBO), version 1, layout SWIZZLE_128B or SWIZZLE_64B.
template <int ROW_BYTES>
__device__ __forceinline__ uint64_t sw_desc(uint32_t addr) {
  static_assert(ROW_BYTES == 128 || ROW_BYTES == 64);
  return static_cast<uint64_t>((addr >> 4) & 0x3fffu) | (static_cast<uint64_t>(1) << 16) |
         (static_cast<uint64_t>(8 * ROW_BYTES >> 4) << 32) | (static_cast<uint64_t>(1) << 46) |
         (static_cast<uint64_t>(ROW_BYTES == 128 ? 2 : 4) << 61);
}
__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits for the phase of the given parity to complete; false after about kWaitNs.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  if (mbar_try(bar, parity)) return true;
  const unsigned long long t0 = now_ns();
  while (!mbar_try(bar, parity)) {
    if (now_ns() - t0 > kWaitNs) return false;
  }
  return true;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int32_t x, int32_t y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ float to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}
template <int BN>
__device__ __forceinline__ void mma_tf32(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
      "l"(adesc), "l"(bdesc), "r"(kIdescTf32<BN>), "r"(accumulate)
      : "memory");
}
template <int BN>
__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
      "l"(adesc), "l"(bdesc), "r"(kIdescBf16<BN>), "r"(accumulate)
      : "memory");
}
// bfloat16 of x rounded to nearest even, as raw bits (x finite or infinite; NaN stays NaN).
__device__ __forceinline__ uint32_t bf16_bits(float x) {
  uint32_t r;
  asm("{\n\t.reg .b16 h;\n\tcvt.rn.bf16.f32 h, %1;\n\tmov.b32 %0, {h, h};\n\t}" : "=r"(r) : "f"(x));
  return r & 0xffffu;
}
__device__ __forceinline__ float bf16_value(uint32_t bits) { return __uint_as_float(bits << 16); }
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Row m of the pass (element b = m / rows, row r = m % rows = hi * n_lo + lo) stores its column j
// at b * f_out + j * s_j + hi * pitch_out + lo.
struct RotOut {
  int64_t M;          // rows of the batch (B * rows)
  int32_t N;          // output columns (the transformed axis)
  int32_t kblocks;    // ceil(K / 32)
  int32_t npad;       // row offset of the lo basis in the basis tensor
  int64_t rows;       // rows per element
  int64_t n_lo;       // extent of the fastest row axis
  int64_t pitch_out;  // padded extent of the output's contiguous axis
  int64_t s_j;        // output stride of the transformed axis
  int64_t f_out;      // output samples per element
  int32_t n_tiles;    // tiles along N
  int64_t tiles;      // tiles of the pass
};

// Whether a tile of rows [m0, m0 + 128) holds a row of an element that runs.
__device__ __forceinline__ bool tile_runs(const RotOut& ro, const int32_t* __restrict__ run, int64_t m0) {
  const int64_t m1 = min(m0 + kBM, ro.M) - 1;
  for (int64_t b = m0 / ro.rows; b <= m1 / ro.rows; ++b) {
    if (run[b] != 0) return true;
  }
  return false;
}

template <bool BF16, int BN>
__global__ void __launch_bounds__(kThreadsTc, 1)
    gemm_tc(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, RotOut ro,
            float* __restrict__ out, const int32_t* __restrict__ run, int32_t* __restrict__ err) {
  using L = Stage<BF16, BN>;
  constexpr int kStages = L::kStages, kBK = L::kBK;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + kStages * L::kBytes);
  // bars: full[kStages], split[kStages], empty[kStages], acc_full[2], acc_empty[2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * kStages + 4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const auto full_bar = [&](int i) { return smem_u32(&bars[i]); };
  const auto split_bar = [&](int i) { return smem_u32(&bars[kStages + i]); };
  const auto empty_bar = [&](int i) { return smem_u32(&bars[2 * kStages + i]); };
  const auto acc_full = [&](int i) { return smem_u32(&bars[3 * kStages + i]); };
  const auto acc_empty = [&](int i) { return smem_u32(&bars[3 * kStages + 2 + i]); };
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(full_bar(i), 1);
      mbar_init(split_bar(i), 128);
      mbar_init(empty_bar(i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(acc_full(i), 1);
      mbar_init(acc_empty(i), 128);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(2 * BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  // Every role walks the CTA's tiles (those of elements that run) and counts k-blocks (it: the stage
  // and phase of the ring) and tiles (j: the accumulator and its phase) alike.
  bool ok = true;
  if (warp == 4) {
    if (lane == 0) {
      uint32_t it = 0;
      for (int64_t t = blockIdx.x; ok && t < ro.tiles; t += gridDim.x) {
        const int64_t m0 = t / ro.n_tiles * kBM;
        const int32_t n0 = static_cast<int32_t>(t % ro.n_tiles) * BN;
        if (!tile_runs(ro, run, m0)) continue;
        for (int32_t kb = 0; kb < ro.kblocks; ++kb, ++it) {
          const int s = static_cast<int>(it % kStages);
          if (!mbar_wait(empty_bar(s), ((it / kStages) & 1u) ^ 1u)) {
            ok = false;
            break;
          }
          unsigned char* st = base + s * L::kBytes;
          mbar_expect_tx(full_bar(s), L::kTmaBytes);
          tma_load_2d(smem_u32(st), &ta, kb * kBK, static_cast<int32_t>(m0), full_bar(s));
          tma_load_2d(smem_u32(st + L::kBhi), &tb, kb * kBK, n0, full_bar(s));
          tma_load_2d(smem_u32(st + L::kBlo), &tb, kb * kBK, ro.npad + n0, full_bar(s));
        }
      }
      // the copies of the last stages complete before the CTA may leave
      for (uint32_t k = it > kStages ? it - kStages : 0; k < it; ++k) {
        if (!mbar_wait(full_bar(static_cast<int>(k % kStages)), (k / kStages) & 1u)) ok = false;
      }
    }
  } else if (warp == 5) {
    if (lane == 0) {
      uint32_t it = 0, j = 0;
      for (int64_t t = blockIdx.x; ok && t < ro.tiles; t += gridDim.x) {
        if (!tile_runs(ro, run, t / ro.n_tiles * kBM)) continue;
        const int buf = static_cast<int>(j & 1u);
        const uint32_t acc = tmem + static_cast<uint32_t>(buf * BN);
        if (!mbar_wait(acc_empty(buf), ((j >> 1) & 1u) ^ 1u)) {  // the epilogue has read it
          ok = false;
          break;
        }
        for (int32_t kb = 0; kb < ro.kblocks; ++kb, ++it) {
          const int s = static_cast<int>(it % kStages);
          if (!mbar_wait(split_bar(s), (it / kStages) & 1u)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t st = smem_u32(base + s * L::kBytes);
          const uint32_t a_hi = st + L::kAhi, a_lo = st + L::kAlo, b_hi = st + L::kBhi, b_lo = st + L::kBlo;
          if constexpr (BF16) {
#pragma unroll
            for (int kk = 0; kk < kBK / 16; ++kk) {
              const uint32_t off = kk * 32;  // 16 bfloat16 of K inside the 64-byte swizzled row
              mma_bf16<BN>(acc, sw_desc<L::kRowBytes>(a_hi + off), sw_desc<L::kRowBytes>(b_hi + off), (kb | kk) != 0);
              mma_bf16<BN>(acc, sw_desc<L::kRowBytes>(a_hi + off), sw_desc<L::kRowBytes>(b_lo + off), 1u);
              mma_bf16<BN>(acc, sw_desc<L::kRowBytes>(a_lo + off), sw_desc<L::kRowBytes>(b_hi + off), 1u);
            }
          } else {
#pragma unroll
            for (int kk = 0; kk < kBK / 8; ++kk) {
              const uint32_t off = kk * 32;  // 8 tf32 of K inside the swizzled row
              mma_tf32<BN>(acc, sw_desc<L::kRowBytes>(a_hi + off), sw_desc<L::kRowBytes>(b_hi + off), (kb | kk) != 0);
              mma_tf32<BN>(acc, sw_desc<L::kRowBytes>(a_hi + off), sw_desc<L::kRowBytes>(b_lo + off), 1u);
              mma_tf32<BN>(acc, sw_desc<L::kRowBytes>(a_lo + off), sw_desc<L::kRowBytes>(b_hi + off), 1u);
            }
          }
          mma_commit(empty_bar(s));
        }
        mma_commit(acc_full(buf));
        ++j;
      }
    }
  } else if (warp < 4) {
    // warps 0-3: split the A tile of every stage
    const int tid = threadIdx.x;  // 0..127
    uint32_t it = 0;
    for (int64_t t = blockIdx.x; ok && t < ro.tiles; t += gridDim.x) {
      if (!tile_runs(ro, run, t / ro.n_tiles * kBM)) continue;
      for (int32_t kb = 0; kb < ro.kblocks; ++kb, ++it) {
        const int s = static_cast<int>(it % kStages);
        if (!mbar_wait(full_bar(s), (it / kStages) & 1u)) {
          ok = false;
          break;
        }
        unsigned char* st = base + s * L::kBytes;
        float4* a = reinterpret_cast<float4*>(st);
        if constexpr (BF16) {
          // the float32 tile (128-byte rows, 16-byte unit u of row r at unit u ^ (r & 7)) into the hi
          // and lo bfloat16 tiles (64-byte rows, 16-byte unit u of row r at unit u ^ ((r >> 1) & 3))
#pragma unroll
          for (int i = 0; i < L::kTileF32 / 16 / 128; ++i) {
            const int idx = tid + 128 * i;  // the physical float4 of the float32 tile
            const int r = idx >> 3;
            const int k0 = ((idx & 7) ^ (r & 7)) * 4;  // its first K column
            const float4 v = a[idx];
            const float f[4] = {v.x, v.y, v.z, v.w};
            uint32_t hb[4], lb[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              hb[q] = bf16_bits(f[q]);
              lb[q] = bf16_bits(__fsub_rn(f[q], bf16_value(hb[q])));
            }
            const int at = r * 64 + ((((k0 >> 3) ^ ((r >> 1) & 3))) << 4) + ((k0 & 7) << 1);
            *reinterpret_cast<uint2*>(st + L::kAhi + at) = make_uint2(hb[0] | (hb[1] << 16), hb[2] | (hb[3] << 16));
            *reinterpret_cast<uint2*>(st + L::kAlo + at) = make_uint2(lb[0] | (lb[1] << 16), lb[2] | (lb[3] << 16));
          }
        } else {
          float4* alo = reinterpret_cast<float4*>(st + L::kAlo);
#pragma unroll
          for (int i = 0; i < L::kTileF32 / 16 / 128; ++i) {
            const int idx = tid + 128 * i;
            const float4 v = a[idx];
            float4 h, l;
            h.x = to_tf32(v.x);
            h.y = to_tf32(v.y);
            h.z = to_tf32(v.z);
            h.w = to_tf32(v.w);
            l.x = to_tf32(__fsub_rn(v.x, h.x));
            l.y = to_tf32(__fsub_rn(v.y, h.y));
            l.z = to_tf32(__fsub_rn(v.z, h.z));
            l.w = to_tf32(__fsub_rn(v.w, h.w));
            a[idx] = h;
            alo[idx] = l;
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_arrive(split_bar(s));
      }
    }
  } else {
    // warps 6-9: the epilogue of every tile (warp w reads the TMEM lanes of quarter w mod 4)
    const int quarter = warp & 3;
    uint32_t j = 0;
    for (int64_t t = blockIdx.x; ok && t < ro.tiles; t += gridDim.x) {
      const int64_t m0 = t / ro.n_tiles * kBM;
      const int32_t n0 = static_cast<int32_t>(t % ro.n_tiles) * BN;
      if (!tile_runs(ro, run, m0)) continue;
      const int buf = static_cast<int>(j & 1u);
      // the tcgen05.ld below is warp-collective: the warp decides together
      if (!__all_sync(0xffffffffu, mbar_wait(acc_full(buf), (j >> 1) & 1u))) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int64_t m = m0 + quarter * 32 + lane;
      bool valid = m < ro.M;
      int64_t obase = 0;
      if (valid) {
        const int64_t b = m / ro.rows, r = m - b * ro.rows;
        const int64_t hi = r / ro.n_lo, lo = r - hi * ro.n_lo;
        valid = run[b] != 0;
        obase = b * ro.f_out + hi * ro.pitch_out + lo;
      }
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        float v[32];
        tmem_ld32(tmem + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(buf * BN + c * 32), v);
        if (valid) {
#pragma unroll
          for (int jj = 0; jj < 32; ++jj) {
            const int32_t col = n0 + c * 32 + jj;
            if (col < ro.N) out[obase + static_cast<int64_t>(col) * ro.s_j] = v[jj];
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      mbar_arrive(acc_empty(buf));
      ++j;
    }
  }
  if (!ok) atomicExch(err, 1);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 5) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN) : "memory");
  }
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link against libcuda).
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_fn() {
  static std::once_flag once;
  static EncodeTiled fn = nullptr;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiled>(p);
    }
    (void)cudaGetLastError();
  });
  if (!fn) throw CudaError("eda: cuTensorMapEncodeTiled is unavailable", static_cast<int>(cudaErrorNotSupported));
  return fn;
}

// A 2-D tensor map of float32 or bfloat16 elements: inner extent `inner` (contiguous), `outer` rows
// `stride` elements apart, boxes of box_k x box_rows elements, a swizzled row of 64 or 128 bytes each; reads
// past the extents return zeros.
CUtensorMap make_map(const void* base, bool bf16, uint64_t inner, uint64_t outer, uint64_t stride, int box_k, int box_rows) {
  CUtensorMap m;
  std::memset(&m, 0, sizeof m);
  const cuuint64_t dims[2] = {inner, outer};
  const cuuint64_t strides[1] = {stride * (bf16 ? 2 : 4)};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_k), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = encode_fn()(&m, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
                                 const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                 box_k * (bf16 ? 2 : 4) == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                                 CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    throw CudaError("eda: cuTensorMapEncodeTiled failed (" + std::to_string(static_cast<int>(r)) + ")",
                    static_cast<int>(cudaErrorInvalidValue));
  }
  return m;
}

template <bool BF16, int BN>
void launch(cudaStream_t s, const RotPass& p, const void* basis, int32_t kpad, int32_t npad, const float* in, float* out,
            const int32_t* run, int32_t* err, RotOut ro, int sms) {
  using L = Stage<BF16, BN>;
  const CUtensorMap ta = make_map(in, false, static_cast<uint64_t>(p.K), static_cast<uint64_t>(p.M),
                                  static_cast<uint64_t>(p.pitch_in), L::kBK, kBM);
  const CUtensorMap tb = make_map(basis, BF16, static_cast<uint64_t>(kpad), static_cast<uint64_t>(2 * npad),
                                  static_cast<uint64_t>(kpad), L::kBK, BN);
  ro.kblocks = (p.K + L::kBK - 1) / L::kBK;
  ro.n_tiles = (p.K + BN - 1) / BN;
  ro.tiles = (p.M + kBM - 1) / kBM * ro.n_tiles;
  once_on_device(reinterpret_cast<const void*>(gemm_tc<BF16, BN>), [] {
    EDAB_CUDA(cudaFuncSetAttribute(gemm_tc<BF16, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kSmem));
  });
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>(ro.tiles, sms));
  enqueue(gemm_tc<BF16, BN>, grid, kThreadsTc, L::kSmem, s, ta, tb, ro, out, run, err);
}

}  // namespace tc

// One rotated axis pass on the tensor cores (orient.cuh): see RotPass.
void rot_pass_tc(cudaStream_t s, const RotPass& p, const void* basis, bool bf16, int32_t kpad, int32_t npad,
                 const float* in, float* out, const int32_t* run, int32_t* err) {
  if (p.M < 1) return;
  tc::RotOut ro{};
  ro.M = p.M;
  ro.N = p.K;
  ro.npad = npad;
  ro.rows = p.rows;
  ro.n_lo = p.n_lo;
  ro.pitch_out = p.pitch_out;
  ro.s_j = p.s_j;
  ro.f_out = p.f_out;
  int sms = 148, dev = 0;
  EDAB_CUDA(cudaGetDevice(&dev));
  EDAB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // Tiles of 256 columns take half the MMAs (at M = 128 one of N = 256 runs in 1.5 times one of N = 128) and
  // half the reads of A: 16 fields of 1000 x 768 101 us per pass (138 with 128 columns), 64 of 512 x 512 88
  // us (102). While the tiles of 128 fit the SMs at once, the shorter tiles win: one field of 301 x 443 16 us
  // (22 with 256). So: by the waves, a wide tile counted 1.5.
  const auto waves = [&](int64_t bn) { return ((p.M + tc::kBM - 1) / tc::kBM * ((p.K + bn - 1) / bn) + sms - 1) / sms; };
  const bool w = 3 * waves(256) <= 2 * waves(128);
  const auto go = [&](auto launch) { launch(s, p, basis, kpad, npad, in, out, run, err, ro, sms); };
  if (bf16) go(tc::launch<true, 128>);
  else if (w) go(tc::launch<false, 256>);
  else go(tc::launch<false, 128>);
}

}  // namespace edab
