// Tiled tensor-core path for banded masks on 16-bit tensors (float16 / bfloat16 Q, K, V, m, l, O): the structure of
// band_forward_kernel (tile_kernels_sm100.cuh: roles, barriers, lazy per-row reference, bounded waits) around
// tcgen05.mma kind::f16, whose products of 16-bit operands are exact and whose accumulators are fp32.
//
// One CTA owns 128 query rows and walks 64-key tiles; two CTAs share an SM for every head dimension, because a Q tile of
// d = 128 is 32 KB here. Per key tile:
//   S  = Q K_j^T           128 x 64 fp32 in TMEM (two buffers)
//   P  = exp2(S c - shift) fp32 in registers, split into two 16-bit terms hi = rn(p), lo = rn(p - hi), packed two keys to a
//                          column: hi takes the first half of S's columns and lo the second, so P needs no room of its own
//   O += hi V_j + lo V_j   the fp32 probability is carried with 22 (float16, down to 2^-10 of the row's reference, steps of
//                          2^-31 of it below) or 16 (bfloat16) significant bits; the TF32 path that these calls converted
//                          to before carried 11
// Bound: the per-CTA chain S -> softmax -> P V and the last wave. Per key tile the tensor pipe has 128 x 64 x d products for S and
// twice that for P V: 29 GFLOP at L = 32768, d = 128, w = 512, in 37 us half of the measured rate, with 256 CTAs on 296 slots.
// Rows of 32 elements are staged as 64-byte rows with the 64-byte swizzle, wider ones as 128-byte pieces.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "tile_kernels_sm100.cuh"

namespace spfa {
namespace tile {

struct Band16Params {
  int64_t n_keys;     // rows of this residue's key sequence
  int64_t u_q_first;  // first query u of the shard for this residue
  int64_t n_q;        // number of query rows
  int64_t w;          // band half-width in u
  int64_t s, r;       // stride and residue: abs_row = r + u*s
  int64_t row_begin;  // first absolute row of the shard
  float scale_log2e;
  int overlap;        // as in BandParams
};

// Register split: the softmax threads take what the loading and issuing warps can spare. At 200 / 56 both types spill 8 bytes
// (stores; 24 loads), at 176 / 80 float16 spilled 16-52 (112-144) and ran 1 to 3 % longer.
template <int D>
struct Plan16 {
  static constexpr int kThreads = 256, kRegsLaunch = 128, kRegsSoftmax = 200, kRegsAux = 56;
  static_assert(kRegsSoftmax * 128 + kRegsAux * 128 <= kRegsLaunch * kThreads, "setmaxnreg budgets exceed the launch pool");
  static constexpr int BN = 64, NS = (D == 128) ? 2 : 3;           // keys per tile, K and V stages
  static constexpr int kRowBytes = (D * 2 < 128) ? D * 2 : 128;    // one swizzled row of a chunk
  static constexpr int kCols = kRowBytes / 2, kChunks = D / kCols;
  static constexpr int kQChunkBytes = 128 * kRowBytes, kKVChunkBytes = BN * kRowBytes;
  static constexpr int kQBytes = kChunks * kQChunkBytes, kStageBytes = kChunks * kKVChunkBytes;
  static constexpr int kOffQ = 0, kOffK = kQBytes, kOffV = kOffK + NS * kStageBytes, kOffBar = kOffV + NS * kStageBytes;
  static constexpr int kNumBars = 1 + 4 * NS + 6;  // q_full, k_full, k_empty, v_full, v_empty [NS], s/p/o_ready [2]
  static constexpr int kOffMisc = kOffBar + kNumBars * 8;
  static constexpr int kDynSmem = kOffMisc + 16 + 1024;
  static_assert(2 * (kDynSmem + 1024) <= 228 * 1024, "two CTAs share an SM");
  static constexpr int kColS = 0, kColO = 2 * BN, kTmemCols = 256;
  static_assert(kColO + D <= kTmemCols, "S buffers and the O accumulator exceed the TMEM allocation");
  static constexpr uint32_t kLayout = (kRowBytes == 128) ? 2u : 4u;  // shared-memory descriptors: 128- or 64-byte swizzle
  // 16-byte unit `u` of row `row` of a chunk
  static __device__ __forceinline__ uint32_t unit(int row, int u) {
    return (uint32_t)(row * kRowBytes + ((u ^ (kRowBytes == 128 ? (row & 7) : ((row >> 1) & 3))) << 4));
  }
};

// Instruction descriptor of kind::f16 (fields as in idesc_tf32; operand formats 0 = float16, 1 = bfloat16).
template <class T>
__host__ __device__ constexpr uint32_t idesc_16(int M, int N, int b_mn_major) {
  return (1u << 4) | ((std::is_same<T, __nv_bfloat16>::value ? 1u : 0u) << 7) |
         ((std::is_same<T, __nv_bfloat16>::value ? 1u : 0u) << 10) | ((uint32_t)b_mn_major << 16) |
         ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void mma16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void mma16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(acc)
      : "memory");
}

template <class T> struct Half16;
template <> struct Half16<__half> {
  static __device__ __forceinline__ uint32_t down(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  static __device__ __forceinline__ float2 up(uint32_t x) { return __half22float2(*reinterpret_cast<const __half2*>(&x)); }
  static __device__ __forceinline__ float up1(__half x) { return __half2float(x); }
  static __device__ __forceinline__ __half down1(float x) { return __float2half_rn(x); }
};
template <> struct Half16<__nv_bfloat16> {
  static __device__ __forceinline__ uint32_t down(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  static __device__ __forceinline__ float2 up(uint32_t x) {
    return make_float2(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u));
  }
  static __device__ __forceinline__ float up1(__nv_bfloat16 x) { return __bfloat162float(x); }
  static __device__ __forceinline__ __nv_bfloat16 down1(float x) { return __float2bfloat16_rn(x); }
};

// p V_j for an infinite V_j is that infinity, but the products of p's two terms need not add up to it: a term that is zero or
// negative makes NaN. Where a row's accumulator is not finite, V itself tells what it has to hold: an infinity in the row's
// window [lo, hi] (offsets into the n_here keys that the CTA multiplied) counts with its sign, both signs or NaN give NaN, and so
// does an infinity outside the window, whose weight is 0. All rows of the warp together, 32 columns at once (one per lane).
// Returned: bit c set where column c is +inf (x), -inf (y), NaN (z).
template <class T>
__device__ __noinline__ uint3 find_infinities(const T* V, int64_t pitch, int n_here, int lo, int hi) {
  const float inf = __int_as_float(0x7f800000);
  uint3 at = make_uint3(0u, 0u, 0u);
#pragma unroll 4
  for (int k = 0; k < n_here; ++k) {
    const float x = Half16<T>::up1(V[(int64_t)k * pitch + (threadIdx.x & 31)]);
    const uint32_t p = __ballot_sync(kFullMask, x == inf), n = __ballot_sync(kFullMask, x == -inf);
    const uint32_t q = __ballot_sync(kFullMask, x != x);
    const bool mine = k >= lo && k <= hi;
    at.x |= mine ? p : 0u;
    at.y |= mine ? n : 0u;
    at.z |= q | (mine ? 0u : (p | n));
  }
  at.z |= at.x & at.y;
  return at;
}

template <int D, class T>
__global__ void __launch_bounds__(256, 2)
band16_forward_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                      T* __restrict__ m_out, T* __restrict__ l_out, T* __restrict__ O_out, const T* __restrict__ V_in,
                      const Band16Params prm, int* __restrict__ err) {
  using P = Plan16<D>;
  using H = Half16<T>;
  constexpr int BN = P::BN, NS = P::NS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + P::kOffBar;
  auto bar = [&](int i) { return bar0 + 8u * i; };
  constexpr int B_QFULL = 0, B_KFULL = 1, B_KEMPTY = 1 + NS, B_VFULL = 1 + 2 * NS, B_VEMPTY = 1 + 3 * NS,
                B_SREADY = 1 + 4 * NS, B_PREADY = B_SREADY + 2, B_OREADY = B_SREADY + 4;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + P::kOffMisc + 4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  const int64_t uq0 = prm.u_q_first + (int64_t)blockIdx.x * 128;
  const int64_t uq_end = prm.u_q_first + prm.n_q;
  const int64_t rows_here = (uq_end - uq0 < 128) ? (uq_end - uq0) : 128;
  const int64_t kv_lo = (uq0 - prm.w > 0) ? (uq0 - prm.w) : 0;
  const int64_t kv_hi = (uq0 + rows_here + prm.w < prm.n_keys) ? (uq0 + rows_here + prm.w) : prm.n_keys;
  const int nT = (int)((kv_hi - kv_lo + BN - 1) / BN);  // at least one: a row's own key is in its band

  if ((prm.overlap & 1) && threadIdx.x == 96) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (threadIdx.x == 64) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmQ)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmK)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmV)) : "memory");
  }
  if (threadIdx.x == 0) {
    mbar_init(bar(B_QFULL), 1);
    for (int s = 0; s < 4 * NS; ++s) mbar_init(bar(B_KFULL + s), 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar(B_SREADY + b), 1);
      mbar_init(bar(B_PREADY + b), 128);
      mbar_init(bar(B_OREADY + b), 1);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 4) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + P::kOffMisc), "r"(P::kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + P::kOffMisc);

  if (warp >= 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(P::kRegsAux));
    if (warp == 4 && lane == 0) {
      // =============================== TMA producer ===============================
      mbar_expect_tx(bar(B_QFULL), P::kQBytes);
#pragma unroll
      for (int c = 0; c < P::kChunks; ++c)
        tma_load_3d(sbase + P::kOffQ + c * P::kQChunkBytes, &tmQ, c * P::kCols, (int32_t)(uq0 - prm.u_q_first), 0, bar(B_QFULL));
      bool ok = true;
      auto load = [&](const CUtensorMap* tm, int off, int full, int empty, int j) {
        const int st = j % NS;
        if (!mbar_wait(bar(empty + st), (uint32_t)((j / NS) & 1) ^ 1u, abort_flag, err, 111)) return false;
        mbar_expect_tx(bar(full + st), P::kStageBytes);
#pragma unroll
        for (int c = 0; c < P::kChunks; ++c)
          tma_load_3d(sbase + off + st * P::kStageBytes + c * P::kKVChunkBytes, tm, c * P::kCols, (int32_t)(kv_lo + (int64_t)j * BN),
                      0, bar(full + st));
        return true;
      };
      for (int j = 0; j < NS && j < nT && ok; ++j) ok = load(&tmK, P::kOffK, B_KFULL, B_KEMPTY, j);
      for (int j = 0; j < nT && ok; ++j) {
        ok = load(&tmV, P::kOffV, B_VFULL, B_VEMPTY, j);
        if (ok && j + NS < nT) ok = load(&tmK, P::kOffK, B_KFULL, B_KEMPTY, j + NS);
      }
    } else if (warp == 5) {
      // =============================== MMA issuer ===============================
      const bool el = elect_one();
      auto wait = [&](int b, uint32_t parity, int code) -> bool {
        return __all_sync(kFullMask, mbar_wait(bar(b), parity, abort_flag, err, code));
      };
      constexpr uint32_t kIdescS = idesc_16<T>(128, BN, 0);
      constexpr uint32_t kIdescO = idesc_16<T>(128, D, 1);
      bool ok = wait(B_QFULL, 0, 211);
      const uint64_t qd = smem_desc(sbase + P::kOffQ, 16, 8 * P::kRowBytes, P::kLayout);
      auto issue_S = [&](int j) -> bool {
        if (j >= nT) return true;
        const int st = j % NS;
        if (!wait(B_KFULL + st, (uint32_t)((j / NS) & 1), 212)) return false;
        tc_fence_after();
        const uint64_t kd = smem_desc(sbase + P::kOffK + st * P::kStageBytes, 16, 8 * P::kRowBytes, P::kLayout);
        if (el) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {  // 16 elements (32 bytes) of the contraction per MMA
            const int c = kk * 16 / P::kCols, in = kk * 32 % P::kRowBytes;
            mma16_ss(tmem + P::kColS + BN * (j & 1), qd + (uint64_t)((c * P::kQChunkBytes + in) >> 4),
                     kd + (uint64_t)((c * P::kKVChunkBytes + in) >> 4), kIdescS, kk ? 1u : 0u);
          }
          tc_commit(bar(B_SREADY + (j & 1)));
          tc_commit(bar(B_KEMPTY + st));
        }
        __syncwarp();
        return true;
      };
      ok = ok && issue_S(0) && issue_S(1);
      for (int j = 0; j < nT && ok; ++j) {
        const int st = j % NS;
        ok = wait(B_PREADY + (j & 1), (uint32_t)((j >> 1) & 1), 213) && wait(B_VFULL + st, (uint32_t)((j / NS) & 1), 214);
        if (!ok) break;
        tc_fence_after();
        // 16 keys per MMA = two 8-row swizzle groups; pieces of kCols dimensions are kKVChunkBytes apart
        const uint64_t vd = smem_desc(sbase + P::kOffV + st * P::kStageBytes, P::kKVChunkBytes, 8 * P::kRowBytes, P::kLayout);
        const uint32_t a_t = tmem + P::kColS + BN * (j & 1);
        if (el) {
#pragma unroll
          for (int part = 0; part < 2; ++part)
#pragma unroll
            for (int kk = 0; kk < BN / 16; ++kk)
              mma16_ts(tmem + P::kColO, a_t + part * (BN / 2) + kk * 8, vd + (uint64_t)((kk * 16 * P::kRowBytes) >> 4), kIdescO,
                       (part | kk) ? 1u : (j > 0 ? 1u : 0u));
          tc_commit(bar(B_OREADY + (j & 1)));
          tc_commit(bar(B_VEMPTY + st));
        }
        __syncwarp();
        ok = issue_S(j + 2);  // its S buffer is free once the PVs above are queued (the pipe runs them in order)
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(P::kRegsSoftmax));
    // =============================== softmax group: one thread owns one query row ===============================
    constexpr int NC = BN / 32;
    constexpr float kShiftSlack = 8.0f;  // P stays below 2^8 relative to the reference
    // float16 terms: P is lifted by 2^7 (its largest value, 2^15, still fits), so that the two terms hold 22 bits of it down to
    // 2^-10 of the reference and steps of 2^-31 below, where unlifted ones fade from 2^-3 on and are gone at 2^-25. The shift
    // carries the factor; the sums and O_tmem hold it until the epilogue's rel.
    constexpr float kLift = std::is_same<T, __half>::value ? 7.0f : 0.0f;
    const int row = threadIdx.x;
    const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
    const uint32_t tO = tmem + lane_base + P::kColO;
    const int64_t uq = uq0 + row;
    const bool row_valid = uq < uq_end;
    const int64_t rl = prm.r + uq * prm.s - prm.row_begin;  // row of the shard
    // the row's keys as offsets from the CTA's first key; both ends grow with the row, so the first and last row of a warp
    // bound every row of it and the chunk classes below are uniform
    const int64_t n1 = prm.n_keys - 1;
    const int lo_q = (int)(((uq - prm.w > 0) ? (uq - prm.w) : 0) - kv_lo);
    const int hi_q = (int)(((uq + prm.w < n1) ? (uq + prm.w) : n1) - kv_lo);
    const int lo_a = __shfl_sync(kFullMask, lo_q, 0), lo_b = __shfl_sync(kFullMask, lo_q, 31);
    const int hi_a = __shfl_sync(kFullMask, hi_q, 0), hi_b = __shfl_sync(kFullMask, hi_q, 31);
    // A row whose incoming l is 0 and whose O starts with a finite value carries no information (0 * O_in = 0): its old O row
    // is not read. Looked at here, where the first S tile is still on its way.
    float m_in = neg_inf(), l_in = 0.f;
    bool fresh = true;
    if (row_valid) {
      m_in = H::up1(m_out[rl]);
      l_in = H::up1(l_out[rl]);
      fresh = (l_in == 0.f) && (fabsf(H::up1(O_out[(size_t)rl * D])) <= 3.402823466e38f);
    }
    float m_true = neg_inf(), shift = neg_inf();
    uint64_t l2[2] = {0ull, 0ull};  // four partial row sums
    const float sc = prm.scale_log2e;
    const uint64_t sc2 = pack2(sc, sc), minus1 = pack2(-1.f, -1.f);
    bool ok = true;
    for (int j = 0; j < nT && ok; ++j) {
      const int c_lo = lo_q - j * BN, c_hi = hi_q - j * BN;
      const int w_lo = lo_b - j * BN, w_hi = hi_a - j * BN, v_lo = lo_a - j * BN, v_hi = hi_b - j * BN;
      int cls[NC];  // 2: every pair of the chunk is in the band, 0: none, 1: mixed (uniform over the warp)
      uint32_t vmask[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int cb = c * 32;
        const int a = c_lo - cb, b = c_hi - cb;
        vmask[c] = ((a <= 0) ? 0xffffffffu : (a >= 32 ? 0u : (0xffffffffu << a))) &
                   ((b >= 31) ? 0xffffffffu : (b < 0 ? 0u : (0xffffffffu >> (31 - b))));
        cls[c] = (cb >= w_lo && cb + 31 <= w_hi) ? 2 : ((cb + 31 < v_lo || cb > v_hi) ? 0 : 1);
      }
      const uint32_t tS = tmem + lane_base + P::kColS + BN * (j & 1);
      ok = __all_sync(kFullMask, mbar_wait(bar(B_SREADY + (j & 1)), (uint32_t)((j >> 1) & 1), abort_flag, err, 311));
      if (!ok) break;
      tc_fence_after();
      uint32_t sr[NC][32];
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (cls[c] != 0) tmem_ld32(tS + c * 32, sr[c]);
      tc_wait_ld();
      // masked columns become -inf once; the code after is the same for every chunk class
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (cls[c] == 1) {
#pragma unroll
          for (int e = 0; e < 32; ++e) sr[c][e] = ((vmask[c] >> e) & 1u) ? sr[c][e] : 0xff800000u;
        }
      float mx[4] = {neg_inf(), neg_inf(), neg_inf(), neg_inf()};
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (cls[c] != 0) {
#pragma unroll
          for (int e = 0; e < 32; e += 2)
            mx[(e >> 1) & 3] = fmaxf(fmaxf(mx[(e >> 1) & 3], __uint_as_float(sr[c][e])), __uint_as_float(sr[c][e + 1]));
        }
      const float t_max = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sc;  // sc > 0
      m_true = fmaxf(m_true, t_max);
      const bool move = t_max > shift + (kShiftSlack + kLift);
      if (__any_sync(kFullMask, move)) {
        const float new_shift = move ? t_max - kLift : shift;
        const float f = move ? ((shift == neg_inf()) ? 0.f : fast_exp2(shift - new_shift)) : 1.0f;
        const uint64_t f2 = pack2(f, f);
        l2[0] = fma2(l2[0], f2, 0ull);
        l2[1] = fma2(l2[1], f2, 0ull);
        if (j > 0) {  // O of this row up to the previous tile is final once that tile's barrier has completed
          ok = __all_sync(kFullMask, mbar_wait(bar(B_OREADY + ((j - 1) & 1)), (uint32_t)(((j - 1) >> 1) & 1), abort_flag, err, 312));
          if (!ok) break;
          tc_fence_after();
          uint32_t ob[8];  // small pieces: the S row stays in registers across this
#pragma unroll 1
          for (int c = 0; c < D / 8; ++c) {
            tmem_ld8(tO + c * 8, ob);
            tc_wait_ld();
#pragma unroll
            for (int e = 0; e < 8; ++e) ob[e] = __float_as_uint(__uint_as_float(ob[e]) * f);
            tmem_st8(tO + c * 8, ob);
          }
        }
        shift = new_shift;
      }
      const float neg_shift = (shift == neg_inf()) ? 0.f : -shift;
      const uint64_t ns2 = pack2(neg_shift, neg_shift);
      uint32_t hi[32], lo[32];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        if (cls[c] == 0) {
#pragma unroll
          for (int e = 0; e < 16; ++e) hi[c * 16 + e] = lo[c * 16 + e] = 0u;
          continue;
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          float x0, x1;
          unpack2(fma2(pack2(__uint_as_float(sr[c][2 * e]), __uint_as_float(sr[c][2 * e + 1])), sc2, ns2), x0, x1);
          const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
          const uint64_t p = pack2(p0, p1);
          l2[e & 1] = add2(l2[e & 1], p);
          const uint32_t h = H::down(p0, p1);
          const float2 hf = H::up(h);
          float r0, r1;
          unpack2(fma2(pack2(hf.x, hf.y), minus1, p), r0, r1);  // exact
          hi[c * 16 + e] = h;
          lo[c * 16 + e] = H::down(r0, r1);
        }
      }
      tmem_st32(tS, hi);
      tmem_st32(tS + 32, lo);
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(bar(B_PREADY + (j & 1)));
    }
    float la, lb, lc, ld;
    unpack2(l2[0], la, lb);
    unpack2(l2[1], lc, ld);
    const float l_run = (la + lb) + (lc + ld);
    // ---- epilogue ----
    if (ok && nT > 1)
      ok = __all_sync(kFullMask, mbar_wait(bar(B_OREADY + ((nT - 2) & 1)), (uint32_t)(((nT - 2) >> 1) & 1), abort_flag, err, 313));
    ok = ok && __all_sync(kFullMask, mbar_wait(bar(B_OREADY + ((nT - 1) & 1)), (uint32_t)(((nT - 1) >> 1) & 1), abort_flag, err, 314));
    // one barrier tells every thread whether all warps got here and whether the whole tile can leave as one bulk store
    auto all_of = [&](bool x) {
      uint32_t r;
      asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                   : "=r"(r)
                   : "r"((uint32_t)x)
                   : "memory");
      return r != 0;
    };
    if (all_of(ok)) {
      tc_fence_after();
      const bool store = row_valid && l_run > 0.f;
      float ca = 0.f, cb = 0.f;  // O_out = ca * O_in + cb * O_tmem
      if (store) {
        const float rel = fast_exp2(shift - m_true);
        const float m_loc = m_true * 0.6931471805599453f;
        const float m_o = fmaxf(m_in, m_loc);
        const float a = l_in * fast_exp2((m_in - m_o) * kLog2e);
        const float bt = fast_exp2((m_loc - m_o) * kLog2e);
        const float l_o = fmaf(l_run * rel, bt, a);
        const float inv = 1.0f / l_o;
        ca = a * inv;
        cb = bt * rel * inv;
        m_out[rl] = H::down1(m_o);
        l_out[rl] = H::down1(l_o);
      }
      // 32 columns of O_tmem, infinities of V put right (every thread of the warp takes part)
      auto load_O = [&](int c, uint32_t (&ob)[32]) {
        tmem_ld32(tO + c * 32, ob);
        tc_wait_ld();
        uint64_t zero[4] = {0ull, 0ull, 0ull, 0ull};  // stay 0 while every value is finite; four short chains
#pragma unroll
        for (int e = 0; e < 32; e += 2)
          zero[(e >> 1) & 3] = fma2(pack2(__uint_as_float(ob[e]), __uint_as_float(ob[e + 1])), 0ull, zero[(e >> 1) & 3]);
        if (__any_sync(kFullMask, ((zero[0] | zero[1] | zero[2] | zero[3]) & 0x7fffffff7fffffffull) != 0ull)) {
          const int64_t left = prm.n_keys - kv_lo;
          const uint3 at = find_infinities<T>(V_in + kv_lo * prm.s * D + c * 32, prm.s * D,
                                              (left < nT * BN) ? (int)left : nT * BN, lo_q, hi_q);
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const uint32_t bit = 1u << e;
            ob[e] = (at.z & bit) ? 0x7fc00000u : (at.x & bit) ? 0x7f800000u : (at.y & bit) ? 0xff800000u : ob[e];
          }
        }
      };
      if (all_of(!row_valid || (store && fresh))) {
        // cb * O_tmem is the output: staged where Q was (every S MMA has completed) in the layout of a Q tile, stored by the
        // bulk-copy engine; rows past the end of the shard are clipped by the tensor map
        uint8_t* stage = smem + P::kOffQ;
        uint32_t ob[32];
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          load_O(c, ob);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint4 x;
            x.x = H::down(cb * __uint_as_float(ob[8 * u + 0]), cb * __uint_as_float(ob[8 * u + 1]));
            x.y = H::down(cb * __uint_as_float(ob[8 * u + 2]), cb * __uint_as_float(ob[8 * u + 3]));
            x.z = H::down(cb * __uint_as_float(ob[8 * u + 4]), cb * __uint_as_float(ob[8 * u + 5]));
            x.w = H::down(cb * __uint_as_float(ob[8 * u + 6]), cb * __uint_as_float(ob[8 * u + 7]));
            const int col = c * 32 + u * 8;
            *reinterpret_cast<uint4*>(stage + col / P::kCols * P::kQChunkBytes + P::unit(row, col % P::kCols / 8)) = x;
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (row == 0) {
#pragma unroll
          for (int c = 0; c < P::kChunks; ++c)
            asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(
                             reinterpret_cast<uint64_t>(&tmO)),
                         "r"(c * P::kCols), "r"((int32_t)(uq0 - prm.u_q_first)), "r"(0), "r"(sbase + P::kOffQ + c * P::kQChunkBytes)
                         : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        }
      } else {  // a row with old state, or one that must not be written: each thread merges its own row
        uint32_t ob[32];
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
          load_O(c, ob);
          if (store) {
            uint4* po = reinterpret_cast<uint4*>(O_out + (size_t)rl * D + c * 32);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              uint4 x = make_uint4(0u, 0u, 0u, 0u);
              if (!fresh) x = po[u];
              uint32_t wv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float2 o = H::up(wv[i]);
                wv[i] = H::down(fmaf(ca, o.x, cb * __uint_as_float(ob[8 * u + 2 * i])),
                                fmaf(ca, o.y, cb * __uint_as_float(ob[8 * u + 2 * i + 1])));
              }
              po[u] = make_uint4(wv[0], wv[1], wv[2], wv[3]);
            }
          }
          __syncwarp();
        }
      }
    }
  }

  // ---- common exit: everyone is done with TMEM before it is released ----
  tc_fence_before();
  __syncthreads();
  if ((prm.overlap & 2) && threadIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
  if (warp == 4) {
    tc_fence_after();
    if (*abort_flag && lane == 0) {  // copies that may still be in flight land before the CTA's shared memory is reused
      const uint64_t t0 = globaltimer();
      while (globaltimer() - t0 < 2000000ull) {
      }
    }
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(P::kTmemCols) : "memory");
  }
}

}  // namespace tile
}  // namespace spfa
