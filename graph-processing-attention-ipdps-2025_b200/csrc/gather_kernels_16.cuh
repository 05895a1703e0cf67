// Gather path with 16-bit storage: Q, K, V, O, m, l are __half or __nv_bfloat16 in memory, all arithmetic is fp32.
//
// The reference instantiates its kernels for Half as well (AT_DISPATCH_FLOATING_TYPES_AND_HALF,
// sp_flatt_csr_kernel.cu:270) and there accumulates in half; here only the loads and stores are 16-bit, so results
// are at least as accurate as the reference's, and an HBM-bound gather moves half the bytes of the fp32 path.
// Same structure as gather_kernels.cuh: one warp per query row, a key row is covered by LPK = D/8 lanes with one
// 128-bit load each (8 elements), KPS = 32/LPK keys per warp step, four keys in flight per lane group, online
// softmax state per group, groups merged once per row, long rows walked by all warps of the CTA.
// D in {32, 64, 128} (LPK >= 4); other sizes take the generic kernel (gather_generic.cuh) with 16-bit loads.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "gather_kernels.cuh"
#include "spfa_common.cuh"

namespace spfa {

struct GnlAnyRowCols;

template <class T> struct Cvt16;
template <> struct Cvt16<__half> {
  static __device__ __forceinline__ float2 up(uint32_t x) { return __half22float2(*reinterpret_cast<const __half2*>(&x)); }
  static __device__ __forceinline__ uint32_t down(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  static __device__ __forceinline__ float up1(__half x) { return __half2float(x); }
  static __device__ __forceinline__ __half down1(float x) { return __float2half_rn(x); }
};
template <> struct Cvt16<__nv_bfloat16> {
  static __device__ __forceinline__ float2 up(uint32_t x) {  // a bfloat16 is the upper half of a float
    return make_float2(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u));
  }
  static __device__ __forceinline__ uint32_t down(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  static __device__ __forceinline__ float up1(__nv_bfloat16 x) { return __bfloat162float(x); }
  static __device__ __forceinline__ __nv_bfloat16 down1(float x) { return __float2bfloat16_rn(x); }
};

struct Vec8 {
  float v[8];
};

template <class T>
__device__ __forceinline__ Vec8 ldg8(const T* p) {  // 16 bytes = 8 elements, read-only path
  const uint4 u = __ldg(reinterpret_cast<const uint4*>(p));
  Vec8 r;
  float2 f;
  f = Cvt16<T>::up(u.x); r.v[0] = f.x; r.v[1] = f.y;
  f = Cvt16<T>::up(u.y); r.v[2] = f.x; r.v[3] = f.y;
  f = Cvt16<T>::up(u.z); r.v[4] = f.x; r.v[5] = f.y;
  f = Cvt16<T>::up(u.w); r.v[6] = f.x; r.v[7] = f.y;
  return r;
}

// q . k of one 16-byte piece; k stays packed until it is used (eight pieces in flight are 32 registers, not 64).
template <class T>
__device__ __forceinline__ float dot8(const Vec8& q, const uint4 k) {
  float2 f = Cvt16<T>::up(k.x);
  float p = q.v[0] * f.x;
  p = fmaf(q.v[1], f.y, p);
  f = Cvt16<T>::up(k.y);
  p = fmaf(q.v[2], f.x, p);
  p = fmaf(q.v[3], f.y, p);
  f = Cvt16<T>::up(k.z);
  p = fmaf(q.v[4], f.x, p);
  p = fmaf(q.v[5], f.y, p);
  f = Cvt16<T>::up(k.w);
  p = fmaf(q.v[6], f.x, p);
  return fmaf(q.v[7], f.y, p);
}

struct RowAcc8 {
  float m, l;
  Vec8 acc;
  __device__ __forceinline__ void clear() {
    m = neg_inf();
    l = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc.v[i] = 0.f;
  }
};

template <int LPK, class T>
__device__ __forceinline__ void softmax_step4_16(float mine, int grp, const uint4 (&v)[4], RowAcc8& st) {
  float mc = fmaxf(mine, __shfl_xor_sync(kFullMask, mine, LPK / 2));
  mc = fmaxf(mc, __shfl_xor_sync(kFullMask, mc, LPK / 4));
  const float m_new = fmaxf(st.m, mc);
  const float m_safe = (m_new == neg_inf()) ? 0.f : m_new;
  const float corr = fast_exp2((st.m - m_safe) * kLog2e);
  const float pm = fast_exp2((mine - m_safe) * kLog2e);
  const int base = grp * LPK;
  const float p0 = __shfl_sync(kFullMask, pm, base);
  const float p1 = __shfl_sync(kFullMask, pm, base + LPK / 4);
  const float p2 = __shfl_sync(kFullMask, pm, base + LPK / 2);
  const float p3 = __shfl_sync(kFullMask, pm, base + LPK / 2 + LPK / 4);
#pragma unroll
  for (int i = 0; i < 8; ++i) st.acc.v[i] *= corr;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const float p = (u == 0) ? p0 : (u == 1) ? p1 : (u == 2) ? p2 : p3;
    const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = Cvt16<T>::up(w[i]);
      st.acc.v[2 * i] = fmaf(p, f.x, st.acc.v[2 * i]);
      st.acc.v[2 * i + 1] = fmaf(p, f.y, st.acc.v[2 * i + 1]);
    }
  }
  st.l = fmaf(st.l, corr, (p0 + p1) + (p2 + p3));
  st.m = m_new;
}

template <int D, class T, class Cols>
__device__ __forceinline__ void accumulate_slots16(const Cols& cols, const typename Cols::Row& row, int64_t t0, int64_t t1,
                                                   const Vec8& q, const T* __restrict__ K, const T* __restrict__ V,
                                                   float scale, int lane, RowAcc8& st) {
  constexpr int LPK = D / 8;
  constexpr int KPS = 32 / LPK;
  static_assert(LPK >= 4 && LPK <= 32, "16-bit rows of 32 to 256 elements");
  const int grp = lane / LPK, sub = lane % LPK;
  const int own = (((sub & (LPK / 2)) != 0) ? 2 : 0) + (((sub & (LPK / 4)) != 0) ? 1 : 0);
  const T* Kl = K + sub * 8;
  const T* Vl = V + sub * 8;
  int32_t c_next = (t0 + lane < t1) ? cols.slot(row, t0 + lane) : -1;
  for (int64_t base = t0; base < t1; base += 32) {
    const int32_t c_lane = c_next;  // the next batch's columns travel while this batch's K/V rows are worked on
    c_next = (base + 32 + lane < t1) ? cols.slot(row, base + 32 + lane) : -1;
    if (__all_sync(kFullMask, c_lane >= 0)) {  // 32 real keys: no predicates
#pragma unroll 1
      for (int j0 = 0; j0 < LPK; j0 += 4) {
        uint4 k[4], v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t c = (uint32_t)__shfl_sync(kFullMask, c_lane, grp + (j0 + u) * KPS);
          k[u] = __ldg(reinterpret_cast<const uint4*>(Kl + (size_t)c * D));
          v[u] = __ldg(reinterpret_cast<const uint4*>(Vl + (size_t)c * D));
        }
        const float mine = reduce4_transposed<LPK>(dot8<T>(q, k[0]), dot8<T>(q, k[1]), dot8<T>(q, k[2]), dot8<T>(q, k[3]), sub) * scale;
        softmax_step4_16<LPK, T>(mine, grp, v, st);
      }
      continue;
    }
    const int nb = (t1 - base < 32) ? (int)(t1 - base) : 32;
#pragma unroll 1
    for (int j0 = 0; j0 < LPK; j0 += 4) {
      if (j0 * KPS >= nb) break;  // warp-uniform
      uint4 k[4], v[4];
      int32_t c_own = -1;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int32_t c = __shfl_sync(kFullMask, c_lane, grp + (j0 + u) * KPS);
        if (c >= 0) {
          k[u] = __ldg(reinterpret_cast<const uint4*>(Kl + (size_t)c * D));
          v[u] = __ldg(reinterpret_cast<const uint4*>(Vl + (size_t)c * D));
        } else {  // a masked key contributes probability 0; zero V keeps 0 * V finite
          k[u] = v[u] = make_uint4(0u, 0u, 0u, 0u);
        }
        if (u == own) c_own = c;
      }
      float mine = reduce4_transposed<LPK>(dot8<T>(q, k[0]), dot8<T>(q, k[1]), dot8<T>(q, k[2]), dot8<T>(q, k[3]), sub) * scale;
      if (c_own < 0) mine = neg_inf();
      softmax_step4_16<LPK, T>(mine, grp, v, st);
    }
  }
}

template <int LPK>
__device__ __forceinline__ void merge_groups16(RowAcc8& st) {
#pragma unroll
  for (int o = LPK; o < 32; o <<= 1) {
    const float mo = __shfl_xor_sync(kFullMask, st.m, o);
    const float lo = __shfl_xor_sync(kFullMask, st.l, o);
    const float mn = fmaxf(st.m, mo);
    const float ms = (mn == neg_inf()) ? 0.f : mn;
    const float c1 = fast_exp2((st.m - ms) * kLog2e);
    const float c2 = fast_exp2((mo - ms) * kLog2e);
    st.l = st.l * c1 + lo * c2;
#pragma unroll
    for (int i = 0; i < 8; ++i) st.acc.v[i] = st.acc.v[i] * c1 + __shfl_xor_sync(kFullMask, st.acc.v[i], o) * c2;
    st.m = mn;
  }
}

// Fold a finished row into the caller's 16-bit state (same recurrence as store_row of the fp32 path).
template <int D, class T>
__device__ __forceinline__ void store_row16(const RowAcc8& st, T* __restrict__ m, T* __restrict__ l, T* __restrict__ O,
                                            int64_t r, int lane) {
  constexpr int LPK = D / 8;
  const float m_in = Cvt16<T>::up1(m[r]), l_in = Cvt16<T>::up1(l[r]);
  const float m_out = fmaxf(m_in, st.m);
  const float a = l_in * fast_exp2((m_in - m_out) * kLog2e);
  const float b = fast_exp2((st.m - m_out) * kLog2e);
  const float l_out = fmaf(st.l, b, a);
  const float inv = 1.0f / l_out;
  if (lane < LPK) {
    T* op = O + (size_t)r * D + lane * 8;
    const Vec8 o = ldg8<T>(op);
    float y[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) y[i] = (a * o.v[i] + b * st.acc.v[i]) * inv;
    uint4 u;
    u.x = Cvt16<T>::down(y[0], y[1]);
    u.y = Cvt16<T>::down(y[2], y[3]);
    u.z = Cvt16<T>::down(y[4], y[5]);
    u.w = Cvt16<T>::down(y[6], y[7]);
    *reinterpret_cast<uint4*>(op) = u;
  }
  if (lane == 0) {
    m[r] = Cvt16<T>::down1(m_out);
    l[r] = Cvt16<T>::down1(l_out);
  }
}

// Rows cut into slices (explicit masks whose caller gave scratch): a power-law graph holds most of its entries in a few rows,
// and a row walked by one warp or one CTA is a chain of dependent loads (about a microsecond per 16 keys): at L = 50021,
// d = 64, 1.96M f16 entries in rows of up to 8192 the launch took 314 us with single-CTA long rows, 300 us when clusters of
// eight CTAs shared them, because every resident warp that waits for a long row is a load that is not in flight. So rows of
// more than a slice (kSliceSlots slots, more for huge masks) are cut into slices that single warps walk independently; partial
// states go to scratch and the warp that finishes a row's last slice folds them in slice order: 109 us for the whole call. A
// slice is a multiple of the 32-slot batch, long enough that the few partial states cost nothing beside the K/V rows (2 * D * 2
// bytes per entry).
constexpr int kSliceSlots = 256;

struct RowSlices {
  unsigned long long* count;  // [0] slices that the long rows asked for, [1] rows that got none; zero before row_slices_kernel<false>
  int4* items;          // [cap] {row, slice, slices of the row, index of the row's first item}; no slices: nothing to do
  unsigned int* done;   // [cap] at a row's first item: slices finished
  float* part;          // [cap][d + 4]: un-normalised accumulator, then m, l
  int* whole;           // [n_rows] long rows for which the list had no room left: one warp each
  unsigned int cap;
  int slots;            // of a slice; longer rows are cut
};

// ALONE: one CTA, which needs no zeroed counts (a memory operation less in front of a short call).
template <bool ALONE>
__global__ void row_slices_kernel(const uint64_t* __restrict__ row_off, int64_t n_rows, const RowSlices sl) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  __shared__ unsigned long long s_count[2];
  unsigned long long* count = ALONE ? s_count : sl.count;
  if (ALONE) {
    if (threadIdx.x < 2) s_count[threadIdx.x] = 0ull;
    __syncthreads();
  }
#pragma unroll 4
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t n = (int64_t)row_off[r + 1] - (int64_t)row_off[r];
    if (n <= sl.slots) continue;
    const unsigned long long ns = (unsigned long long)((n + sl.slots - 1) / sl.slots);
    const unsigned long long first = atomicAdd(count, ns);
    // cap covers ascending offsets (2 nnz / slots slices). Rows that share entries, or offsets beyond the caller's nnz, can
    // need more: such a row stays whole, and what is left of the list is made neutral
    if (first + ns > sl.cap) {
      for (unsigned long long s = first; s < sl.cap; ++s) sl.items[s] = make_int4(0, 0, 0, 0);
      sl.whole[atomicAdd(count + 1, 1ull)] = (int)r;
      continue;
    }
    sl.done[first] = 0u;
    for (unsigned int s = 0; s < ns; ++s) sl.items[first + s] = make_int4((int)r, (int)s, (int)ns, (int)first);
  }
  if (ALONE) {
    __syncthreads();
    if (threadIdx.x < 2) sl.count[threadIdx.x] = s_count[threadIdx.x];
  }
}

// One warp per query row at a time, rows claimed from the CTA's counter. With SLICED, blocks [list_begin, list_begin +
// list_blocks) walk the listed slices, one per warp, and the other blocks leave the listed rows out; the list is produced by
// the launch before this one, which this one may overlap (only the list blocks wait for it). The list blocks come after a
// first wave of ordinary blocks, which covers the time the list takes. Without SLICED (implicit masks, or a CSR call without
// scratch) rows beyond kHeavyRowSlots are shared by the four warps of their CTA.
// Global-no-local: the first nG blocks take a listed row each and share it among their warps, the others leave the listed rows
// out. Listed rows are as long as the sequence and often lie side by side; in one CTA's share they would run one after the other
// (d = 64, L = 131072, 16 leading listed rows: 12.0 ms with shares of 12 rows, 1.4 ms so; 16 random ones: 1.27 and 1.21 ms).
template <int D, class T, class Cols, bool SLICED>
__global__ void __launch_bounds__(kRowWarps * 32, 6)
gather_rows16_kernel(const T* __restrict__ Q, const T* __restrict__ K, const T* __restrict__ V, T* __restrict__ m,
                     T* __restrict__ l, T* __restrict__ O, const Cols cols, int64_t row_begin, int64_t n_rows, int use_nan,
                     float scale, int rows_per_cta, int long_slots, const RowSlices sl, int list_begin, int list_blocks) {
  constexpr int LPK = D / 8;
  __shared__ int s_heavy[kMaxRowsPerCta];
  __shared__ int s_n_heavy, s_next;
  __shared__ float s_ml[kRowWarps][2];
  __shared__ float s_acc[kRowWarps][D];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t block = blockIdx.x;
  if (SLICED) {
    if ((int)blockIdx.x >= list_begin && (int)blockIdx.x < list_begin + list_blocks) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      const volatile unsigned long long* count = sl.count;
      for (unsigned int it = ((int)blockIdx.x - list_begin) * kRowWarps + warp;; it += (unsigned int)list_blocks * kRowWarps) {
        // read again for each item: two registers less in the walk
        const unsigned int n_items = (count[0] < sl.cap) ? (unsigned int)count[0] : sl.cap;
        if (it >= n_items + (unsigned int)count[1]) break;
        const int4 item = (it < n_items) ? sl.items[it] : make_int4(sl.whole[it - n_items], 0, 1, 0);
        if (item.z == 0) continue;
        const int64_t r = item.x;
        const typename Cols::Row row = cols.open(r, row_begin + r);
        const int64_t t0 = (int64_t)item.y * long_slots;
        const int64_t t1 = (item.z > 1 && t0 + long_slots < row.n) ? (t0 + long_slots) : row.n;
        const Vec8 q = ldg8<T>(Q + (size_t)r * D + (lane % LPK) * 8);
        RowAcc8 st;
        st.clear();
        accumulate_slots16<D, T, Cols>(cols, row, t0, t1, q, K, V, scale, lane, st);
        merge_groups16<LPK>(st);
        if (item.z > 1) {
          float* part = sl.part + (size_t)it * (D + 4);
          if (lane < LPK) {
            float4* a = reinterpret_cast<float4*>(part + lane * 8);
            a[0] = make_float4(st.acc.v[0], st.acc.v[1], st.acc.v[2], st.acc.v[3]);
            a[1] = make_float4(st.acc.v[4], st.acc.v[5], st.acc.v[6], st.acc.v[7]);
          }
          if (lane == 0) *reinterpret_cast<float2*>(part + D) = make_float2(st.m, st.l);
          __threadfence();
          __syncwarp();
          unsigned int before = 0;
          if (lane == 0) before = atomicAdd(sl.done + item.w, 1u);
          if (__shfl_sync(kFullMask, before, 0) != (unsigned int)item.z - 1u) continue;
          __threadfence();
          const float* p0 = sl.part + (size_t)item.w * (D + 4);
          float mx = neg_inf();
          for (int s = lane; s < item.z; s += 32) mx = fmaxf(mx, __ldcg(p0 + (size_t)s * (D + 4) + D));
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(kFullMask, mx, o));
          const float ms = (mx == neg_inf()) ? 0.f : mx;
          st.clear();
          st.m = mx;
#pragma unroll 2
          for (int s = 0; s < item.z; ++s) {
            const float* p = p0 + (size_t)s * (D + 4);
            const float2 ml = __ldcg(reinterpret_cast<const float2*>(p + D));
            const float4 a0 = __ldcg(reinterpret_cast<const float4*>(p) + 2 * (lane % LPK));
            const float4 a1 = __ldcg(reinterpret_cast<const float4*>(p) + 2 * (lane % LPK) + 1);
            const float c = fast_exp2((ml.x - ms) * kLog2e);
            st.l = fmaf(ml.y, c, st.l);
            st.acc.v[0] = fmaf(a0.x, c, st.acc.v[0]);
            st.acc.v[1] = fmaf(a0.y, c, st.acc.v[1]);
            st.acc.v[2] = fmaf(a0.z, c, st.acc.v[2]);
            st.acc.v[3] = fmaf(a0.w, c, st.acc.v[3]);
            st.acc.v[4] = fmaf(a1.x, c, st.acc.v[4]);
            st.acc.v[5] = fmaf(a1.y, c, st.acc.v[5]);
            st.acc.v[6] = fmaf(a1.z, c, st.acc.v[6]);
            st.acc.v[7] = fmaf(a1.w, c, st.acc.v[7]);
          }
        }
        if (st.l > 0.f) store_row16<D, T>(st, m, l, O, r, lane);
      }
      return;
    }
    if ((int)blockIdx.x >= list_begin) block -= list_blocks;
  }
  constexpr bool kListed = std::is_same<Cols, GnlAnyRowCols>::value;
  int64_t first = block * rows_per_cta;
  bool one_row = false;
  if constexpr (kListed) {
    if (block < cols.list.nG) {
      first = (int64_t)cols.list.G[block] - row_begin;
      if (!cols.list_live[block] || first < 0 || first >= n_rows) return;
      one_row = true;
      rows_per_cta = 0;
    } else {
      first = (block - cols.list.nG) * rows_per_cta;
    }
  }
  if (threadIdx.x == 0) {
    s_heavy[0] = 0;
    s_n_heavy = one_row;
    s_next = kRowWarps;
  }
  __syncthreads();
  for (int i = warp; i < rows_per_cta && first + i < n_rows;) {  // warp-uniform
    const int64_t r = first + i;
    const typename Cols::Row row = cols.open(r, row_begin + r);
    bool listed = false;
    if constexpr (kListed) listed = row.is_global;
    if (listed) {
    } else if (row.n <= 0) {
      if (Cols::kNanFillEmpty && use_nan && lane < LPK) {
        const uint32_t nn = Cvt16<T>::down(__int_as_float(0x7fc00000), __int_as_float(0x7fc00000));
        *reinterpret_cast<uint4*>(O + (size_t)r * D + lane * 8) = make_uint4(nn, nn, nn, nn);
      }
    } else if (row.n > long_slots) {
      if (!SLICED && lane == 0) s_heavy[atomicAdd(&s_n_heavy, 1)] = i;
    } else {
      const Vec8 q = ldg8<T>(Q + (size_t)r * D + (lane % LPK) * 8);
      RowAcc8 st;
      st.clear();
      accumulate_slots16<D, T, Cols>(cols, row, 0, row.n, q, K, V, scale, lane, st);
      merge_groups16<LPK>(st);
      if (st.l > 0.f) store_row16<D, T>(st, m, l, O, r, lane);
    }
    if (rows_per_cta <= kRowWarps) break;
    int nxt = 0;
    if (lane == 0) nxt = atomicAdd(&s_next, 1);
    i = __shfl_sync(kFullMask, nxt, 0);
  }
  if (SLICED) return;
  __syncthreads();
  const int n_heavy = s_n_heavy;  // uniform over the CTA
  for (int h = 0; h < n_heavy; ++h) {  // long rows: every warp of the CTA takes a share of the slots
    const int64_t rh = first + s_heavy[h];
    const typename Cols::Row row = cols.open(rh, row_begin + rh);
    int64_t per = (row.n + kRowWarps - 1) / kRowWarps;
    per = (per + 31) / 32 * 32;
    const int64_t t0 = (int64_t)warp * per;
    int64_t t1 = t0 + per;
    if (t1 > row.n) t1 = row.n;
    RowAcc8 st;
    st.clear();
    if (t0 < t1) {
      const Vec8 q = ldg8<T>(Q + (size_t)rh * D + (lane % LPK) * 8);
      accumulate_slots16<D, T, Cols>(cols, row, t0, t1, q, K, V, scale, lane, st);
      merge_groups16<LPK>(st);
    }
    if (lane < LPK) {
#pragma unroll
      for (int i = 0; i < 8; ++i) s_acc[warp][lane * 8 + i] = st.acc.v[i];
    }
    if (lane == 0) {
      s_ml[warp][0] = st.m;
      s_ml[warp][1] = st.l;
    }
    __syncthreads();
    if (warp == 0) {
      RowAcc8 tot;
      tot.clear();
      const int sub = lane % LPK;
      for (int wv = 0; wv < kRowWarps; ++wv) {  // in slot order, like the single-warp walk
        const float mo = s_ml[wv][0], lo = s_ml[wv][1];
        const float mn = fmaxf(tot.m, mo);
        const float ms = (mn == neg_inf()) ? 0.f : mn;
        const float c1 = fast_exp2((tot.m - ms) * kLog2e), c2 = fast_exp2((mo - ms) * kLog2e);
        tot.l = tot.l * c1 + lo * c2;
#pragma unroll
        for (int i = 0; i < 8; ++i) tot.acc.v[i] = tot.acc.v[i] * c1 + s_acc[wv][sub * 8 + i] * c2;
        tot.m = mn;
      }
      if (tot.l > 0.f) store_row16<D, T>(tot, m, l, O, rh, lane);
    }
    __syncthreads();
  }
}

}  // namespace spfa
