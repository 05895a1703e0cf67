// C ABI, 16-bit storage on the tensor cores: banded masks (Local, Local-1D-dilated) through band16_forward_kernel.
#include <atomic>
#include <cmath>

#include "capi_common.cuh"
#include "tensor_map.cuh"
#include "tile_kernels_16.cuh"

namespace spfa {

// The rule of the fp32 tiled path (kTileMinHalfWidth, kTileMaxStride), so that a mask takes the same kind of kernel in either
// storage. Narrower bands read each key row for a handful of query rows and stay on the gather path.
constexpr int64_t kTile16MinHalfWidth = 32, kTile16MaxStride = 16;
// float16 probabilities below 2^-32 of the row's largest drop out of P V (not out of l). A window of 2 w + 1 < 2^18 such keys
// loses less than 2^-14 of V's magnitude, a quarter of what the stored result is rounded by; wider windows are converted.
constexpr int64_t kTile16MaxHalfWidthF16 = 1LL << 17;

// [rows, d] 16-bit matrix with a row pitch, fetched as boxes of box_rows x kCols elements. Rows outside read as zeros.
template <int D, class T>
bool make_row_map_16(CUtensorMap* tm, const T* base, int64_t rows, int64_t pitch_bytes, int box_rows) {
  using P = tile::Plan16<D>;
  TensorMapEncodeTiledFn enc = tensor_map_encoder();
  if (!enc) return false;
  cuuint64_t dims[3] = {(cuuint64_t)D, (cuuint64_t)rows, 1u};
  cuuint64_t strides[2] = {(cuuint64_t)pitch_bytes, (cuuint64_t)((rows > 0 ? rows : 1) * pitch_bytes)};
  cuuint32_t box[3] = {(cuuint32_t)P::kCols, (cuuint32_t)box_rows, 1u};
  cuuint32_t estr[3] = {1u, 1u, 1u};
  return enc(tm, std::is_same<T, __half>::value ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3,
             const_cast<T*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             P::kRowBytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// As band_kernel_usable of the fp32 path: setmaxnreg.inc must be covered by what the launch allocates.
template <int D, class T>
bool band16_usable() {
  using P = tile::Plan16<D>;
  static std::atomic<int> cached[64];  // per device: 0 unknown, 1 usable, 2 not
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  int v = cached[dev].load(std::memory_order_relaxed);
  if (v == 0) {
    cudaFuncAttributes attr;
    auto kern = tile::band16_forward_kernel<D, T>;
    const bool ok = cudaFuncGetAttributes(&attr, kern) == cudaSuccess &&
                    attr.numRegs * P::kThreads >= (P::kRegsSoftmax + P::kRegsAux) * 128 &&
                    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, P::kDynSmem) == cudaSuccess;
    v = ok ? 1 : 2;
    cached[dev].store(v, std::memory_order_relaxed);
  }
  return v == 1;
}

template <class F>
int with_shape_16(int dtype, int d, F&& f) {
  auto by_d = [&](auto t) {
    if (d == 32) return f(t, std::integral_constant<int, 32>());
    if (d == 64) return f(t, std::integral_constant<int, 64>());
    if (d == 128) return f(t, std::integral_constant<int, 128>());
    return (int)SPFA_ERR_EMBED_DIM;
  };
  if (dtype == SPFA_DTYPE_F16) return by_d(static_cast<__half*>(nullptr));
  if (dtype == SPFA_DTYPE_BF16) return by_d(static_cast<__nv_bfloat16*>(nullptr));
  return SPFA_ERR_BAD_ARG;
}

// Band |u_q - u_k| <= w on every residue class of stride s; one launch per class, consecutive ones overlap (disjoint rows).
template <int D, class T>
int launch_band16(const T* Q, const T* K, const T* V, T* m, T* l, T* O, int64_t L, int64_t w, int64_t s, int64_t row_begin,
                  int64_t row_end, cudaStream_t st) {
  using P = tile::Plan16<D>;
  if (!band16_usable<D, T>()) return SPFA_ERR_REGISTER_BUDGET;
  int* err = tile_error_word();
  if (!err) return SPFA_ERR_LAUNCH;
  bool launched = false;
  for (int64_t r = 0; r < s && r < L; ++r) {
    tile::Band16Params prm{};
    prm.n_keys = (L - r + s - 1) / s;
    prm.u_q_first = (row_begin > r) ? (row_begin - r + s - 1) / s : 0;
    int64_t u_end = (row_end > r) ? (row_end - r + s - 1) / s : 0;
    if (u_end > prm.n_keys) u_end = prm.n_keys;
    if (u_end <= prm.u_q_first) continue;
    prm.n_q = u_end - prm.u_q_first;
    prm.w = w;
    prm.s = s;
    prm.r = r;
    prm.row_begin = row_begin;
    prm.scale_log2e = (1.0f / sqrtf((float)D)) * kLog2e;
    prm.overlap = ((r + 1 < s && r + 1 < L) ? 1 : 0) | (launched ? 2 : 0);
    const int64_t pitch = s * D * 2, first = (r + prm.u_q_first * s - row_begin) * D;
    CUtensorMap tmQ, tmK, tmV, tmO;
    if (!make_row_map_16<D>(&tmQ, Q + first, prm.n_q, pitch, 128) || !make_row_map_16<D>(&tmO, O + first, prm.n_q, pitch, 128) ||
        !make_row_map_16<D>(&tmK, K + r * D, prm.n_keys, pitch, P::BN) ||
        !make_row_map_16<D>(&tmV, V + r * D, prm.n_keys, pitch, P::BN))
      return SPFA_ERR_LAUNCH;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((prm.n_q + 127) / 128));
    cfg.blockDim = dim3(P::kThreads);
    cfg.dynamicSmemBytes = P::kDynSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = launched ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, tile::band16_forward_kernel<D, T>, tmQ, tmK, tmV, tmO, m, l, O, V + r * D, prm, err) != cudaSuccess)
      return SPFA_ERR_LAUNCH;
    g_launches.fetch_add(1);
    launched = true;
  }
  g_last_path.store(SPFA_PATH_TILED);
  return launch_status();
}

inline int band16_forward(int dtype, const void* Q, const void* K, const void* V, void* m, void* l, void* O, int64_t L, int d,
                          int64_t w, int64_t s, int64_t row_begin, int64_t row_end, void* stream) {
  if (!Q || !K || !V || !m || !l || !O) return SPFA_ERR_BAD_ARG;
  if (!aligned16(Q) || !aligned16(K) || !aligned16(V) || !aligned16(O) || !aligned2(m) || !aligned2(l)) return SPFA_ERR_BAD_ARG;
  const int rc = check_rows(L, row_begin, row_end);
  if (rc) return rc;
  if (w < 0 || w > L - 1) return SPFA_ERR_LOCAL_SIZE;
  if (s < 1) return SPFA_ERR_DILATION_NEG;
  if (s > kTile16MaxStride) return SPFA_ERR_BAD_ARG;
  return with_shape_16(dtype, d, [&](auto* tag, auto dim) {
    using T = typename std::remove_pointer<decltype(tag)>::type;
    return launch_band16<decltype(dim)::value>((const T*)Q, (const T*)K, (const T*)V, (T*)m, (T*)l, (T*)O, L, w, s, row_begin,
                                               row_end, (cudaStream_t)stream);
  });
}

}  // namespace spfa

using namespace spfa;

extern "C" {

int spfa_tiled_16_usable(int dtype, int d, int64_t w, int64_t stride) {
  if (g_path.load() == SPFA_PATH_GATHER || w < kTile16MinHalfWidth || stride < 1 || stride > kTile16MaxStride) return 0;
  if (dtype == SPFA_DTYPE_F16 && w >= kTile16MaxHalfWidthF16) return 0;
  return with_shape_16(dtype, d, [&](auto* tag, auto dim) {
           using T = typename std::remove_pointer<decltype(tag)>::type;
           return band16_usable<decltype(dim)::value, T>() ? 1 : 0;
         }) == 1;
}

int spfa_local_forward_tiled_16(int dtype, const void* Q, const void* K, const void* V, void* m, void* l, void* O, int64_t L,
                                int d, int64_t w, int64_t row_begin, int64_t row_end, void* stream) {
  return band16_forward(dtype, Q, K, V, m, l, O, L, d, w, 1, row_begin, row_end, stream);
}

int spfa_local_1d_dilated_forward_tiled_16(int dtype, const void* Q, const void* K, const void* V, void* m, void* l, void* O,
                                           int64_t L, int d, int64_t w, int64_t dil, int64_t row_begin, int64_t row_end,
                                           void* stream) {
  if (dil < 0) return SPFA_ERR_DILATION_NEG;
  if (dil >= kTile16MaxStride) return SPFA_ERR_BAD_ARG;
  return band16_forward(dtype, Q, K, V, m, l, O, L, d, w, dil + 1, row_begin, row_end, stream);
}

}  // extern "C"
