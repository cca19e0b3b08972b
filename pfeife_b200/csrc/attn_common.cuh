// Shared by the attention forward (attn_sm100.cu) and backward (attn_bwd_sm100.cu): operand tiles in
// shared memory, the tcgen05 products over them, and the tensor maps of [B, S, H, D] views.
#pragma once
#include <cstring>
#include "common.cuh"

namespace pf {

constexpr int ATT_BM = 128;   // query rows per tile
constexpr int ATT_BN = 128;   // key rows per tile
constexpr int ATT_BLK = 16384;  // bytes of one [128 rows x 64 x 16-bit] swizzled block
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;

template <typename T>
__device__ __forceinline__ uint32_t pack2(float a, float b);
template <> __device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

// eight fp32 bit patterns -> 16 bytes of 16-bit values
template <typename T>
__device__ __forceinline__ uint4 pack8(const uint32_t* r) {
  return make_uint4(pack2<T>(__uint_as_float(r[0]), __uint_as_float(r[1])),
                    pack2<T>(__uint_as_float(r[2]), __uint_as_float(r[3])),
                    pack2<T>(__uint_as_float(r[4]), __uint_as_float(r[5])),
                    pack2<T>(__uint_as_float(r[6]), __uint_as_float(r[7])));
}

// 32 values of row `r` of a 16-bit box of 32 x 32 in the 64-byte swizzle
template <typename T>
__device__ __forceinline__ void box_row16(uint8_t* box, int r, const uint32_t (&v)[32]) {
#pragma unroll
  for (int c = 0; c < 4; ++c)
    *reinterpret_cast<uint4*>(box + r * 64 + ((c ^ ((r >> 1) & 3)) << 4)) = pack8<T>(v + c * 8);
}

// one [128 rows x DP] tile = DP/64 (rounded up) swizzled blocks, loaded with one TMA per block
template <int NBLK>
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* map, uint64_t* bar,
                                          int h, int s0, int b) {
  mbar_expect_tx(bar, NBLK * ATT_BLK);
#pragma unroll
  for (int i = 0; i < NBLK; ++i) tma_load_4d(dst + i * ATT_BLK, map, bar, i * 64, h, s0, b);
}

// Products over [128 rows x 64] blocks in shared memory, by the issuing thread.  Unrolled, so that a
// step costs an addition per operand.
// A[128 x K] (K-major blocks) . B[N x K]^T (K-major blocks), K = KSTEPS * 16
template <int KSTEPS>
__device__ __forceinline__ void mma_kk(uint32_t d_tmem, uint32_t sa, uint32_t sb, uint32_t idesc) {
  const uint32_t a = desc_lo(sa, 16), b = desc_lo(sb, 16);
#pragma unroll
  for (int k = 0; k < KSTEPS; ++k) {
    const uint32_t off = ((k >> 2) * ATT_BLK + (k & 3) * 32) >> 4;
    tc_mma_f16(d_tmem, a + off, b + off, idesc, k > 0);
  }
}
// A[128 x 128] K-major . B given as [K=128 rows][N] (N contiguous, MN-major blocks of 64)
__device__ __forceinline__ void mma_k_mn(uint32_t d_tmem, uint32_t sa, uint32_t sb, uint32_t idesc,
                                         bool accumulate_first, int ksteps) {
  const uint32_t a = desc_lo(sa, 16), b = desc_lo(sb, ATT_BLK);
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (k < ksteps)
      tc_mma_f16(d_tmem, a + (((k >> 2) * ATT_BLK + (k & 3) * 32) >> 4), b + (k * 2048 >> 4), idesc,
                 (k > 0) || accumulate_first);
}
// A given as [K=128 rows][M=128] (M contiguous) . B given as [K=128 rows][N] (N contiguous)
__device__ __forceinline__ void mma_mn_mn(uint32_t d_tmem, uint32_t sa, uint32_t sb, uint32_t idesc,
                                          int ksteps) {
  const uint32_t a = desc_lo(sa, ATT_BLK), b = desc_lo(sb, ATT_BLK);
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (k < ksteps) tc_mma_f16(d_tmem, a + (k * 2048 >> 4), b + (k * 2048 >> 4), idesc, k > 0);
}
// A in TMEM (16-bit pairs, 8 columns per step; its second half `half_cols` columns after the first),
// B given as [K=128 rows][N] (N contiguous)
__device__ __forceinline__ void mma_t_mn(uint32_t d_tmem, uint32_t ta, uint32_t half_cols, uint32_t sb,
                                         uint32_t idesc, bool accumulate_first, int ksteps) {
  const uint32_t b = desc_lo(sb, ATT_BLK);
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (k < ksteps)
      tc_mma_f16_ts(d_tmem, ta + (k >> 2) * half_cols + (k & 3) * 8, b + (k * 2048 >> 4), idesc,
                    (k > 0) || accumulate_first);
}

// ------------------------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeTiledFn attn_get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) ==
            cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

// [B, S, H, D] view with element strides (sb, ss, sh, 1); box = 64 x 1 x 128 x 1
inline int make_tmap_bshd(CUtensorMap* map, const void* base, int fmt, int B, int S, int H, int D,
                          long long sb, long long ss, long long sh) {
  EncodeTiledFn enc = attn_get_encode();
  if (!enc) return -100;
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)S, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)sh * 2, (cuuint64_t)ss * 2, (cuuint64_t)sb * 2};
  cuuint32_t box[4] = {64, 1, 128, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = enc(map, fmt ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                   4, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -(1000 + (int)r);
}

// 16-bit [B, S, H, D] view with element strides; box = 32 x 1 x 32 x 1 in the 64-byte swizzle
inline int make_tmap_box32(CUtensorMap* map, const void* base, int fmt, int B, int S, int H, int D,
                          const long long* st) {
  EncodeTiledFn enc = attn_get_encode();
  if (!enc) return -100;
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)S, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)st[2] * 2, (cuuint64_t)st[1] * 2, (cuuint64_t)st[0] * 2};
  cuuint32_t box[4] = {32, 1, 32, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = enc(map, fmt ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                   4, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                   CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -(1000 + (int)r);
}

// `done` must be a distinct array per kernel instantiation (kernels of equal signature share
// one function-pointer type), so the callers own it.
template <typename K>
inline int set_smem(K kern, int bytes, bool* done) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return (int)e;
    if (dev >= 0 && dev < 64) done[dev] = true;
  }
  return 0;
}

inline int attn_sm_count() {
  static int sms[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 148;
  if (!sms[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 148;
    sms[dev] = n;
  }
  return sms[dev];
}

inline bool strides_ok(const void* ptr, long long sb, long long ss, long long sh) {
  return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0 && sb % 8 == 0 && ss % 8 == 0 && sh % 8 == 0;
}

}  // namespace pf

#define PF_ATTN_DISPATCH(FN, ...)                                              \
  do {                                                                         \
    const int DP = (D + 31) / 32 * 32;                                         \
    if (dtype == PF_F16) {                                                     \
      switch (DP) {                                                            \
        case 32: return FN<__half, 32>(__VA_ARGS__);                            \
        case 64: return FN<__half, 64>(__VA_ARGS__);                            \
        case 96: return FN<__half, 96>(__VA_ARGS__);                            \
        case 128: return FN<__half, 128>(__VA_ARGS__);                          \
      }                                                                        \
    } else {                                                                   \
      switch (DP) {                                                            \
        case 32: return FN<__nv_bfloat16, 32>(__VA_ARGS__);                     \
        case 64: return FN<__nv_bfloat16, 64>(__VA_ARGS__);                     \
        case 96: return FN<__nv_bfloat16, 96>(__VA_ARGS__);                     \
        case 128: return FN<__nv_bfloat16, 128>(__VA_ARGS__);                   \
      }                                                                        \
    }                                                                          \
    return -3;                                                                 \
  } while (0)
