// UNet support kernels, channels-last (NHWC) throughout:
//   * im2col / col2im for KxK convolutions: the convolution itself runs on the tcgen05 GEMM
//     (forward: cols . W^T ; dgrad: dY . W -> col2im ; wgrad: dY^T . cols accumulated in fp32).
//     1x1 convolutions skip these kernels entirely (they are plain GEMMs on the NHWC tensor).
//   * GroupNorm with optional fused SiLU, forward and backward.
//   * nearest-neighbour 2x upsampling and its backward.
#include <type_traits>
#include "common.cuh"
#include "api.h"

namespace pf {

// cols[(b, ho, wo), (r, s, c)] = x[b, ho*stride - pad + r, wo*stride - pad + s, c]  (0 outside)
// One thread moves 8 channels (16 bytes).
template <typename T>
__global__ void __launch_bounds__(256)
im2col_kernel(const T* __restrict__ x, T* __restrict__ cols, int B, int H, int W, int C, int KH,
              int KW, int Ho, int Wo, int stride, int pad, long long ldc) {
  after_previous();
  const int cv = C / 8;
  const long long total = (long long)B * Ho * Wo * KH * KW * cv;
  const long long gstride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gstride) {
    const int c8 = (int)(i % cv);
    long long t = i / cv;
    const int s = (int)(t % KW); t /= KW;
    const int r = (int)(t % KH); t /= KH;
    const int wo = (int)(t % Wo); t /= Wo;
    const int ho = (int)(t % Ho);
    const int b = (int)(t / Ho);
    const int hi = ho * stride - pad + r, wi = wo * stride - pad + s;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (hi >= 0 && hi < H && wi >= 0 && wi < W)
      v = reinterpret_cast<const uint4*>(x + (((long long)b * H + hi) * W + wi) * C)[c8];
    const long long row = ((long long)b * Ho + ho) * Wo + wo;
    reinterpret_cast<uint4*>(cols + row * ldc + ((long long)r * KW + s) * C)[c8] = v;
  }
}

// dx[b, hi, wi, c] = sum over (r, s) of dcols[(b, ho, wo), (r, s, c)] with hi = ho*stride-pad+r
// Gather form (no atomics): each thread owns 8 channels of one input pixel.
template <typename T>
__global__ void __launch_bounds__(256)
col2im_kernel(const T* __restrict__ dcols, T* __restrict__ dx, int B, int H, int W, int C, int KH,
              int KW, int Ho, int Wo, int stride, int pad, long long ldc) {
  after_previous();
  const int cv = C / 8;
  const long long total = (long long)B * H * W * cv;
  const long long gstride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gstride) {
    const int c8 = (int)(i % cv);
    long long t = i / cv;
    const int wi = (int)(t % W); t /= W;
    const int hi = (int)(t % H);
    const int b = (int)(t / H);
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int r = 0; r < KH; ++r) {
      const int hn = hi + pad - r;
      if (hn < 0 || hn % stride) continue;
      const int ho = hn / stride;
      if (ho >= Ho) continue;
      for (int s = 0; s < KW; ++s) {
        const int wn = wi + pad - s;
        if (wn < 0 || wn % stride) continue;
        const int wo = wn / stride;
        if (wo >= Wo) continue;
        const long long row = ((long long)b * Ho + ho) * Wo + wo;
        uint4 q = reinterpret_cast<const uint4*>(dcols + row * ldc + ((long long)r * KW + s) * C)[c8];
        const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += to_f32<T>(e[j]);
      }
    }
    uint4 o;
    T* e = reinterpret_cast<T*>(&o);
#pragma unroll
    for (int j = 0; j < 8; ++j) e[j] = from_f32<T>(acc[j]);
    reinterpret_cast<uint4*>(dx + (((long long)b * H + hi) * W + wi) * C)[c8] = o;
  }
}

// ------------------------------------------------------------------------------ conv weights
// Between the [Cout, Cin, taps] order of a convolution's weight and the orders its products read.
// Each CTA moves a tile through shared memory so that both sides are contiguous in global memory,
// 16 bytes a thread and request (`vec`: the weight's rows start on 16 bytes; else element by
// element); rows and channels beyond Cout / Cin (the products need multiples of 8) are zero.
// Bound by the latency of one short pass through L2.  640 x 640 x 9 bf16: packed 4.2 us, flipped
// 6.0, gradient 7.8 (with 2 bytes a request 9.9, 17.4 and 12.6, as strided copies 8.1, 25.5 and
// 12.9).  Convolution forward and backward, bf16: 640 -> 640 channels on [4, 64, 64] 546 -> 509 us
// against strided copies, 2560 -> 1280 on [1, 32, 32] 807 -> 511 us.
constexpr int CONV_PACK_TAPS = 64;     // most taps (7 x 7 fits)
constexpr int CONV_TILE = 4096;        // elements of a tile: 8 channels of 64 taps fit

// out[co, t, ci] = w[co, ci, t]; a tile is `per` channels (a multiple of 8) of one co
__global__ void __launch_bounds__(128)
conv_pack_kernel(const uint16_t* __restrict__ w, uint16_t* __restrict__ out, int Cout, int Cin,
                 int taps, int cin8, int per, int vec) {
  after_previous();
  __shared__ __align__(16) uint16_t tile[CONV_TILE];
  const int co = blockIdx.x, ci0 = blockIdx.y * per;
  const int n_in = co < Cout ? max(0, min(per, Cin - ci0)) : 0, n_out = min(per, cin8 - ci0) / 8;
  const uint16_t* src = w + ((long long)co * Cin + ci0) * taps;
  if (vec) {
    for (int i = threadIdx.x; i < n_in * taps / 8; i += 128)
      reinterpret_cast<uint4*>(tile)[i] = __ldg(reinterpret_cast<const uint4*>(src) + i);
  } else {
    for (int i = threadIdx.x; i < n_in * taps; i += 128) tile[i] = src[i];
  }
  __syncthreads();
  uint16_t* dst = out + (long long)co * taps * cin8 + ci0;
  for (int i = threadIdx.x; i < taps * n_out; i += 128) {
    const int t = i / n_out, c = (i - t * n_out) * 8;
    uint4 q;
    uint16_t* e = reinterpret_cast<uint16_t*>(&q);
#pragma unroll
    for (int j = 0; j < 8; ++j) e[j] = c + j < n_in ? tile[(c + j) * taps + t] : 0;
    *reinterpret_cast<uint4*>(dst + (long long)t * cin8 + c) = q;
  }
}

// out[ci, taps - 1 - t, co] = w[co, ci, t]: taps flipped, channel roles swapped; a tile is 8 input
// channels of `per` output channels (a multiple of 8)
__global__ void __launch_bounds__(256)
conv_pack_flip_kernel(const uint16_t* __restrict__ w, uint16_t* __restrict__ out, int Cout, int Cin,
                      int taps, int cout8, int per, int vec) {
  after_previous();
  // [per][8 * taps + 2]: rows lie an odd number of words apart
  extern __shared__ __align__(16) uint16_t ftile[];
  const int ci0 = blockIdx.x * 8, co0 = blockIdx.y * per;
  const int n_ci = max(0, min(8, Cin - ci0)), n_co = max(0, min(per, Cout - co0));
  const int row = n_ci * taps, pitch = 8 * taps + 2;
  const uint16_t* src = w + ((long long)co0 * Cin + ci0) * taps;
  if (vec) {
    for (int i = threadIdx.x; i < n_co * (row / 8); i += 256) {
      const int c = i / (row / 8), k = (i - c * (row / 8)) * 8;
      const uint4 q = __ldg(reinterpret_cast<const uint4*>(src + (long long)c * Cin * taps + k));
      uint32_t* d = reinterpret_cast<uint32_t*>(ftile + c * pitch + k);
      d[0] = q.x; d[1] = q.y; d[2] = q.z; d[3] = q.w;
    }
  } else {
    for (int i = threadIdx.x; i < n_co * row; i += 256) {
      const int c = i / row, k = i - c * row;
      ftile[c * pitch + k] = src[(long long)c * Cin * taps + k];
    }
  }
  __syncthreads();
  const int o_co = min(per, cout8 - co0) / 8;
  for (int i = threadIdx.x; i < 8 * taps * o_co; i += 256) {
    const int k = i / o_co, c = (i - k * o_co) * 8, ci = k / taps, t = k - ci * taps;
    uint4 q;
    uint16_t* e = reinterpret_cast<uint16_t*>(&q);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      e[j] = (c + j < n_co && ci < n_ci) ? ftile[(c + j) * pitch + k] : 0;
    *reinterpret_cast<uint4*>(out + ((long long)(ci0 + ci) * taps + (taps - 1 - t)) * cout8 + co0 +
                              c) = q;
  }
}

// dw[co, ci, t] = src[co, t, ci] (fp32 sums with cin8 channels a row), converted to the weight's
// type; a tile is `per` channels (a multiple of 8) of one co
template <typename T>
__global__ void __launch_bounds__(128)
conv_unpack_kernel(const float* __restrict__ src, T* __restrict__ dw, int Cin, int taps, int cin8,
                   int per, int vec) {
  after_previous();
  constexpr int V = 16 / sizeof(T);
  __shared__ float tile[CONV_TILE + 64];
  const int co = blockIdx.x, ci0 = blockIdx.y * per, n = min(per, Cin - ci0);
  const int pitch = taps | 1;          // odd: the transposing stores spread over the banks
  const int n4 = (n + 3) / 4;          // a row of sums has channels up to a multiple of 8
  const float* s0 = src + (long long)co * taps * cin8 + ci0;
  for (int i = threadIdx.x; i < taps * n4; i += 128) {
    const int t = i / n4, c = (i - t * n4) * 4;
    const float4 q = __ldg(reinterpret_cast<const float4*>(s0 + (long long)t * cin8 + c));
    float* d = tile + c * pitch + t;
    d[0] = q.x; d[pitch] = q.y; d[2 * pitch] = q.z; d[3 * pitch] = q.w;
  }
  __syncthreads();
  T* dst = dw + ((long long)co * Cin + ci0) * taps;
  const int step = vec ? V : 1;
  for (int i = threadIdx.x * step; i < n * taps; i += 128 * step) {
    int c = i / taps, t = i - c * taps;
    if (!vec) { dst[i] = from_f32<T>(tile[c * pitch + t]); continue; }
    uint4 q;
    T* e = reinterpret_cast<T*>(&q);
#pragma unroll
    for (int j = 0; j < V; ++j) {
      e[j] = from_f32<T>(tile[c * pitch + t]);
      if (++t == taps) { t = 0; ++c; }
    }
    *reinterpret_cast<uint4*>(dst + i) = q;
  }
}

// ------------------------------------------------------------------------------ GroupNorm
// NHWC, C a multiple of 8, three launches per direction: per-channel sums of slabs of pixels, a
// fold of the slabs, and the element-wise pass (which finds a tensor of up to the L2's size there).
// Every thread of the first and third owns one 8-channel vector and a stripe of pixels: the CTA is
// (C/8) columns x R rows of threads, the grid (slabs, B), so whatever depends on the channel
// alone (group, mean, scale) is looked up once per thread and not per element.  The sums of a slab
// go to scratch (per group [B, slabs, 2, G], in the backward per channel [B, slabs, 2, C] as well):
// nothing to clear, no atomics, the same result every time.
// Bound by memory and, below some 10 MB, by the latency of three dependent launches.
// [4, 128, 128, 320] bf16, L2 flushed: forward 82 -> 46 us, backward 124 -> 83, now 64 (atomics into
// cleared sums, a division and four lookups per element before).

// rows of C/8 threads in a CTA
static inline int gn_rows(int C) { const int ncv = C / 8; return ncv >= 256 ? 1 : 256 / ncv; }

// Slabs of pixels per image, at least eight pixels per thread.  `per_sm` CTAs of up to 256 threads per
// SM make one wave: 4 of the forward's, at 41 registers and at 64, which the bound of 1024 threads holds them to,
// and 3 of the backward's at 80 (4 left a third of them to a second wave: 110 us against 83).
constexpr int GN_FWD_PER_SM = 4, GN_BWD_PER_SM = 3;
static inline int gn_slabs(int B, int HW, int rows, int sm_count, int per_sm) {
  int slabs = (per_sm * (sm_count > 0 ? sm_count : 148)) / B;
  const int most = (HW + 8 * rows - 1) / (8 * rows);
  if (slabs > most) slabs = most;
  return slabs < 1 ? 1 : slabs;
}

// The backward's two passes over dy and x run out of registers before they have enough loads under
// way: each thread keeps a ring of its next pixels in shared memory, filled by asynchronous copies of
// its own, which needs no barriers.  Four sizes of CTA: up to 256 threads (2048 channels) and up to 400
// with a ring, up to 800 and up to 1024 (8192 channels) without.  They compile to 80, 72, 72 and 64
// registers; the second pass with SiLU spills 44, 64, 8 and 88 bytes per thread, the first 4, 32, 36 and
// 124, the others next to nothing.  Without a ring the loads of two pixels go out together only as
// read-only ones, past the store between them ([4, 32, 32, 6080] 134 us, now 116).  Up to 256 threads three CTAs share an SM, up to 400 two, beyond one,
// while the slabs are cut for three: wider images take more than one wave.  Backward, both passes and
// the fold, L2 flushed: [4, 128, 128, 320] 78 -> 64 us, [4, 128, 128, 640] 141 -> 102,
// [4, 64, 64, 1920] 108 -> 85, [4, 32, 32, 2560] 65 -> 57.
constexpr int GN_RING = 6, GN_RING_THREADS = 400;
// fold and ring of 400 threads
constexpr int GN_MAX_SMEM = 2 * 8 * GN_RING_THREADS * 4 + GN_RING * 2 * GN_RING_THREADS * 16;
constexpr int gn_min_ctas(int max_threads) {
  return max_threads <= 256 ? GN_BWD_PER_SM : max_threads <= GN_RING_THREADS ? 2 : 1;
}
static inline int gn_ring_smem(int threads) {
  return threads <= GN_RING_THREADS ? GN_RING * 2 * threads * 16 : 0;
}

// dz of two channels: dy times the derivative of the activation at z = xhat * gamma + beta
template <bool SILU>
__device__ __forceinline__ uint64_t gn_dz2(uint64_t dy, uint64_t xhat, uint64_t ga, uint64_t be) {
  if (!SILU) return dy;
  const uint64_t z = fma2(xhat, ga, be), one = f2_pack(1.f, 1.f);
  float a, b;
  f2_unpack(mul2(z, f2_pack(-1.4426950408889634f, -1.4426950408889634f)), a, b);
  f2_unpack(add2(f2_pack(exp2f(a), exp2f(b)), one), a, b);
  const uint64_t s = f2_pack(rcp_approx(a), rcp_approx(b));
  // s (1 + z (1 - s))
  return mul2(dy, mul2(s, fma2(z, fma2(s, f2_pack(-1.f, -1.f), one), one)));
}

// shared memory of a fold: [rows][2][C] sums (16 KB, or 8 bytes per channel when rows is 1)
static inline int gn_smem(int rows, int C) { return rows * 2 * C * (int)sizeof(float); }

// folds the rows of a CTA: every thread brings 8 + 8 sums of its channels; leaves [2][C] in `chan`
__device__ __forceinline__ void gn_fold(float* chan, const float (&a)[8], const float (&q)[8],
                                        int c0, int r, int rows, int C) {
  float4* d0 = reinterpret_cast<float4*>(chan + r * 2 * C + c0);
  float4* d1 = reinterpret_cast<float4*>(chan + r * 2 * C + C + c0);
  d0[0] = make_float4(a[0], a[1], a[2], a[3]);
  d0[1] = make_float4(a[4], a[5], a[6], a[7]);
  d1[0] = make_float4(q[0], q[1], q[2], q[3]);
  d1[1] = make_float4(q[4], q[5], q[6], q[7]);
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * C; i += blockDim.x) {
    float t = chan[i];
    for (int k = 1; k < rows; ++k) t += chan[k * 2 * C + i];
    chan[i] = t;                        // read by this thread alone
  }
  __syncthreads();
}

// 41 registers, without a bound on its CTAs: with one it comes out at 43 and 2 to 7 % slower.
template <typename T>
__global__ void gn_stats_kernel(const T* __restrict__ x, float* __restrict__ part, int HW, int C,
                                int G, int rows) {
  after_previous();
  extern __shared__ __align__(16) float chan[];       // [rows][2][C]
  const int ncv = C / 8;
  const int cv = threadIdx.x % ncv, r = threadIdx.x / ncv;
  const int b = blockIdx.y;
  const int per = (HW + gridDim.x - 1) / gridDim.x;
  const int p0 = blockIdx.x * per, p1 = min(HW, p0 + per);
  float s[8] = {0, 0, 0, 0, 0, 0, 0, 0}, q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const T* base = x + (long long)b * HW * C + cv * 8;
#pragma unroll 8
  for (int p = p0 + r; p < p1; p += rows) {
    const uint4 u = *reinterpret_cast<const uint4*>(base + (long long)p * C);
    const T* e = reinterpret_cast<const T*>(&u);
#pragma unroll
    for (int j = 0; j < 8; ++j) { const float v = to_f32<T>(e[j]); s[j] += v; q[j] = fmaf(v, v, q[j]); }
  }
  gn_fold(chan, s, q, cv * 8, r, rows, C);
  const int cpg = C / G;
  float* out = part + ((long long)b * gridDim.x + blockIdx.x) * 2 * G;
  for (int i = threadIdx.x; i < 2 * G; i += blockDim.x) {
    const float* p = chan + i * cpg;      // [0, G): sums, [G, 2G): squares (at chan + C)
    float t = 0.f;
    for (int j = 0; j < cpg; ++j) t += p[j];
    out[i] = t;
  }
}

// sums of one group over the slabs -> (mean, rstd); one warp per (group, image)
__global__ void __launch_bounds__(128)
gn_finalize_kernel(const float* __restrict__ part, float* __restrict__ mean,
                   float* __restrict__ rstd, int slabs, int G, int n_groups, float inv_n,
                   float eps) {
  after_previous();
  const int i = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= n_groups) return;
  const int b = i / G, g = i - b * G;
  const float* p = part + (long long)b * slabs * 2 * G + g;
  float a = 0.f, c = 0.f;
#pragma unroll 4
  for (int s = lane; s < slabs; s += 32) {
    a += p[(long long)s * 2 * G];
    c += p[(long long)s * 2 * G + G];
  }
  a = warp_sum(a);
  c = warp_sum(c);
  if (lane == 0) {
    const float m = a * inv_n;
    mean[i] = m;
    rstd[i] = rsqrtf(fmaxf(c * inv_n - m * m, 0.f) + eps);
  }
}

// y = act((x - mean) * rstd * gamma + beta), act = SiLU or identity.  With SiLU two special-function
// instructions per value bound it (9 of 13 us at [4, 128, 128, 320]), so the others work on pairs and the
// next GN_AHEAD pixels are on their way while these are worked on (20 us with single values and loads
// that waited for the stores before).
constexpr int GN_AHEAD = 2;
template <typename T, bool SILU>
__global__ void __launch_bounds__(1024) gn_apply_kernel(const T* __restrict__ x, const float* __restrict__ mean,
                                const float* __restrict__ rstd, const float* __restrict__ gamma,
                                const float* __restrict__ beta, T* __restrict__ y, int HW, int C,
                                int G, int rows) {
  after_previous();
  const int ncv = C / 8, cpg = C / G;
  const int cv = threadIdx.x % ncv, r = threadIdx.x / ncv;
  const int b = blockIdx.y, c0 = cv * 8;
  const int per = (HW + gridDim.x - 1) / gridDim.x;
  const int p0 = blockIdx.x * per + r, p1 = min(HW, (int)(blockIdx.x + 1) * per);
  const long long off = (long long)b * HW * C + c0;
  auto load = [&](int p) {
    return p < p1 ? __ldg(reinterpret_cast<const uint4*>(x + off + (long long)p * C))
                  : make_uint4(0, 0, 0, 0);
  };
  uint4 next[GN_AHEAD];
#pragma unroll
  for (int u = 0; u < GN_AHEAD; ++u) next[u] = load(p0 + u * rows);
  uint64_t nm[4], sc[4], be[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int c = c0 + 2 * j, s0 = b * G + c / cpg, s1 = b * G + (c + 1) / cpg;
    nm[j] = f2_pack(-mean[s0], -mean[s1]);
    sc[j] = f2_pack(rstd[s0] * gamma[c], rstd[s1] * gamma[c + 1]);
    be[j] = f2_pack(beta[c], beta[c + 1]);
  }
  for (int p = p0; p < p1; p += GN_AHEAD * rows) {
    uint4 now[GN_AHEAD];
#pragma unroll
    for (int u = 0; u < GN_AHEAD; ++u) {
      now[u] = next[u];
      next[u] = load(p + (GN_AHEAD + u) * rows);
    }
#pragma unroll
    for (int u = 0; u < GN_AHEAD; ++u) {
      const T* e = reinterpret_cast<const T*>(&now[u]);
      uint4 o;
      T* oe = reinterpret_cast<T*>(&o);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint64_t v = fma2(add2(f2_pack(to_f32<T>(e[2 * j]), to_f32<T>(e[2 * j + 1])), nm[j]), sc[j], be[j]);
        float a, c;
        if (SILU) {
          f2_unpack(mul2(v, f2_pack(-1.4426950408889634f, -1.4426950408889634f)), a, c);
          f2_unpack(add2(f2_pack(exp2f(a), exp2f(c)), f2_pack(1.f, 1.f)), a, c);
          v = mul2(v, f2_pack(rcp_approx(a), rcp_approx(c)));
        }
        f2_unpack(v, a, c);
        oe[2 * j] = from_f32<T>(a);
        oe[2 * j + 1] = from_f32<T>(c);
      }
      if (p + u * rows < p1) *reinterpret_cast<uint4*>(y + off + (long long)(p + u * rows) * C) = o;
    }
  }
}

// Calls f(p, x, dy) for pixels p = p0, p0 + rows, ... below p1 with a thread's 8 channels of both
// tensors as pairs of fp32 values
template <typename T, bool RING, typename F>
__device__ __forceinline__ void gn_pixels(const T* x, const T* dy, float* ring, int p0, int p1,
                                          int rows, int C, F f) {
  auto work = [&](int p, const uint4& ux, const uint4& ud) {
    const T* ex = reinterpret_cast<const T*>(&ux);
    const T* ed = reinterpret_cast<const T*>(&ud);
    uint64_t vx[4], vd[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      vx[j] = f2_pack(to_f32<T>(ex[2 * j]), to_f32<T>(ex[2 * j + 1]));
      vd[j] = f2_pack(to_f32<T>(ed[2 * j]), to_f32<T>(ed[2 * j + 1]));
    }
    f(p, vx, vd);
  };
  if constexpr (RING) {
    auto slot = [&](int st, int which) {
      return reinterpret_cast<uint4*>(ring) + (st * 2 + which) * blockDim.x + threadIdx.x;
    };
    auto fetch = [&](int p, int st) {
      if (p < p1) {
        cp_async16(slot(st, 0), x + (long long)p * C);
        cp_async16(slot(st, 1), dy + (long long)p * C);
      }
      cp_async_commit();               // an empty group past the last pixel
    };
#pragma unroll
    for (int i = 0; i < GN_RING - 1; ++i) fetch(p0 + i * rows, i);
    int st = 0;
    for (int p = p0; p < p1; p += rows) {
      cp_async_wait<GN_RING - 2>();
      const uint4 ux = *slot(st, 0), ud = *slot(st, 1);
      fetch(p + (GN_RING - 1) * rows, st == 0 ? GN_RING - 1 : st - 1);   // read in the last round
      st = st == GN_RING - 1 ? 0 : st + 1;
      work(p, ux, ud);
    }
  } else {
#pragma unroll 2
    for (int p = p0; p < p1; p += rows)
      work(p, __ldg(reinterpret_cast<const uint4*>(x + (long long)p * C)),
           __ldg(reinterpret_cast<const uint4*>(dy + (long long)p * C)));
  }
}

// Backward pass 1: per-channel sums of dz * xhat and dz (dz = dy * act'(z)); over all slabs they
// are the parameter gradients (dgamma, dbeta) and, weighted by gamma and folded per group, the two
// sums A = sum(dz * gamma), Bq = sum(dz * gamma * xhat) the second pass needs.
template <typename T, bool SILU, int MAXT>
__global__ void __launch_bounds__(MAXT, gn_min_ctas(MAXT))
gn_bwd_stats_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                    const float* __restrict__ mean, const float* __restrict__ rstd,
                    const float* __restrict__ gamma, const float* __restrict__ beta,
                    float* __restrict__ part, float* __restrict__ gpart, int HW,
                    int C, int G, int rows) {
  after_previous();
  extern __shared__ __align__(16) float chan[];       // [rows][2][C]: sum dz * xhat, sum dz; the ring
  const int ncv = C / 8, cpg = C / G;
  const int cv = threadIdx.x % ncv, r = threadIdx.x / ncv;
  const int b = blockIdx.y, c0 = cv * 8;
  uint64_t nm[4], rs[4], ga[4], be[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int s0 = b * G + (c0 + 2 * j) / cpg, s1 = b * G + (c0 + 2 * j + 1) / cpg;
    nm[j] = f2_pack(-mean[s0], -mean[s1]);
    rs[j] = f2_pack(rstd[s0], rstd[s1]);
    ga[j] = f2_pack(gamma[c0 + 2 * j], gamma[c0 + 2 * j + 1]);
    be[j] = f2_pack(beta[c0 + 2 * j], beta[c0 + 2 * j + 1]);
  }
  const int per = (HW + gridDim.x - 1) / gridDim.x;
  const int p0 = blockIdx.x * per, p1 = min(HW, p0 + per);
  uint64_t sx2[4] = {0, 0, 0, 0}, sd2[4] = {0, 0, 0, 0};
  const long long off = (long long)b * HW * C + c0;
  gn_pixels<T, (MAXT <= GN_RING_THREADS)>(x + off, dy + off, chan + rows * 2 * C, p0 + r, p1, rows, C,
                     [&](int, const uint64_t (&vx)[4], const uint64_t (&vd)[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint64_t xhat = mul2(add2(vx[j], nm[j]), rs[j]);
      const uint64_t dz = gn_dz2<SILU>(vd[j], xhat, ga[j], be[j]);
      sd2[j] = add2(sd2[j], dz);
      sx2[j] = fma2(dz, xhat, sx2[j]);
    }
  });
  float sx[8], sd[8];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    f2_unpack(sx2[j], sx[2 * j], sx[2 * j + 1]);
    f2_unpack(sd2[j], sd[2 * j], sd[2 * j + 1]);
  }
  gn_fold(chan, sx, sd, c0, r, rows, C);
  const long long slab = (long long)b * gridDim.x + blockIdx.x;
  for (int i = threadIdx.x; i < 2 * C; i += blockDim.x) part[slab * 2 * C + i] = chan[i];
  for (int i = threadIdx.x; i < 2 * G; i += blockDim.x) {
    // [0, G): sum gamma dz xhat, [G, 2G): sum gamma dz
    const int g = i < G ? i : i - G;
    float t = 0.f;
    for (int j = 0; j < cpg; ++j) t = fmaf(gamma[g * cpg + j], chan[i * cpg + j], t);
    gpart[slab * 2 * G + i] = t;
  }
}

// Folds the slabs.  The first CTAs: one warp per (group, image), A and Bq.  The others: 32 channels
// each, dgamma and dbeta over all images and slabs, shared by the 32 warps.
__global__ void __launch_bounds__(1024)
gn_bwd_fold_kernel(const float* __restrict__ part, const float* __restrict__ gpart,
                   float* __restrict__ sumA, float* __restrict__ sumB, float* __restrict__ dgamma,
                   float* __restrict__ dbeta, int B, int slabs, int C, int G) {
  after_previous();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int group_ctas = (B * G + 31) / 32;
  if ((int)blockIdx.x < group_ctas) {
    const int i = blockIdx.x * 32 + warp;
    if (i >= B * G) return;
    const int b = i / G, g = i - b * G;
    const float* p = gpart + (long long)b * slabs * 2 * G + g;
    float a = 0.f, q = 0.f;
#pragma unroll 4
    for (int s = lane; s < slabs; s += 32) {
      q += p[(long long)s * 2 * G];
      a += p[(long long)s * 2 * G + G];
    }
    a = warp_sum(a);
    q = warp_sum(q);
    if (lane == 0) { sumA[i] = a; sumB[i] = q; }
    return;
  }
  __shared__ float red[2][32][33];
  const int c = ((int)blockIdx.x - group_ctas) * 32 + lane;
  float g = 0.f, d = 0.f;
  if (c < C) {
#pragma unroll 4
    for (int k = warp; k < B * slabs; k += 32) {
      g += part[(long long)k * 2 * C + c];
      d += part[(long long)k * 2 * C + C + c];
    }
  }
  red[0][lane][warp] = g;
  red[1][lane][warp] = d;
  __syncthreads();
  // warp w finishes channel w of the 32
  const int cw = ((int)blockIdx.x - group_ctas) * 32 + warp;
  g = warp_sum(red[0][warp][lane]);
  d = warp_sum(red[1][warp][lane]);
  if (lane == 0 && cw < C) {
    dgamma[cw] = g;
    dbeta[cw] = d;
  }
}

// Backward pass 2: dx = rstd * (dz*gamma - A/n - xhat * B/n)
template <typename T, bool SILU, int MAXT>
__global__ void __launch_bounds__(MAXT, gn_min_ctas(MAXT))
gn_bwd_apply_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                    const float* __restrict__ mean, const float* __restrict__ rstd,
                    const float* __restrict__ gamma, const float* __restrict__ beta,
                    const float* __restrict__ sumA, const float* __restrict__ sumB,
                    T* __restrict__ dx, int HW, int C, int G, int rows) {
  after_previous();
  extern __shared__ __align__(16) float ring[];
  const int ncv = C / 8, cpg = C / G;
  const float inv_n = 1.f / ((float)HW * cpg);
  const int cv = threadIdx.x % ncv, r = threadIdx.x / ncv;
  const int b = blockIdx.y, c0 = cv * 8;
  uint64_t nm[4], rs[4], ga[4], be[4], nA[4], nB[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int s0 = b * G + (c0 + 2 * j) / cpg, s1 = b * G + (c0 + 2 * j + 1) / cpg;
    nm[j] = f2_pack(-mean[s0], -mean[s1]);
    rs[j] = f2_pack(rstd[s0], rstd[s1]);
    ga[j] = f2_pack(gamma[c0 + 2 * j], gamma[c0 + 2 * j + 1]);
    be[j] = f2_pack(beta[c0 + 2 * j], beta[c0 + 2 * j + 1]);
    nA[j] = f2_pack(-sumA[s0] * inv_n, -sumA[s1] * inv_n);
    nB[j] = f2_pack(-sumB[s0] * inv_n, -sumB[s1] * inv_n);
  }
  const int per = (HW + gridDim.x - 1) / gridDim.x;
  const int p0 = blockIdx.x * per, p1 = min(HW, p0 + per);
  const long long off = (long long)b * HW * C + c0;
  gn_pixels<T, (MAXT <= GN_RING_THREADS)>(x + off, dy + off, ring, p0 + r, p1, rows, C,
                     [&](int p, const uint64_t (&vx)[4], const uint64_t (&vd)[4]) {
    uint4 o;
    T* oe = reinterpret_cast<T*>(&o);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint64_t xhat = mul2(add2(vx[j], nm[j]), rs[j]);
      const uint64_t dz = gn_dz2<SILU>(vd[j], xhat, ga[j], be[j]);
      float a0, a1;
      f2_unpack(mul2(rs[j], fma2(xhat, nB[j], fma2(dz, ga[j], nA[j]))), a0, a1);
      oe[2 * j] = from_f32<T>(a0);
      oe[2 * j + 1] = from_f32<T>(a1);
    }
    *reinterpret_cast<uint4*>(dx + off + (long long)p * C) = o;
  });
}

// nearest 2x upsample (NHWC) and its backward (sum of the 4 children)
template <typename T>
__global__ void __launch_bounds__(256)
upsample2x_kernel(const T* __restrict__ x, T* __restrict__ y, int B, int H, int W, int C,
                  int backward) {
  after_previous();
  const int cv = C / 8;
  const long long total = backward ? (long long)B * H * W * cv : (long long)B * 4 * H * W * cv;
  const long long gstride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gstride) {
    const int c8 = (int)(i % cv);
    long long t = i / cv;
    if (!backward) {
      const int wo = (int)(t % (2 * W)); t /= 2 * W;
      const int ho = (int)(t % (2 * H));
      const int b = (int)(t / (2 * H));
      reinterpret_cast<uint4*>(y + (((long long)b * 2 * H + ho) * 2 * W + wo) * C)[c8] =
          reinterpret_cast<const uint4*>(x + (((long long)b * H + ho / 2) * W + wo / 2) * C)[c8];
    } else {   // x = dy [B, 2H, 2W, C], y = dx [B, H, W, C]
      const int wi = (int)(t % W); t /= W;
      const int hi = (int)(t % H);
      const int b = (int)(t / H);
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      for (int dh = 0; dh < 2; ++dh)
        for (int dw = 0; dw < 2; ++dw) {
          uint4 q = reinterpret_cast<const uint4*>(
              x + (((long long)b * 2 * H + 2 * hi + dh) * 2 * W + 2 * wi + dw) * C)[c8];
          const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[j] += to_f32<T>(e[j]);
        }
      uint4 o;
      T* e = reinterpret_cast<T*>(&o);
#pragma unroll
      for (int j = 0; j < 8; ++j) e[j] = from_f32<T>(acc[j]);
      reinterpret_cast<uint4*>(y + (((long long)b * H + hi) * W + wi) * C)[c8] = o;
    }
  }
}

static inline int grid_for(long long n, int sm_count) {
  long long b = (n + 255) / 256;
  const long long cap = (long long)(sm_count > 0 ? sm_count : 148) * 16;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}

}  // namespace pf

using namespace pf;

#define PF_DISPATCH_H(dtype, ...)                               \
  switch (dtype) {                                             \
    case PF_F16: { using T = __half; __VA_ARGS__; } break;      \
    case PF_BF16: { using T = __nv_bfloat16; __VA_ARGS__; } break; \
    default: return -1;                                        \
  }

PF_API int pf_im2col(const void* x, void* cols, int B, int H, int W, int C, int KH, int KW, int Ho,
                     int Wo, int stride, int pad, long long ldc, int dtype, int sm_count,
                     void* stream) {
  if (C % 8 || ldc % 8 || !on_vectors(x, cols)) return -2;
  const long long total = (long long)B * Ho * Wo * KH * KW * (C / 8);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  PF_DISPATCH_H(dtype, (after(im2col_kernel<T>, grid_for(total, sm_count), 256, 0, st)(
      (const T*)x, (T*)cols, B, H, W, C, KH, KW, Ho, Wo, stride, pad, ldc)));
  PF_CHECK_LAUNCH();
  return 0;
}

PF_API int pf_col2im(const void* dcols, void* dx, int B, int H, int W, int C, int KH, int KW,
                     int Ho, int Wo, int stride, int pad, long long ldc, int dtype, int sm_count,
                     void* stream) {
  if (C % 8 || ldc % 8 || !on_vectors(dcols, dx)) return -2;
  const long long total = (long long)B * H * W * (C / 8);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  PF_DISPATCH_H(dtype, (after(col2im_kernel<T>, grid_for(total, sm_count), 256, 0, st)(
      (const T*)dcols, (T*)dx, B, H, W, C, KH, KW, Ho, Wo, stride, pad, ldc)));
  PF_CHECK_LAUNCH();
  return 0;
}

// slabs per image of the two entry points below; they need scratch of B * slabs * 2 * G floats
// (forward) and B * slabs * 2 * (C + G) floats (backward)
PF_API int pf_groupnorm_slabs(int B, int HW, int C, int sm_count) {
  return C >= 8 ? gn_slabs(B, HW, gn_rows(C), sm_count, GN_FWD_PER_SM) : 1;
}

#define PF_GN_SILU(KERN, ...)                                 \
  do {                                                        \
    if (act_silu) after(KERN<T, true>, grid, threads, smem, st)(__VA_ARGS__); \
    else after(KERN<T, false>, grid, threads, smem, st)(__VA_ARGS__);         \
  } while (0)

// `done`: per kernel and device, whether it may already use more than 48 KB of shared memory
template <typename... P, typename... A>
static int gn_launch(void (*kern)(P...), bool* done, dim3 grid, int threads, int smem,
                     cudaStream_t st, A... args) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (smem > 48 * 1024 && (dev < 0 || dev >= 64 || !done[dev])) {
    const cudaError_t e = cudaFuncSetAttribute((const void*)kern,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, GN_MAX_SMEM);
    if (e != cudaSuccess) return (int)e;
    if (dev >= 0 && dev < 64) done[dev] = true;
  }
  after(kern, grid, threads, smem, st)(args...);
  return (int)cudaGetLastError();
}

PF_API int pf_groupnorm_fwd(const void* x, const void* gamma, const void* beta, void* y,
                            void* mean, void* rstd, void* scratch, int B, int HW, int C, int G,
                            float eps, int act_silu, int dtype, int sm_count, void* stream) {
  if (C % G || C % 8 || !on_vectors(x, y)) return -2;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int rows = gn_rows(C);
  const int threads = rows * (C / 8);
  if (threads > 1024) return -2;
  const int slabs = gn_slabs(B, HW, rows, sm_count, GN_FWD_PER_SM);
  const dim3 grid(slabs, B);
  PF_DISPATCH_H(dtype, {
    static bool done[64] = {};
    const int r = gn_launch(gn_stats_kernel<T>, done, grid, threads, gn_smem(rows, C), st,
                            (const T*)x, (float*)scratch, HW, C, G, rows);
    if (r) return r;
    after(gn_finalize_kernel, (B * G + 3) / 4, 128, 0, st)(
        (const float*)scratch, (float*)mean, (float*)rstd, slabs, G, B * G,
        1.f / ((float)HW * (C / G)), eps);
    const int smem = 0;
    PF_GN_SILU(gn_apply_kernel, (const T*)x, (const float*)mean, (const float*)rstd,
               (const float*)gamma, (const float*)beta, (T*)y, HW, C, G, rows);
  });
  PF_CHECK_LAUNCH();
  return 0;
}

template <typename F>
static int gn_bwd_launch(int act_silu, int threads, F f) {
  auto sized = [&](auto silu) {
    if (threads <= 256) return f(silu, std::integral_constant<int, 256>());
    if (threads <= GN_RING_THREADS) return f(silu, std::integral_constant<int, GN_RING_THREADS>());
    if (threads <= 800) return f(silu, std::integral_constant<int, 800>());
    return f(silu, std::integral_constant<int, 1024>());
  };
  return act_silu ? sized(std::true_type()) : sized(std::false_type());
}

// sums: fp32 scratch [2][B*G]; dgamma / dbeta fp32 [C]
PF_API int pf_groupnorm_bwd(const void* dy, const void* x, const void* mean, const void* rstd,
                            const void* gamma, const void* beta, void* dx, void* dgamma,
                            void* dbeta, void* sums, void* scratch, int B, int HW, int C, int G,
                            int act_silu, int dtype, int sm_count, void* stream) {
  if (C % G || C % 8 || !on_vectors(dy, x, dx)) return -2;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  float* sA = (float*)sums;
  float* sB = sA + (long long)B * G;
  const int rows = gn_rows(C);
  const int threads = rows * (C / 8);
  if (threads > 1024) return -2;
  const int slabs = gn_slabs(B, HW, rows, sm_count, GN_BWD_PER_SM);
  const dim3 grid(slabs, B);
  float* part = (float*)scratch;
  float* gpart = part + (long long)B * slabs * 2 * C;
  PF_DISPATCH_H(dtype, {
    int r = gn_bwd_launch(act_silu, threads, [&](auto silu, auto most) {
      constexpr bool S = decltype(silu)::value;
      constexpr int R = decltype(most)::value;
      static bool done[64] = {};       // one per instantiation
      return gn_launch(gn_bwd_stats_kernel<T, S, R>, done, grid, threads,
                       gn_smem(rows, C) + gn_ring_smem(threads), st, (const T*)dy, (const T*)x,
                       (const float*)mean, (const float*)rstd, (const float*)gamma,
                       (const float*)beta, part, gpart, HW, C, G, rows);
    });
    if (r) return r;
    after(gn_bwd_fold_kernel, (B * G + 31) / 32 + (C + 31) / 32, 1024, 0, st)(
        part, gpart, sA, sB, (float*)dgamma, (float*)dbeta, B, slabs, C, G);
    r = gn_bwd_launch(act_silu, threads, [&](auto silu, auto most) {
      constexpr bool S = decltype(silu)::value;
      constexpr int R = decltype(most)::value;
      static bool done[64] = {};       // one per instantiation
      return gn_launch(gn_bwd_apply_kernel<T, S, R>, done, grid, threads, gn_ring_smem(threads), st,
                       (const T*)dy, (const T*)x, (const float*)mean, (const float*)rstd,
                       (const float*)gamma, (const float*)beta, sA, sB, (T*)dx, HW, C, G, rows);
    });
    if (r) return r;
  });
  PF_CHECK_LAUNCH();
  return 0;
}

// Channels per tile: equal shares, multiples of 8, of no more than `most`.
static inline int conv_share(int channels, int most) {
  const int tiles = (channels + most - 1) / most;
  return ((channels + tiles - 1) / tiles + 7) / 8 * 8;
}

// 16-bit weights [Cout, Cin, taps] -> [cout8, taps, cin8], or with `flip` [cin8, taps reversed,
// cout8]; cout8 / cin8 are multiples of 8, `out` lies on 16 bytes
PF_API int pf_conv_pack(const void* w, void* out, int Cout, int Cin, int taps, int cout8, int cin8,
                        int flip, void* stream) {
  if (taps < 1 || taps > CONV_PACK_TAPS || cout8 % 8 || cin8 % 8) return -3;
  if (!on_vectors(out)) return -2;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int vec = (reinterpret_cast<uintptr_t>(w) & 15) == 0 && (long long)Cin * taps % 8 == 0;
  if (!flip) {
    const int per = conv_share(cin8, CONV_TILE / taps / 8 * 8);
    after(conv_pack_kernel, dim3(cout8, (cin8 + per - 1) / per), 128, 0, st)(
        (const uint16_t*)w, (uint16_t*)out, Cout, Cin, taps, cin8, per, vec);
  } else {
    // tiles of 5 to 8 thousand elements; 64 channels make whole 128-byte lines of the output
    const int per = taps <= 9 ? 64 : taps <= 25 ? 32 : 16;
    after(conv_pack_flip_kernel, dim3(cin8 / 8, (cout8 + per - 1) / per), 256,
                            per * (8 * taps + 2) * 2, st)((const uint16_t*)w, (uint16_t*)out,
                                                            Cout, Cin, taps, cout8, per, vec);
  }
  PF_CHECK_LAUNCH();
  return 0;
}

// fp32 [>= Cout, taps, cin8] on 16 bytes -> [Cout, Cin, taps] of `dtype`; cin8 is a multiple of 8
PF_API int pf_conv_unpack(const void* src, void* dw, int Cout, int Cin, int taps, int cin8,
                          int dtype, void* stream) {
  if (taps < 1 || taps > CONV_PACK_TAPS || cin8 % 8) return -3;
  if (!on_vectors(src)) return -2;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int per = conv_share(cin8, CONV_TILE / (taps | 1) / 8 * 8);
  const dim3 grid(Cout, (Cin + per - 1) / per);
  const int vec = (reinterpret_cast<uintptr_t>(dw) & 15) == 0 &&
                  (long long)Cin * taps % (dtype == PF_F32 ? 4 : 8) == 0;
  const float* s = (const float*)src;
  switch (dtype) {
    case PF_F32: after(conv_unpack_kernel<float>, grid, 128, 0, st)(s, (float*)dw, Cin, taps, cin8, per, vec); break;
    case PF_F16: after(conv_unpack_kernel<__half>, grid, 128, 0, st)(s, (__half*)dw, Cin, taps, cin8, per, vec); break;
    case PF_BF16: after(conv_unpack_kernel<__nv_bfloat16>, grid, 128, 0, st)(s, (__nv_bfloat16*)dw, Cin, taps, cin8, per, vec); break;
    default: return -1;
  }
  PF_CHECK_LAUNCH();
  return 0;
}

PF_API int pf_upsample2x(const void* x, void* y, int B, int H, int W, int C, int backward,
                         int dtype, int sm_count, void* stream) {
  if (C % 8 || !on_vectors(x, y)) return -2;
  const long long total = (long long)B * H * W * (C / 8) * (backward ? 1 : 4);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  PF_DISPATCH_H(dtype, (after(upsample2x_kernel<T>, grid_for(total, sm_count), 256, 0, st)(
      (const T*)x, (T*)y, B, H, W, C, backward)));
  PF_CHECK_LAUNCH();
  return 0;
}
