// LayerNorm and RMSNorm, forward and backward, one CTA per row with the row held in registers
// (16-byte loads, two block reductions).  The forward can fuse the residual add of a
// pre-norm transformer block:  h = x + res ;  y = norm(h) * gamma (+ beta).
// The backward writes dx (optionally + the gradient that flows around the norm through the
// residual branch) and per-CTA partial sums of dgamma / dbeta into a scratch buffer that a
// second small kernel folds into the fp32 parameter gradients.
#include "no_alloc.h"
#include "common.cuh"
#include "api.h"

namespace pf {

constexpr int NORM_MAX_VEC = 4;   // 16-byte vectors per thread: N <= 256 * 4 * 8 = 8192 (16-bit)

template <int THREADS>
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (l < THREADS / 32) ? red[l] : 0.f;
  t = warp_sum(t);
  return t;
}

// rms != 0 -> RMSNorm (no mean subtraction, no beta)
template <typename T, int THREADS>
__global__ void __launch_bounds__(THREADS)
norm_fwd_kernel(const T* __restrict__ x, const T* __restrict__ res, const float* __restrict__ gamma,
                const float* __restrict__ beta, T* __restrict__ y, T* __restrict__ h_out,
                float* __restrict__ mean_out, float* __restrict__ rstd_out, int N, float eps,
                int rms) {
  after_previous();
  constexpr int V = 16 / sizeof(T);
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const int nvec = N / V;
  const T* xr = x + row * N;
  float vals[NORM_MAX_VEC][V];
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < NORM_MAX_VEC; ++i) {
    const int idx = threadIdx.x + i * THREADS;
    if (idx < nvec) {
      uint4 q = reinterpret_cast<const uint4*>(xr)[idx];
      const T* e = reinterpret_cast<const T*>(&q);
      if (res) {
        uint4 qr = reinterpret_cast<const uint4*>(res + row * N)[idx];
        const T* er = reinterpret_cast<const T*>(&qr);
        uint4 qh;
        T* eh = reinterpret_cast<T*>(&qh);
#pragma unroll
        for (int j = 0; j < V; ++j) {
          // round the residual stream to its storage type first so fwd and bwd agree
          eh[j] = from_f32<T>(to_f32<T>(e[j]) + to_f32<T>(er[j]));
          vals[i][j] = to_f32<T>(eh[j]);
        }
        if (h_out) reinterpret_cast<uint4*>(h_out + row * N)[idx] = qh;
      } else {
#pragma unroll
        for (int j = 0; j < V; ++j) vals[i][j] = to_f32<T>(e[j]);
      }
#pragma unroll
      for (int j = 0; j < V; ++j) s += vals[i][j];
    }
  }
  float mean = 0.f;
  if (!rms) mean = block_sum<THREADS>(s, red) / N;
  float sq = 0.f;
#pragma unroll
  for (int i = 0; i < NORM_MAX_VEC; ++i) {
    const int idx = threadIdx.x + i * THREADS;
    if (idx < nvec) {
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const float d = vals[i][j] - mean;
        sq += d * d;
      }
    }
  }
  const float var = block_sum<THREADS>(sq, red) / N;
  const float rstd = rsqrtf(var + eps);
  if (threadIdx.x == 0) {
    if (mean_out) mean_out[row] = mean;
    rstd_out[row] = rstd;
  }
#pragma unroll
  for (int i = 0; i < NORM_MAX_VEC; ++i) {
    const int idx = threadIdx.x + i * THREADS;
    if (idx < nvec) {
      uint4 q;
      T* e = reinterpret_cast<T*>(&q);
      const float4* g4 = reinterpret_cast<const float4*>(gamma + idx * V);
      float g[V], b[V];
#pragma unroll
      for (int j = 0; j < V / 4; ++j) {
        float4 t = __ldg(g4 + j);
        g[4 * j] = t.x; g[4 * j + 1] = t.y; g[4 * j + 2] = t.z; g[4 * j + 3] = t.w;
      }
      if (beta) {
        const float4* b4 = reinterpret_cast<const float4*>(beta + idx * V);
#pragma unroll
        for (int j = 0; j < V / 4; ++j) {
          float4 t = __ldg(b4 + j);
          b[4 * j] = t.x; b[4 * j + 1] = t.y; b[4 * j + 2] = t.z; b[4 * j + 3] = t.w;
        }
      }
#pragma unroll
      for (int j = 0; j < V; ++j) {
        float o = (vals[i][j] - mean) * rstd * g[j];
        if (beta) o += b[j];
        e[j] = from_f32<T>(o);
      }
      reinterpret_cast<uint4*>(y + row * N)[idx] = q;
    }
  }
}

// Backward.  Grid = G persistent CTAs striding over rows; each thread keeps dgamma/dbeta
// partials for its own columns and writes them to scratch[blockIdx][2][N] at the end.
template <typename T, int THREADS>
__global__ void __launch_bounds__(THREADS)
norm_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ h, const float* __restrict__ gamma,
                const float* __restrict__ mean, const float* __restrict__ rstd,
                const T* __restrict__ dres, T* __restrict__ dx, float* __restrict__ scratch,
                long long rows, int N, int rms) {
  after_previous();
  constexpr int V = 16 / sizeof(T);
  __shared__ float red[32];
  const int nvec = N / V;
  float dg[NORM_MAX_VEC][V], db[NORM_MAX_VEC][V], g[NORM_MAX_VEC][V];
#pragma unroll
  for (int i = 0; i < NORM_MAX_VEC; ++i) {
    const int idx = threadIdx.x + i * THREADS;
#pragma unroll
    for (int j = 0; j < V; ++j) {
      dg[i][j] = 0.f; db[i][j] = 0.f;
      g[i][j] = (idx < nvec) ? gamma[idx * V + j] : 0.f;
    }
  }
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const float mu = rms ? 0.f : mean[row];
    const float rs = rstd[row];
    float xh[NORM_MAX_VEC][V], dyv[NORM_MAX_VEC][V];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < NORM_MAX_VEC; ++i) {
      const int idx = threadIdx.x + i * THREADS;
      if (idx < nvec) {
        uint4 qd = reinterpret_cast<const uint4*>(dy + row * N)[idx];
        uint4 qh = reinterpret_cast<const uint4*>(h + row * N)[idx];
        const T* ed = reinterpret_cast<const T*>(&qd);
        const T* eh = reinterpret_cast<const T*>(&qh);
#pragma unroll
        for (int j = 0; j < V; ++j) {
          const float d = to_f32<T>(ed[j]);
          const float xhat = (to_f32<T>(eh[j]) - mu) * rs;
          xh[i][j] = xhat;
          dyv[i][j] = d * g[i][j];
          dg[i][j] += d * xhat;
          db[i][j] += d;
          s1 += dyv[i][j];
          s2 += dyv[i][j] * xhat;
        }
      }
    }
    float m1 = 0.f;
    if (!rms) m1 = block_sum<THREADS>(s1, red) / N;
    const float m2 = block_sum<THREADS>(s2, red) / N;
#pragma unroll
    for (int i = 0; i < NORM_MAX_VEC; ++i) {
      const int idx = threadIdx.x + i * THREADS;
      if (idx < nvec) {
        uint4 q;
        T* e = reinterpret_cast<T*>(&q);
        uint4 qr;
        const T* er = reinterpret_cast<const T*>(&qr);
        if (dres) qr = reinterpret_cast<const uint4*>(dres + row * N)[idx];
#pragma unroll
        for (int j = 0; j < V; ++j) {
          float o = rs * (dyv[i][j] - m1 - xh[i][j] * m2);
          if (dres) o += to_f32<T>(er[j]);
          e[j] = from_f32<T>(o);
        }
        reinterpret_cast<uint4*>(dx + row * N)[idx] = q;
      }
    }
  }
  float* sg = scratch + (long long)blockIdx.x * 2 * N;
  float* sb = sg + N;
#pragma unroll
  for (int i = 0; i < NORM_MAX_VEC; ++i) {
    const int idx = threadIdx.x + i * THREADS;
    if (idx < nvec) {
#pragma unroll
      for (int j = 0; j < V; ++j) {
        sg[idx * V + j] = dg[i][j];
        sb[idx * V + j] = db[i][j];
      }
    }
  }
}

// Forward for rows of up to 2048 16-bit elements: one warp per row, shuffle reductions only (no
// CTA barrier), 8 rows per CTA.  The row stays in registers in its packed 16-bit form and is
// expanded once per pass (sum, squared deviations, output): a third of the registers of an fp32
// copy.  Bound by HBM: x and the residual are requested together, without a register limit that
// would spill them; bf16 with residual 6168 x 1408 29 -> 23 us, 50000 x 1408 129 -> 102 us
// (5.5 TB/s), 20000 x 2048 98 -> 75 us.  Rows of one or two vectors a lane without a residual are
// bound by the instructions around their loads and have a form of their own (MAY_RES false):
// 200000 x 64 47.5 -> 43.7 us.
template <typename T, int NV, bool MAY_RES>
__global__ void __launch_bounds__(256, MAY_RES ? 0 : 4)
norm_fwd_warp_kernel(const T* __restrict__ x, const T* __restrict__ res,
                     const float* __restrict__ gamma, const float* __restrict__ beta,
                     T* __restrict__ y, T* __restrict__ h_out, float* __restrict__ mean_out,
                     float* __restrict__ rstd_out, long long rows, int N, float eps, int rms) {
  after_previous();
  constexpr int V = 8;
  const int nvec = N / V;
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= rows) return;
  uint4 q[NV], qr[MAY_RES ? NV : 1];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int idx = lane + i * 32;
    if (idx < nvec) q[i] = reinterpret_cast<const uint4*>(x + row * N)[idx];
  }
  if (MAY_RES && res) {   // h = x + residual, rounded to the storage type like the unfused sequence
    // both streams are requested before either is used
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int idx = lane + i * 32;
      if (idx < nvec) qr[MAY_RES ? i : 0] = reinterpret_cast<const uint4*>(res + row * N)[idx];
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int idx = lane + i * 32;
      if (idx < nvec) {
        const T* er = reinterpret_cast<const T*>(&qr[MAY_RES ? i : 0]);
        T* e = reinterpret_cast<T*>(&q[i]);
#pragma unroll
        for (int j = 0; j < V; ++j) e[j] = from_f32<T>(to_f32<T>(e[j]) + to_f32<T>(er[j]));
        if (h_out) reinterpret_cast<uint4*>(h_out + row * N)[idx] = q[i];
      }
    }
  }
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (lane + i * 32 < nvec) {
      const T* e = reinterpret_cast<const T*>(&q[i]);
#pragma unroll
      for (int j = 0; j < V; ++j) s += to_f32<T>(e[j]);
    }
  }
  const float mean = rms ? 0.f : warp_sum(s) / N;
  float sq = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (lane + i * 32 < nvec) {
      const T* e = reinterpret_cast<const T*>(&q[i]);
#pragma unroll
      for (int j = 0; j < V; ++j) { const float d = to_f32<T>(e[j]) - mean; sq = fmaf(d, d, sq); }
    }
  }
  const float rstd = rsqrtf(warp_sum(sq) / N + eps);
  if (lane == 0) {
    if (mean_out) mean_out[row] = mean;
    rstd_out[row] = rstd;
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int idx = lane + i * 32;
    if (idx < nvec) {
      const float4 g0 = __ldg(reinterpret_cast<const float4*>(gamma + idx * V));
      const float4 g1 = __ldg(reinterpret_cast<const float4*>(gamma + idx * V) + 1);
      const float g[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
      float b[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (beta) {
        const float4 b0 = __ldg(reinterpret_cast<const float4*>(beta + idx * V));
        const float4 b1 = __ldg(reinterpret_cast<const float4*>(beta + idx * V) + 1);
        b[0] = b0.x; b[1] = b0.y; b[2] = b0.z; b[3] = b0.w;
        b[4] = b1.x; b[5] = b1.y; b[6] = b1.z; b[7] = b1.w;
      }
      const T* ei = reinterpret_cast<const T*>(&q[i]);
      uint4 o;
      T* e = reinterpret_cast<T*>(&o);
#pragma unroll
      for (int j = 0; j < V; ++j)
        e[j] = from_f32<T>((to_f32<T>(ei[j]) - mean) * rstd * g[j] + b[j]);
      reinterpret_cast<uint4*>(y + row * N)[idx] = o;
    }
  }
}

// Backward for rows of up to 2048 16-bit elements, everything in one pass over memory.  A
// persistent CTA walks over tiles of 8 rows that asynchronous copies bring into shared memory, one
// tile ahead; dy and h are then read there twice:
//   by rows      warp <-> row: two shuffle reductions, dx
//   by columns   thread <-> 8 columns of a share of the 8 rows: sums of dy * xhat and dy, kept in
//                registers over all tiles of the CTA
// The CTA's sums go to scratch[blockIdx][2][N], folded by norm_bwd_finish_kernel.
// Bound by HBM: 4 tensors cross it once, where a pass for dx and one for the sums read dy and h
// twice.  bf16, with the fold: 6168 x 1408 50 -> 38 us, 50000 x 1408 249 -> 153 us (3.7 TB/s),
// 20000 x 2048 173 -> 112 us.  Longer rows: norm_bwd_wide_kernel.
constexpr int NORM_TILE_ROWS = 8;
template <typename T, int NV>
__global__ void __launch_bounds__(256)
norm_bwd_fused_kernel(const T* __restrict__ dy, const T* __restrict__ h,
                      const float* __restrict__ gamma, const float* __restrict__ mean,
                      const float* __restrict__ rstd, const T* __restrict__ dres,
                      T* __restrict__ dx, float* __restrict__ scratch, long long rows, int N,
                      int rms) {
  after_previous();
  constexpr int V = 8, R = NORM_TILE_ROWS;
  extern __shared__ __align__(128) uint8_t nsmem[];     // [2 stages][dy, h][R][N]
  const int nvec = N / V, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tile_vec = R * nvec;
  auto stage_ptr = [&](int st, int which) {
    return reinterpret_cast<uint4*>(nsmem) + (st * 2 + which) * tile_vec;
  };
  const long long n_tiles = (rows + R - 1) / R;
  // the rows of a tile are one contiguous piece of each tensor
  auto fetch = [&](long long t, int st) {
    if (t < n_tiles) {
      const int n = (int)min((long long)R, rows - t * R) * nvec;
      const uint4* gd = reinterpret_cast<const uint4*>(dy + t * R * N);
      const uint4* gh = reinterpret_cast<const uint4*>(h + t * R * N);
      for (int i = threadIdx.x; i < n; i += 256) {
        cp_async16(stage_ptr(st, 0) + i, gd + i);
        cp_async16(stage_ptr(st, 1) + i, gh + i);
      }
    }
    cp_async_commit();                 // an empty group past the last tile
  };
  fetch(blockIdx.x, 0);
  // column share: vector cv of rows grp, grp + groups, ...
  const int groups = min(R, 256 / nvec), grp = threadIdx.x / nvec, cv = threadIdx.x - grp * nvec;
  float ag[V] = {0, 0, 0, 0, 0, 0, 0, 0}, ab[V] = {0, 0, 0, 0, 0, 0, 0, 0};
  const float inv_n = 1.f / N;
  int st = 0;
  for (long long t = blockIdx.x; t < n_tiles; t += gridDim.x, st ^= 1) {
    // the other stage was read in the previous round, which ended with a barrier
    fetch(t + gridDim.x, st ^ 1);
    const int live = (int)min((long long)R, rows - t * R);
    const long long row = t * R + warp;
    uint4 qr[NV];
    float mu = 0.f, rs = 0.f;
    if (warp < live) {
      if (!rms) mu = mean[row];
      rs = rstd[row];
      if (dres) {
#pragma unroll
        for (int i = 0; i < NV; ++i)
          if (lane + i * 32 < nvec)
            qr[i] = __ldg(reinterpret_cast<const uint4*>(dres + row * N) + lane + i * 32);
      }
    }
    cp_async_wait<1>();           // this tile has landed, the next one may be under way
    __syncthreads();
    const uint4 *sd = stage_ptr(st, 0), *sh = stage_ptr(st, 1);
    if (warp < live) {
      const uint4 *rd = sd + warp * nvec, *rh = sh + warp * nvec;
      float s1 = 0.f, s2 = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int idx = lane + i * 32;
        if (idx < nvec) {
          const uint4 qd = rd[idx], qh = rh[idx];
          const T* ed = reinterpret_cast<const T*>(&qd);
          const T* eh = reinterpret_cast<const T*>(&qh);
          const float4 g0 = __ldg(reinterpret_cast<const float4*>(gamma + idx * V));
          const float4 g1 = __ldg(reinterpret_cast<const float4*>(gamma + idx * V) + 1);
          const float g[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
          for (int j = 0; j < V; ++j) {
            const float dyg = to_f32<T>(ed[j]) * g[j];
            s1 += dyg;
            s2 += dyg * (to_f32<T>(eh[j]) - mu) * rs;
          }
        }
      }
      const float m1 = rms ? 0.f : warp_sum(s1) * inv_n;
      const float m2 = warp_sum(s2) * inv_n;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int idx = lane + i * 32;
        if (idx < nvec) {
          const uint4 qd = rd[idx], qh = rh[idx];
          const T* ed = reinterpret_cast<const T*>(&qd);
          const T* eh = reinterpret_cast<const T*>(&qh);
          const float4 g0 = __ldg(reinterpret_cast<const float4*>(gamma + idx * V));
          const float4 g1 = __ldg(reinterpret_cast<const float4*>(gamma + idx * V) + 1);
          const float g[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
          const T* er = reinterpret_cast<const T*>(&qr[i]);
          uint4 q;
          T* e = reinterpret_cast<T*>(&q);
#pragma unroll
          for (int j = 0; j < V; ++j) {
            const float xhat = (to_f32<T>(eh[j]) - mu) * rs;
            float o = rs * (to_f32<T>(ed[j]) * g[j] - m1 - xhat * m2);
            if (dres) o += to_f32<T>(er[j]);
            e[j] = from_f32<T>(o);
          }
          reinterpret_cast<uint4*>(dx + row * N)[idx] = q;
        }
      }
    }
    if (grp < groups) {
      for (int r = grp; r < live; r += groups) {
        const float mr = rms ? 0.f : __ldg(mean + t * R + r), rr = __ldg(rstd + t * R + r);
        const uint4 qd = sd[r * nvec + cv], qh = sh[r * nvec + cv];
        const T* ed = reinterpret_cast<const T*>(&qd);
        const T* eh = reinterpret_cast<const T*>(&qh);
#pragma unroll
        for (int j = 0; j < V; ++j) {
          const float d = to_f32<T>(ed[j]);
          ag[j] += d * (to_f32<T>(eh[j]) - mr) * rr;
          ab[j] += d;
        }
      }
    }
    __syncthreads();
  }
  // fold the row groups through the (now unused) tiles: [groups][2][N] floats
  float* red = reinterpret_cast<float*>(nsmem);
  if (grp < groups) {
#pragma unroll
    for (int j = 0; j < V; ++j) {
      red[grp * 2 * N + cv * V + j] = ag[j];
      red[grp * 2 * N + N + cv * V + j] = ab[j];
    }
  }
  __syncthreads();
  float* out = scratch + (long long)blockIdx.x * 2 * N;
  for (int i = threadIdx.x; i < 2 * N; i += 256) {
    float v = red[i];
    for (int k = 1; k < groups; ++k) v += red[k * 2 * N + i];
    out[i] = v;
  }
}

// Backward for rows of 2056 to 4096 16-bit elements, in one pass as well: two stages of eight such
// rows do not fit in shared memory, so a thread owns 8 columns for good and keeps their parameter sums
// in registers, and a row's two sums go through the CTA (one barrier per NORM_WIDE_ROWS rows).  A
// thread only ever reads what it copied itself, so the ring that its asynchronous copies fill three
// batches ahead (144 KB on their way per SM at 4096 columns) needs no barriers.  One CTA per SM.
// Bound by HBM: 4 tensors cross it once.  bf16, with the fold, against a pass for dx (one warp per row,
// 16 vectors of two tensors in registers) and one for the sums: 2048 x 4096 62 -> 28 us,
// 20000 x 4096 441 -> 132, 50000 x 4096 1066 -> 308 (5.3 TB/s), 9000 x 3072 120 -> 60.
constexpr int NORM_WIDE_ROWS = 2, NORM_WIDE_STAGES = 4;
template <typename T, int THREADS>
__global__ void __launch_bounds__(THREADS, 1)
norm_bwd_wide_kernel(const T* __restrict__ dy, const T* __restrict__ h,
                     const float* __restrict__ gamma, const float* __restrict__ mean,
                     const float* __restrict__ rstd, const T* __restrict__ dres,
                     T* __restrict__ dx, float* __restrict__ scratch, long long rows, int N,
                     int rms) {
  after_previous();
  constexpr int V = 8, R = NORM_WIDE_ROWS, S = NORM_WIDE_STAGES, WARPS = THREADS / 32;
  static_assert(WARPS <= 32 && R == 2, "one lane per warp folds the sums of two rows");
  __shared__ float4 red[2][WARPS];             // per warp: s1, s2 of both rows; two batches
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cv = threadIdx.x;
  const bool on = cv < N / V;
  float g[V], ag[V], ab[V];
#pragma unroll
  for (int j = 0; j < V; ++j) {
    g[j] = on ? __ldg(gamma + cv * V + j) : 0.f;
    ag[j] = ab[j] = 0.f;
  }
  const float inv_n = 1.f / N;
  const long long n_batches = (rows + R - 1) / R;
  extern __shared__ __align__(128) uint8_t wsmem[];     // [stage][row][dy, h, dres][thread]
  auto slot = [&](int st, int r, int which) {
    return reinterpret_cast<uint4*>(wsmem) + ((st * R + r) * 3 + which) * THREADS + cv;
  };
  auto fetch = [&](long long b, int st) {
    if (on && b < n_batches) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const long long row = b * R + r;
        if (row < rows) {
          cp_async16(slot(st, r, 0), reinterpret_cast<const uint4*>(dy + row * N) + cv);
          cp_async16(slot(st, r, 1), reinterpret_cast<const uint4*>(h + row * N) + cv);
          if (dres) cp_async16(slot(st, r, 2), reinterpret_cast<const uint4*>(dres + row * N) + cv);
        }
      }
    }
    cp_async_commit();                 // an empty group past the last batch
  };
  const long long step = gridDim.x;
  long long b = blockIdx.x;
#pragma unroll
  for (int i = 0; i < S - 1; ++i) fetch(b + i * step, i);
  int st = 0;
  for (int parity = 0; b < n_batches; b += step, parity ^= 1) {
    uint4 qd[R], qh[R], qr[R];
    float mu[R], rs[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const long long row = min(b * R + r, rows - 1);
      mu[r] = rms ? 0.f : __ldg(mean + row);
      rs[r] = __ldg(rstd + row);
      qd[r] = qh[r] = qr[r] = make_uint4(0, 0, 0, 0);
    }
    cp_async_wait<S - 2>();            // this batch has landed, the later ones may be under way
    if (on) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (b * R + r < rows) {
          qd[r] = *slot(st, r, 0);
          qh[r] = *slot(st, r, 1);
          if (dres) qr[r] = *slot(st, r, 2);
        }
    }
    // into the slots read in the previous round
    fetch(b + (S - 1) * step, st == 0 ? S - 1 : st - 1);
    st = st == S - 1 ? 0 : st + 1;
    float s[2 * R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const T* ed = reinterpret_cast<const T*>(&qd[r]);
      const T* eh = reinterpret_cast<const T*>(&qh[r]);
      float s1 = 0.f, s2 = 0.f;
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const float d = to_f32<T>(ed[j]), xhat = (to_f32<T>(eh[j]) - mu[r]) * rs[r];
        const float dyg = d * g[j];
        s1 += dyg;
        s2 += dyg * xhat;
        ag[j] += d * xhat;
        ab[j] += d;
      }
      s[2 * r] = on ? s1 : 0.f;
      s[2 * r + 1] = on ? s2 : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 2 * R; ++i) s[i] = warp_sum(s[i]);
    if (lane == 0) red[parity][warp] = make_float4(s[0], s[1], s[2], s[3]);
    // the buffer of two batches ago is free: every warp has passed the barrier since it read it
    __syncthreads();
    float4 f = lane < WARPS ? red[parity][lane] : make_float4(0.f, 0.f, 0.f, 0.f);
    f.x = warp_sum(f.x); f.y = warp_sum(f.y); f.z = warp_sum(f.z); f.w = warp_sum(f.w);
    const float m1[R] = {rms ? 0.f : f.x * inv_n, rms ? 0.f : f.z * inv_n};
    const float m2[R] = {f.y * inv_n, f.w * inv_n};
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const long long row = b * R + r;
      if (on && row < rows) {
        const T* ed = reinterpret_cast<const T*>(&qd[r]);
        const T* eh = reinterpret_cast<const T*>(&qh[r]);
        const T* er = reinterpret_cast<const T*>(&qr[r]);
        uint4 q;
        T* e = reinterpret_cast<T*>(&q);
#pragma unroll
        for (int j = 0; j < V; ++j) {
          const float xhat = (to_f32<T>(eh[j]) - mu[r]) * rs[r];
          float o = rs[r] * (to_f32<T>(ed[j]) * g[j] - m1[r] - xhat * m2[r]);
          if (dres) o += to_f32<T>(er[j]);
          e[j] = from_f32<T>(o);
        }
        reinterpret_cast<uint4*>(dx + row * N)[cv] = q;
      }
    }
  }
  if (on) {
    float4* og = reinterpret_cast<float4*>(scratch + (long long)blockIdx.x * 2 * N + cv * V);
    float4* ob = reinterpret_cast<float4*>(scratch + (long long)blockIdx.x * 2 * N + N + cv * V);
    og[0] = make_float4(ag[0], ag[1], ag[2], ag[3]);
    og[1] = make_float4(ag[4], ag[5], ag[6], ag[7]);
    ob[0] = make_float4(ab[0], ab[1], ab[2], ab[3]);
    ob[1] = make_float4(ab[4], ab[5], ab[6], ab[7]);
  }
}

// dgamma[c] (+)= sum_g scratch[g][0][c] ; dbeta likewise.  A CTA owns 32 columns, its 32 warps share
// the G rows (one thread per column over all rows took 29 us of latency at G = 296).
__global__ void __launch_bounds__(1024)
norm_bwd_finish_kernel(const float* __restrict__ scratch, float* __restrict__ dgamma,
                       float* __restrict__ dbeta, int G, int N, int accumulate) {
  after_previous();
  __shared__ float red[2][32][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  float a = 0.f, b = 0.f;
  if (c < N) {
#pragma unroll 4
    for (int g = warp; g < G; g += 32) {
      a += scratch[(long long)g * 2 * N + c];
      b += scratch[(long long)g * 2 * N + N + c];
    }
  }
  red[0][lane][warp] = a;
  red[1][lane][warp] = b;
  __syncthreads();
  // warp w finishes column w of the 32
  const int cw = blockIdx.x * 32 + warp;
  a = warp_sum(red[0][warp][lane]);
  b = warp_sum(red[1][warp][lane]);
  if (lane == 0 && cw < N) {
    // a gradient bucket may be added to by other kernels at the same time
    if (accumulate) atomicAdd(dgamma + cw, a);
    else dgamma[cw] = a;
    if (dbeta && accumulate) atomicAdd(dbeta + cw, b);
    else if (dbeta) dbeta[cw] = b;
  }
}

// the fused backward needs two stages of a tile in shared memory (at most 128 KB)
template <typename T, int NV>
static int norm_bwd_fused_launch(const void* dy, const void* h, const float* gamma,
                                 const float* mean, const float* rstd, const void* dres, void* dx,
                                 float* scratch, int G, long long rows, int N, int rms,
                                 cudaStream_t st) {
  auto kern = norm_bwd_fused_kernel<T, NV>;
  const int bytes = max(4 * NORM_TILE_ROWS * N * 2, 16384);
  static bool done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         4 * NORM_TILE_ROWS * 2048 * 2);
    if (e != cudaSuccess) return (int)e;
    if (dev >= 0 && dev < 64) done[dev] = true;
  }
  after(kern, G, 256, bytes, st)((const T*)dy, (const T*)h, gamma, mean, rstd, (const T*)dres,
                              (T*)dx, scratch, rows, N, rms);
  return 0;
}

template <typename T, int THREADS>
static int norm_bwd_wide_launch(const void* dy, const void* h, const float* gamma,
                                const float* mean, const float* rstd, const void* dres, void* dx,
                                float* scratch, int G, long long rows, int N, int rms,
                                cudaStream_t st) {
  auto kern = norm_bwd_wide_kernel<T, THREADS>;
  constexpr int bytes = NORM_WIDE_STAGES * NORM_WIDE_ROWS * 3 * THREADS * 16;
  static bool done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return (int)e;
    if (dev >= 0 && dev < 64) done[dev] = true;
  }
  after(kern, G, THREADS, bytes, st)((const T*)dy, (const T*)h, gamma, mean, rstd, (const T*)dres,
                                  (T*)dx, scratch, rows, N, rms);
  return 0;
}

template <typename T>
static int norm_fwd_launch(const void* x, const void* res, const float* gamma, const float* beta,
                           void* y, void* h_out, float* mean, float* rstd, long long rows, int N,
                           float eps, int rms, cudaStream_t st) {
  constexpr int V = 16 / sizeof(T);
  if (N % V) return -2;
  const int nvec = N / V;
  if constexpr (sizeof(T) == 2) if (nvec <= 32 * 8) {
    const unsigned grid = (unsigned)((rows + 7) / 8);
#define PF_NORM_FWD_WARP(NV, MAY_RES)                                                         \
    after(norm_fwd_warp_kernel<T, NV, MAY_RES>, grid, 256, 0, st)((const T*)x, (const T*)res, gamma, \
        beta, (T*)y, (T*)h_out, mean, rstd, rows, N, eps, rms)
    if (nvec <= 32 * 2 && !res) PF_NORM_FWD_WARP(2, false);
    else if (nvec <= 32 * 2) PF_NORM_FWD_WARP(2, true);
    else if (nvec <= 32 * 4) PF_NORM_FWD_WARP(4, true);
    else if (nvec <= 32 * 6) PF_NORM_FWD_WARP(6, true);
    else PF_NORM_FWD_WARP(8, true);
#undef PF_NORM_FWD_WARP
    return 0;
  }
  if (nvec <= 128 * NORM_MAX_VEC)
    after(norm_fwd_kernel<T, 128>, (unsigned)rows, 128, 0, st)((const T*)x, (const T*)res, gamma,
        beta, (T*)y, (T*)h_out, mean, rstd, N, eps, rms);
  else if (nvec <= 256 * NORM_MAX_VEC)
    after(norm_fwd_kernel<T, 256>, (unsigned)rows, 256, 0, st)((const T*)x, (const T*)res, gamma,
        beta, (T*)y, (T*)h_out, mean, rstd, N, eps, rms);
  else if (nvec <= 1024 * NORM_MAX_VEC)
    after(norm_fwd_kernel<T, 1024>, (unsigned)rows, 1024, 0, st)((const T*)x, (const T*)res, gamma,
        beta, (T*)y, (T*)h_out, mean, rstd, N, eps, rms);
  else
    return -3;
  return 0;
}

template <typename T>
static int norm_bwd_launch(const void* dy, const void* h, const float* gamma, const float* mean,
                           const float* rstd, const void* dres, void* dx, float* scratch, int& G,
                           long long rows, int N, int rms, int sm_count, cudaStream_t st) {
  constexpr int V = 16 / sizeof(T);
  if (N % V) return -2;
  const int nvec = N / V;
  if constexpr (sizeof(T) == 2) if (nvec <= 32 * 8) {
#define PF_NORM_BWD_FUSED(NV)                                                                     \
    norm_bwd_fused_launch<T, NV>(dy, h, gamma, mean, rstd, dres, dx, scratch, G, rows, N, rms, st)
    if (nvec <= 32 * 2) return PF_NORM_BWD_FUSED(2);
    if (nvec <= 32 * 4) return PF_NORM_BWD_FUSED(4);
    if (nvec <= 32 * 6) return PF_NORM_BWD_FUSED(6);
    return PF_NORM_BWD_FUSED(8);
#undef PF_NORM_BWD_FUSED
  }
  if constexpr (sizeof(T) == 2) if (nvec <= 32 * 16) {
    // rows of up to 4096 16-bit elements (Llama's hidden size): one CTA per SM fills its shared memory
    if (G > sm_count) G = sm_count;
#define PF_NORM_BWD_WIDE(THREADS)                                                                 \
    norm_bwd_wide_launch<T, THREADS>(dy, h, gamma, mean, rstd, dres, dx, scratch, G, rows, N, rms, st)
    return nvec <= 384 ? PF_NORM_BWD_WIDE(384) : PF_NORM_BWD_WIDE(512);
#undef PF_NORM_BWD_WIDE
  }
  if (nvec <= 128 * NORM_MAX_VEC)
    after(norm_bwd_kernel<T, 128>, G, 128, 0, st)((const T*)dy, (const T*)h, gamma, mean, rstd,
        (const T*)dres, (T*)dx, scratch, rows, N, rms);
  else if (nvec <= 256 * NORM_MAX_VEC)
    after(norm_bwd_kernel<T, 256>, G, 256, 0, st)((const T*)dy, (const T*)h, gamma, mean, rstd,
        (const T*)dres, (T*)dx, scratch, rows, N, rms);
  else if (nvec <= 1024 * NORM_MAX_VEC)
    after(norm_bwd_kernel<T, 1024>, G, 1024, 0, st)((const T*)dy, (const T*)h, gamma, mean, rstd,
        (const T*)dres, (T*)dx, scratch, rows, N, rms);
  else
    return -3;
  return 0;
}

}  // namespace pf

using namespace pf;

PF_API int pf_norm_fwd(const void* x, const void* res, const void* gamma, const void* beta,
                       void* y, void* h_out, void* mean, void* rstd, long long rows, int N,
                       float eps, int rms, int dtype, void* stream) {
  if (rows <= 0) return 0;
  if (!on_vectors(x, res, gamma, beta, y, h_out)) return -2;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  int r = -1;
  switch (dtype) {
    case PF_F32: r = norm_fwd_launch<float>(x, res, (const float*)gamma, (const float*)beta, y, h_out, (float*)mean, (float*)rstd, rows, N, eps, rms, st); break;
    case PF_F16: r = norm_fwd_launch<__half>(x, res, (const float*)gamma, (const float*)beta, y, h_out, (float*)mean, (float*)rstd, rows, N, eps, rms, st); break;
    case PF_BF16: r = norm_fwd_launch<__nv_bfloat16>(x, res, (const float*)gamma, (const float*)beta, y, h_out, (float*)mean, (float*)rstd, rows, N, eps, rms, st); break;
  }
  if (r) return r;
  PF_CHECK_LAUNCH();
  return 0;
}

// Number of CTAs (= rows of the scratch buffer) the backward uses for `rows` rows.
PF_API int pf_norm_bwd_ctas(long long rows, int sm_count) {
  long long g = (long long)(sm_count > 0 ? sm_count : 148) * 2;
  if (g > (rows + 7) / 8) g = (rows + 7) / 8;
  if (g < 1) g = 1;
  return (int)g;
}

// scratch: fp32 [pf_norm_bwd_ctas(rows)][2][N], contents on entry irrelevant.
PF_API int pf_norm_bwd(const void* dy, const void* h, const void* gamma, const void* mean,
                       const void* rstd, const void* dres, void* dx, void* dgamma, void* dbeta,
                       void* scratch, long long rows, int N, int rms, int accumulate, int dtype,
                       int sm_count, void* stream) {
  if (rows <= 0) return 0;
  if (!on_vectors(dy, h, gamma, dres, dx, scratch)) return -2;
  if (sm_count <= 0) sm_count = 148;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  int G = pf_norm_bwd_ctas(rows, sm_count);   // rows of scratch; the launch may use fewer
  int r = -1;
  switch (dtype) {
    case PF_F32: r = norm_bwd_launch<float>(dy, h, (const float*)gamma, (const float*)mean, (const float*)rstd, dres, dx, (float*)scratch, G, rows, N, rms, sm_count, st); break;
    case PF_F16: r = norm_bwd_launch<__half>(dy, h, (const float*)gamma, (const float*)mean, (const float*)rstd, dres, dx, (float*)scratch, G, rows, N, rms, sm_count, st); break;
    case PF_BF16: r = norm_bwd_launch<__nv_bfloat16>(dy, h, (const float*)gamma, (const float*)mean, (const float*)rstd, dres, dx, (float*)scratch, G, rows, N, rms, sm_count, st); break;
  }
  if (r) return r;
  PF_CHECK_LAUNCH();
  after(norm_bwd_finish_kernel, (N + 31) / 32, 1024, 0, st)((const float*)scratch, (float*)dgamma,
                                                         (float*)dbeta, G, N, accumulate);
  PF_CHECK_LAUNCH();
  return 0;
}

// ------------------------------------------------------------------ allocation-free variant

// Partial dgamma / dbeta sums of pf_norm_bwd_static.  One copy per device that loads the
// library; shared by every call on that device.
static __device__ __align__(256) float g_norm_static_scratch[PF_NORM_STATIC_SCRATCH_FLOATS];

// In host code `g_norm_static_scratch` is only a handle for the runtime's symbol table, not
// a device address; the address is queried once per device, with that device current.
static float* norm_static_scratch_ptr(int* err) {
  static float* ptrs[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) { *err = e != cudaSuccess ? (int)e : -3; return nullptr; }
  if (!ptrs[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_norm_static_scratch);
    if (e != cudaSuccess) { *err = (int)e; return nullptr; }
    ptrs[dev] = static_cast<float*>(p);
  }
  *err = 0;
  return ptrs[dev];
}

PF_API int pf_norm_bwd_static(const void* dy, const void* h, const void* gamma, const void* mean,
                              const void* rstd, const void* dres, void* dx, void* dgamma,
                              void* dbeta, long long rows, int N, int rms, int accumulate,
                              int dtype, int sm_count, void* stream) {
  if (rows <= 0) return 0;
  const long long need = (long long)pf_norm_bwd_ctas(rows, sm_count) * 2 * N;
  if (need > PF_NORM_STATIC_SCRATCH_FLOATS) return -3;   // beyond the built-in scratch
  int err = 0;
  float* scratch = norm_static_scratch_ptr(&err);
  if (!scratch) return err;
  return pf_norm_bwd(dy, h, gamma, mean, rstd, dres, dx, dgamma, dbeta, scratch, rows, N, rms,
                     accumulate, dtype, sm_count, stream);
}
