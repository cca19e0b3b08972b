// Softmax cross-entropy (fused log-softmax + NLL, forward and backward), MSE, embedding
// gather / scatter-add, and rotary position embedding.
#include "common.cuh"
#include "api.h"

namespace pf {

// 16-byte vectors of a row: `head` elements up to the first aligned one, then `nvec` vectors of V
// elements, then the rest.  Rows of an odd length start at any element.
template <typename T>
struct RowSplit {
  static constexpr int V = 16 / sizeof(T);
  int head, nvec;
  __device__ __forceinline__ RowSplit(const T* row, int n) {
    const int mis = (int)((reinterpret_cast<uintptr_t>(row) & 15) / sizeof(T));
    head = min(n, mis ? V - mis : 0);
    nvec = (n - head) / V;
  }
};

// (max, sum of exp(x - max)) of two parts of a row; a part without a finite element is (-inf, 0),
// and (-inf, NaN) when it holds a NaN, which no maximum shows: the sums are always added, and
// -inf, which cannot be subtracted from itself, counts as 0 there.
__device__ __forceinline__ void ce_merge(float& m, float& s, float m2, float s2) {
  const float mm = fmaxf(m, m2), sub = mm == -INFINITY ? 0.f : mm;
  s = s * __expf(m - sub) + s2 * __expf(m2 - sub);
  m = mm;
}

// One pass over a row of logits by THREADS threads: every thread keeps the maximum and the sum of
// exponentials of its elements, raised once per 32 elements.  The per-row log-sum-exp is saved so
// the backward never re-reduces.  loss[row] = lse - x[target] (0 for ignore_index rows).
// Bound by HBM: four 16-byte loads per thread are in flight (2047 x 32000 bf16: 53 -> 37 us,
// 3.5 TB/s, against 2-byte loads and a maximum raised per element).
template <typename T, int THREADS>
__global__ void __launch_bounds__(THREADS < 256 ? 256 : THREADS)
ce_fwd_kernel(const T* __restrict__ logits, const long long* __restrict__ target,
              float* __restrict__ loss, float* __restrict__ lse, long long rows, int V, long long ld,
              long long ignore_index) {
  after_previous();
  constexpr int W = THREADS / 32, VN = RowSplit<T>::V, U = 4;
  constexpr int ROWS = THREADS < 256 ? 256 / THREADS : 1;       // rows per CTA, whole warps each
  static_assert(ROWS == 1 || W == 1, "rows that share a CTA are a warp each");
  __shared__ float smax[W], ssum[W];
  const long long row = (long long)blockIdx.x * ROWS + threadIdx.x / THREADS;
  if (row >= rows) return;
  const int tid = threadIdx.x % THREADS;
  const T* x = logits + row * ld;
  const RowSplit<T> part(x, V);
  float m = -INFINITY, s = 0.f;
  const uint4* xv = reinterpret_cast<const uint4*>(x + part.head);
  for (int i0 = tid; i0 < part.nvec; i0 += U * THREADS) {
    uint4 q[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * THREADS < part.nvec) q[u] = __ldg(xv + i0 + u * THREADS);
    float lm = -INFINITY;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * THREADS < part.nvec) {
        const T* e = reinterpret_cast<const T*>(&q[u]);
#pragma unroll
        for (int j = 0; j < VN; ++j) lm = fmaxf(lm, to_f32<T>(e[j]));
      }
    // a NaN does not move the maximum but reaches the sum below, and every merge keeps it; parts
    // that are -inf so far subtract 0, which leaves their exponentials at zero
    const float mm = fmaxf(m, lm), sub = (mm == -INFINITY) ? 0.f : mm;
    if (lm > m) s *= __expf(m - sub);
    float a = 0.f;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * THREADS < part.nvec) {
        const T* e = reinterpret_cast<const T*>(&q[u]);
#pragma unroll
        for (int j = 0; j < VN; ++j) a += __expf(to_f32<T>(e[j]) - sub);
      }
    s += a;
    m = mm;
  }
  // the elements before the first and after the last vector (at most 2 (V - 1))
  for (int i = tid; i < V - part.nvec * VN; i += THREADS) {
    const float v = to_f32<T>(x[i < part.head ? i : part.nvec * VN + i]);
    ce_merge(m, s, v, 1.f);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    ce_merge(m, s, __shfl_xor_sync(0xffffffffu, m, o), __shfl_xor_sync(0xffffffffu, s, o));
  if (W > 1) {
    const int w = tid >> 5, l = tid & 31;
    if (l == 0) { smax[w] = m; ssum[w] = s; }
    __syncthreads();
    if (w > 0) return;
    m = l < W ? smax[l] : -INFINITY;
    s = l < W ? ssum[l] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      ce_merge(m, s, __shfl_xor_sync(0xffffffffu, m, o), __shfl_xor_sync(0xffffffffu, s, o));
  }
  if (tid == 0) {
    const float L = m + logf(s);
    lse[row] = L;
    const long long t = target[row];
    loss[row] = (t == ignore_index || t < 0 || t >= V) ? 0.f : L - to_f32<T>(x[t]);
  }
}

// sums over a CTA of 1024 threads, for its first warp
__device__ __forceinline__ void ce_mean_fold(float& s, int& n) {
  __shared__ float ssum[32];
  __shared__ int scnt[32];
  s = warp_sum(s);
  n = __reduce_add_sync(0xffffffffu, n);
  if ((threadIdx.x & 31) == 0) { ssum[threadIdx.x >> 5] = s; scnt[threadIdx.x >> 5] = n; }
  __syncthreads();
  if (threadIdx.x < 32) {
    s = warp_sum(ssum[threadIdx.x]);
    n = __reduce_add_sync(0xffffffffu, scnt[threadIdx.x]);
  }
}

// Mean of the row losses over the rows whose target is not ignore_index: mean = sum / count,
// inv = 1 / count (count at least 1).  A call of some thousand rows is one CTA, one launch in the
// place of five of elementwise and reduction kernels; beyond CE_MEAN_ROWS (per-pixel losses) the
// CTAs of ce_mean_part_kernel leave a sum and a count each, and `target` is null here: a million
// rows 86 -> 6 us.
constexpr int CE_MEAN_ROWS = 16384;
__global__ void __launch_bounds__(1024)
ce_mean_kernel(const float* __restrict__ loss, const int* __restrict__ counts,
               const long long* __restrict__ target, float* __restrict__ mean,
               float* __restrict__ inv, int n_in, long long ignore_index) {
  after_previous();
  float s = 0.f;
  int n = 0;
  for (int i = threadIdx.x; i < n_in; i += 1024) {
    s += loss[i];
    n += target ? (int)(target[i] != ignore_index) : counts[i];
  }
  ce_mean_fold(s, n);
  if (threadIdx.x == 0) {
    n = max(1, n);
    *mean = __fdiv_rn(s, (float)n);
    *inv = __fdiv_rn(1.f, (float)n);
  }
}
__global__ void __launch_bounds__(1024)
ce_mean_part_kernel(const float* __restrict__ loss, const long long* __restrict__ target,
                    float* __restrict__ sums, int* __restrict__ counts, long long rows,
                    long long ignore_index) {
  after_previous();
  float s = 0.f;
  int n = 0;
#pragma unroll 4
  for (long long i = (long long)blockIdx.x * 1024 + threadIdx.x; i < rows;
       i += gridDim.x * 1024ll) {
    s += loss[i];
    n += target[i] != ignore_index;
  }
  ce_mean_fold(s, n);
  if (threadIdx.x == 0) { sums[blockIdx.x] = s; counts[blockIdx.x] = n; }
}

// dlogits[row, i] = (exp(x - lse) - [i == target]) * gscale[row]
// gscale = upstream gradient per row, or one for all rows (gstride 0: the mean's, already divided by
// the number of valid rows).  THREADS threads per row; with 256 the grid is (row, slab of the row),
// so that calls of few rows still fill the SMs.  Vectors are used when the row and its gradient lie
// equally to 16 bytes.  2047 x 32000 bf16: 70 -> 51 us, 5.1 TB/s.
template <typename T, int THREADS>
__global__ void __launch_bounds__(256)
ce_bwd_kernel(const T* __restrict__ logits, const long long* __restrict__ target,
              const float* __restrict__ lse, const float* __restrict__ gscale,
              T* __restrict__ dlogits, long long rows, int V, long long ld, long long ignore_index,
              long long gstride) {
  after_previous();
  constexpr int VN = RowSplit<T>::V, UNROLL = THREADS < 128 ? 1 : THREADS < 256 ? 2 : 4;
  const long long row = (long long)blockIdx.x * (256 / THREADS) + threadIdx.x / THREADS;
  if (row >= rows) return;
  const T* x = logits + row * ld;
  T* d = dlogits + row * ld;
  const long long t = target[row];
  const float g = (t == ignore_index) ? 0.f : gscale[row * gstride];
  const float L = lse[row];
  auto grad = [&](float v, int i) {
    float p = __expf(v - L);
    if (i == t) p -= 1.f;
    return p * g;
  };
  const int first = blockIdx.y * THREADS + threadIdx.x % THREADS, step = gridDim.y * THREADS;
  if (((reinterpret_cast<uintptr_t>(x) ^ reinterpret_cast<uintptr_t>(d)) & 15) != 0) {
    for (int i = first; i < V; i += step) d[i] = from_f32<T>(grad(to_f32<T>(x[i]), i));
    return;
  }
  const RowSplit<T> part(x, V);
#pragma unroll UNROLL
  for (int i = first; i < part.nvec; i += step) {
    const uint4 q = __ldg(reinterpret_cast<const uint4*>(x + part.head) + i);
    const T* e = reinterpret_cast<const T*>(&q);
    uint4 o;
    T* oe = reinterpret_cast<T*>(&o);
    const int c0 = part.head + i * VN;
#pragma unroll
    for (int j = 0; j < VN; ++j) oe[j] = from_f32<T>(grad(to_f32<T>(e[j]), c0 + j));
    reinterpret_cast<uint4*>(d + part.head)[i] = o;
  }
  for (int k = first; k < V - part.nvec * VN; k += step) {
    const int i = k < part.head ? k : part.nvec * VN + k;
    d[i] = from_f32<T>(grad(to_f32<T>(x[i]), i));
  }
}

// MSE: per-CTA partial sums of (a-b)^2 in fp32 -> atomicAdd into out[0]; backward elementwise.
template <typename T>
__global__ void __launch_bounds__(256)
mse_fwd_kernel(const T* __restrict__ a, const T* __restrict__ b, float* __restrict__ out,
               long long n, float inv_n) {
  after_previous();
  __shared__ float red[8];
  float s = 0.f;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const float d = to_f32<T>(a[i]) - to_f32<T>(b[i]);
    s += d * d;
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int i = 0; i < 8; ++i) t += red[i];
    atomicAdd(out, t * inv_n);
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
mse_bwd_kernel(const T* __restrict__ a, const T* __restrict__ b, const float* __restrict__ gout,
               T* __restrict__ da, long long n, float two_inv_n) {
  after_previous();
  const float g = gout[0] * two_inv_n;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    da[i] = from_f32<T>((to_f32<T>(a[i]) - to_f32<T>(b[i])) * g);
}

// Embedding gather: out[t, :] = table[ids[t], :]   (table fp32 or 16-bit -> out T)
template <typename TT, typename T>
__global__ void __launch_bounds__(256)
embed_fwd_kernel(const TT* __restrict__ table, const long long* __restrict__ ids,
                 T* __restrict__ out, int D, long long vocab) {
  after_previous();
  const long long t = blockIdx.x;
  long long id = ids[t];
  if (id < 0 || id >= vocab) id = 0;
  for (int i = threadIdx.x; i < D; i += 256)
    out[t * D + i] = from_f32<T>(to_f32<TT>(table[id * D + i]));
}

// Embedding scatter-add into an fp32 gradient table
template <typename T>
__global__ void __launch_bounds__(256)
embed_bwd_kernel(const T* __restrict__ dout, const long long* __restrict__ ids,
                 float* __restrict__ dtable, int D, long long vocab) {
  after_previous();
  const long long t = blockIdx.x;
  const long long id = ids[t];
  if (id < 0 || id >= vocab) return;
  for (int i = threadIdx.x; i < D; i += 256)
    atomicAdd(dtable + id * D + i, to_f32<T>(dout[t * D + i]));
}

// Rotary embedding on a (possibly strided) x[B, S, H, D] (half-split convention: pairs
// (i, i + D/2)) into a contiguous output.  inverse != 0 applies the transpose rotation (the backward).
// Rotary embedding, 16 bytes per access: a thread rotates 8 consecutive pairs (x[d], x[d+D/2]),
// d = 8 * v .. 8 * v + 7.  Needs D/2 a multiple of 8 and 16-byte aligned rows.
template <typename T>
__global__ void __launch_bounds__(256)
rope_vec_kernel(const T* __restrict__ x, T* __restrict__ out, const float* __restrict__ cos_t,
                const float* __restrict__ sin_t, long long B, int S, int H, int D,
                long long stride_b, long long stride_s, long long stride_h, int inverse) {
  after_previous();
  const int half = D / 2, hv = half / 8;
  const long long total = B * S * H * hv;
  const long long gstride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gstride) {
    const int v = (int)(i % hv);
    long long r = i / hv;
    const int h = (int)(r % H); r /= H;
    const int s = (int)(r % S);
    const long long b = r / S;
    const T* src = x + b * stride_b + (long long)s * stride_s + (long long)h * stride_h + v * 8;
    const uint4 u1 = *reinterpret_cast<const uint4*>(src);
    const uint4 u2 = *reinterpret_cast<const uint4*>(src + half);
    const float4* cp = reinterpret_cast<const float4*>(cos_t + (long long)s * half + v * 8);
    const float4* sp = reinterpret_cast<const float4*>(sin_t + (long long)s * half + v * 8);
    const float4 c0 = __ldg(cp), c1 = __ldg(cp + 1), s0 = __ldg(sp), s1 = __ldg(sp + 1);
    const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const float sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    const T* e1 = reinterpret_cast<const T*>(&u1);
    const T* e2 = reinterpret_cast<const T*>(&u2);
    uint4 o1, o2;
    T* q1 = reinterpret_cast<T*>(&o1);
    T* q2 = reinterpret_cast<T*>(&o2);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float x1 = to_f32<T>(e1[j]), x2 = to_f32<T>(e2[j]);
      const float sj = inverse ? -sn[j] : sn[j];
      q1[j] = from_f32<T>(x1 * c[j] - x2 * sj);
      q2[j] = from_f32<T>(x2 * c[j] + x1 * sj);
    }
    // the output is always contiguous [B, S, H, D]
    T* dst = out + ((b * S + s) * H + h) * (long long)D + v * 8;
    *reinterpret_cast<uint4*>(dst) = o1;
    *reinterpret_cast<uint4*>(dst + half) = o2;
  }
}

// The same rotation over a whole fused projection [rows = B*S][3][H][D]: slices 0 and 1 (queries, keys)
// are rotated, slice 2 is copied, so that one kernel per direction takes the place of two rotations
// and, in the backward, of the fills, strided copies and additions that join the gradients of three
// slices.  One CTA per row; bound by HBM: the tensor is read and written once.  [1, 2048, 3, 32, 128]
// bf16: 18 us in a decoder layer (26 with L2 flushed) and as much backward, where 34 us went into
// rotations and 137 into joining slices.
template <typename T>
__global__ void __launch_bounds__(256)
rope_qkv_kernel(const T* __restrict__ x, T* __restrict__ out, const float* __restrict__ cos_t,
                const float* __restrict__ sin_t, int S, int H, int D, int inverse) {
  after_previous();
  const int half = D / 2, hv = half / 8;
  const long long row = blockIdx.x;
  const T* src = x + row * 3 * H * D;
  T* dst = out + row * 3 * H * D;
  const float* ct = cos_t + (row % S) * half;
  const float* st = sin_t + (row % S) * half;
  const int n_rot = 2 * H * hv;
  for (int i = threadIdx.x; i < n_rot; i += 256) {
    const int jh = i / hv, v = i - jh * hv, off = jh * D + v * 8;
    const uint4 u1 = *reinterpret_cast<const uint4*>(src + off);
    const uint4 u2 = *reinterpret_cast<const uint4*>(src + off + half);
    const float4* cp = reinterpret_cast<const float4*>(ct + v * 8);
    const float4* sp = reinterpret_cast<const float4*>(st + v * 8);
    const float4 c0 = __ldg(cp), c1 = __ldg(cp + 1), s0 = __ldg(sp), s1 = __ldg(sp + 1);
    const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const float sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    const T* e1 = reinterpret_cast<const T*>(&u1);
    const T* e2 = reinterpret_cast<const T*>(&u2);
    uint4 o1, o2;
    T* q1 = reinterpret_cast<T*>(&o1);
    T* q2 = reinterpret_cast<T*>(&o2);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float x1 = to_f32<T>(e1[j]), x2 = to_f32<T>(e2[j]);
      const float sj = inverse ? -sn[j] : sn[j];
      q1[j] = from_f32<T>(x1 * c[j] - x2 * sj);
      q2[j] = from_f32<T>(x2 * c[j] + x1 * sj);
    }
    *reinterpret_cast<uint4*>(dst + off) = o1;
    *reinterpret_cast<uint4*>(dst + off + half) = o2;
  }
  const uint4* vs = reinterpret_cast<const uint4*>(src + 2 * H * D);
  uint4* vd = reinterpret_cast<uint4*>(dst + 2 * H * D);
  for (int i = threadIdx.x; i < H * D / 8; i += 256) vd[i] = vs[i];
}

template <typename T>
__global__ void __launch_bounds__(256)
rope_kernel(const T* __restrict__ x, T* __restrict__ out, const float* __restrict__ cos_t,
            const float* __restrict__ sin_t, long long B, int S, int H, int D,
            long long stride_b, long long stride_s, long long stride_h, int inverse) {
  after_previous();
  const int half = D / 2;
  const long long total = B * S * H * half;
  const long long gstride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gstride) {
    const int d = (int)(i % half);
    long long r = i / half;
    const int h = (int)(r % H); r /= H;
    const int s = (int)(r % S);
    const long long b = r / S;
    const long long off = b * stride_b + (long long)s * stride_s + (long long)h * stride_h;
    const float c = cos_t[s * half + d];
    float sn = sin_t[s * half + d];
    if (inverse) sn = -sn;
    const float x1 = to_f32<T>(x[off + d]);
    const float x2 = to_f32<T>(x[off + d + half]);
    // the output is always contiguous [B, S, H, D]
    const long long oo = ((b * S + s) * H + h) * (long long)D;
    out[oo + d] = from_f32<T>(x1 * c - x2 * sn);
    out[oo + d + half] = from_f32<T>(x2 * c + x1 * sn);
  }
}

}  // namespace pf

using namespace pf;

#define PF_DISPATCH3(dtype, ...)                               \
  switch (dtype) {                                             \
    case PF_F32: { using T = float; __VA_ARGS__; } break;       \
    case PF_F16: { using T = __half; __VA_ARGS__; } break;      \
    case PF_BF16: { using T = __nv_bfloat16; __VA_ARGS__; } break; \
    default: return -1;                                        \
  }

// Threads per row of the forward: with a CTA per short row a call is bound by the rate of CTAs, so
// a row of up to 1024 elements is a warp's (200000 x 300 bf16: 351 -> 77 us, one row 2.6 -> 2.4); at
// 1500 a CTA of 256 is ahead for few rows (64: 2.8 against 3.0 us).  Calls of no more rows than SMs
// give a long row 1024 threads: 64 x 12000 3.8 -> 3.5 us, 1 x 60001 8.9 -> 5.8, but 64 x 8192
// 3.1 -> 3.4 and 400 x 32000 8.2 -> 8.7.
static int ce_fwd_threads(long long rows, int V, int sm_count) {
  if (V <= 1024) return 32;
  return rows <= sm_count && V > 8192 ? 1024 : 256;
}
// Threads per row of the backward, by the vectors of a row: a warp up to 64 (200000 x 512 bf16:
// 284 -> 77 us), half a CTA up to 512 (20000 x 2048 fp32: 66 -> 54 us) unless the rows are too
// few to fill the SMs (64 x 4096 bf16: 3.2 against 2.4 us).
template <typename T>
static int ce_bwd_threads(long long rows, int V, int sm_count) {
  const int nvec = V / RowSplit<T>::V;
  if (nvec <= 64) return 32;
  return nvec <= 512 && rows > 2 * sm_count ? 128 : 256;
}

PF_API int pf_ce_fwd(const void* logits, const void* target, void* loss, void* lse, long long rows,
                     int V, long long ld, long long ignore_index, int dtype, int sm_count,
                     void* stream) {
  if (rows <= 0) return 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
#define PF_CE_FWD(THREADS)                                                                       \
  after(ce_fwd_kernel<T, THREADS>, (unsigned)(THREADS < 256 ? (rows + 7) / 8 : rows),                 \
                              THREADS < 256 ? 256 : THREADS, 0, st)(                           \
      (const T*)logits, (const long long*)target, (float*)loss, (float*)lse, rows, V, ld,        \
      ignore_index)
  PF_DISPATCH3(dtype, {
    const int threads = ce_fwd_threads(rows, V, sm_count);
    if (threads == 32) PF_CE_FWD(32);
    else if (threads == 256) PF_CE_FWD(256);
    else PF_CE_FWD(1024);
  });
#undef PF_CE_FWD
  PF_CHECK_LAUNCH();
  return 0;
}

// CTAs that share the sum of the row losses; more than one need scratch of that many floats and ints
PF_API int pf_ce_mean_parts(long long rows, int sm_count) {
  if (rows <= CE_MEAN_ROWS) return 1;
  const long long n = (rows + CE_MEAN_ROWS / 4 - 1) / (CE_MEAN_ROWS / 4);
  return (int)(n < sm_count ? n : sm_count);
}

// mean loss over the rows that count, and one over their number
PF_API int pf_ce_mean(const void* loss, const void* target, void* scratch, void* mean, void* inv,
                      long long rows, long long ignore_index, int sm_count, void* stream) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int parts = pf_ce_mean_parts(rows, sm_count);
  if (parts > 1) {
    float* sums = (float*)scratch;
    int* counts = (int*)scratch + parts;
    after(ce_mean_part_kernel, parts, 1024, 0, st)((const float*)loss, (const long long*)target, sums,
                                                counts, rows, ignore_index);
    after(ce_mean_kernel, 1, 1024, 0, st)(sums, counts, nullptr, (float*)mean, (float*)inv, parts,
                                       ignore_index);
  } else {
    after(ce_mean_kernel, 1, 1024, 0, st)((const float*)loss, nullptr, (const long long*)target,
                                       (float*)mean, (float*)inv, (int)rows, ignore_index);
  }
  PF_CHECK_LAUNCH();
  return 0;
}

// gscale: one value per row (gstride 1) or one for all (gstride 0)
PF_API int pf_ce_bwd(const void* logits, const void* target, const void* lse, const void* gscale,
                     void* dlogits, long long rows, int V, long long ld, long long ignore_index,
                     long long gstride, int dtype, int sm_count, void* stream) {
  if (rows <= 0) return 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // up to the eight CTAs that an SM holds where the row length allows it (a slab: 256 vectors or
  // more); one more would be a second round (591 x 8192 bf16: 5.9 -> 5.1 us)
  long long slabs = 8ll * sm_count / rows;
  const long long most = (V + 2047) / 2048;
  if (slabs > most) slabs = most;
  if (slabs < 1) slabs = 1;
#define PF_CE_BWD(THREADS, GRID)                                                                 \
  after(ce_bwd_kernel<T, THREADS>, GRID, 256, 0, st)(                                               \
      (const T*)logits, (const long long*)target, (const float*)lse, (const float*)gscale,       \
      (T*)dlogits, rows, V, ld, ignore_index, gstride)
  PF_DISPATCH3(dtype, {
    const int threads = ce_bwd_threads<T>(rows, V, sm_count);
    if (threads == 32) PF_CE_BWD(32, (unsigned)((rows + 7) / 8));
    else if (threads == 128) PF_CE_BWD(128, (unsigned)((rows + 1) / 2));
    else PF_CE_BWD(256, dim3((unsigned)rows, (unsigned)slabs));
  });
#undef PF_CE_BWD
  PF_CHECK_LAUNCH();
  return 0;
}

PF_API int pf_mse_fwd(const void* a, const void* b, void* out_f32, long long n, int dtype,
                      int sm_count, void* stream) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  cudaMemsetAsync(out_f32, 0, sizeof(float), st);
  if (n <= 0) return 0;
  long long blocks = (n + 255) / 256;
  const long long cap = (long long)(sm_count > 0 ? sm_count : 148) * 8;
  if (blocks > cap) blocks = cap;
  PF_DISPATCH3(dtype, (after(mse_fwd_kernel<T>, (unsigned)blocks, 256, 0, st)(
      (const T*)a, (const T*)b, (float*)out_f32, n, 1.0f / (float)n)));
  PF_CHECK_LAUNCH();
  return 0;
}

PF_API int pf_mse_bwd(const void* a, const void* b, const void* gout_f32, void* da, long long n,
                      int dtype, int sm_count, void* stream) {
  if (n <= 0) return 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  long long blocks = (n + 255) / 256;
  const long long cap = (long long)(sm_count > 0 ? sm_count : 148) * 8;
  if (blocks > cap) blocks = cap;
  PF_DISPATCH3(dtype, (after(mse_bwd_kernel<T>, (unsigned)blocks, 256, 0, st)(
      (const T*)a, (const T*)b, (const float*)gout_f32, (T*)da, n, 2.0f / (float)n)));
  PF_CHECK_LAUNCH();
  return 0;
}

PF_API int pf_embed_fwd(const void* table, const void* ids, void* out, long long tokens, int D,
                        long long vocab, int table_dtype, int out_dtype, void* stream) {
  if (tokens <= 0) return 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const long long* I = (const long long*)ids;
#define PF_EMB(TD, TT_, OD, OT_) \
  if (table_dtype == TD && out_dtype == OD) after(embed_fwd_kernel<TT_, OT_>, (unsigned)tokens, 256, 0, st)((const TT_*)table, I, (OT_*)out, D, vocab);
  PF_EMB(PF_F32, float, PF_F32, float)
  else PF_EMB(PF_F32, float, PF_F16, __half)
  else PF_EMB(PF_F32, float, PF_BF16, __nv_bfloat16)
  else PF_EMB(PF_F16, __half, PF_F16, __half)
  else PF_EMB(PF_BF16, __nv_bfloat16, PF_BF16, __nv_bfloat16)
  else return -1;
  PF_CHECK_LAUNCH();
  return 0;
}

PF_API int pf_embed_bwd(const void* dout, const void* ids, void* dtable_f32, long long tokens,
                        int D, long long vocab, int dtype, void* stream) {
  if (tokens <= 0) return 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  PF_DISPATCH3(dtype, (after(embed_bwd_kernel<T>, (unsigned)tokens, 256, 0, st)(
      (const T*)dout, (const long long*)ids, (float*)dtable_f32, D, vocab)));
  PF_CHECK_LAUNCH();
  return 0;
}

// x, out: [rows = B*S][3][H][D] 16-bit, contiguous; cos / sin fp32 [S, D/2].  Needs D a multiple of 16
// and 16-byte aligned pointers (-2 otherwise).
PF_API int pf_rope_qkv(const void* x, void* out, const void* cos_t, const void* sin_t,
                       long long rows, int S, int H, int D, int inverse, int dtype, void* stream) {
  if (rows <= 0) return 0;
  if (dtype != PF_F16 && dtype != PF_BF16) return -1;
  if (D % 16 || rows > 0x7fffffffll || (reinterpret_cast<uintptr_t>(x) & 15) ||
      (reinterpret_cast<uintptr_t>(out) & 15) || (reinterpret_cast<uintptr_t>(cos_t) & 15) ||
      (reinterpret_cast<uintptr_t>(sin_t) & 15))
    return -2;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (dtype == PF_F16)
    after(rope_qkv_kernel<__half>, (unsigned)rows, 256, 0, st)((const __half*)x, (__half*)out,
        (const float*)cos_t, (const float*)sin_t, S, H, D, inverse);
  else
    after(rope_qkv_kernel<__nv_bfloat16>, (unsigned)rows, 256, 0, st)((const __nv_bfloat16*)x,
        (__nv_bfloat16*)out, (const float*)cos_t, (const float*)sin_t, S, H, D, inverse);
  PF_CHECK_LAUNCH();
  return 0;
}

PF_API int pf_rope(const void* x, void* out, const void* cos_t, const void* sin_t, long long B,
                   int S, int H, int D, long long stride_b, long long stride_s,
                   long long stride_h, int inverse, int dtype, int sm_count, void* stream) {
  const long long total = B * S * H * (D / 2);
  if (total <= 0) return 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const long long cap = (long long)(sm_count > 0 ? sm_count : 148) * 8;
  const bool vec = dtype != PF_F32 && D % 16 == 0 && stride_b % 8 == 0 && stride_s % 8 == 0 &&
                   stride_h % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(out) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(cos_t) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(sin_t) & 15) == 0;
  if (vec) {
    long long vblocks = (total / 8 + 255) / 256;
    if (vblocks > cap) vblocks = cap;
    if (vblocks < 1) vblocks = 1;
    switch (dtype) {
      case PF_F16:
        after(rope_vec_kernel<__half>, (unsigned)vblocks, 256, 0, st)(
            (const __half*)x, (__half*)out, (const float*)cos_t, (const float*)sin_t, B, S, H, D,
            stride_b, stride_s, stride_h, inverse);
        break;
      default:
        after(rope_vec_kernel<__nv_bfloat16>, (unsigned)vblocks, 256, 0, st)(
            (const __nv_bfloat16*)x, (__nv_bfloat16*)out, (const float*)cos_t,
            (const float*)sin_t, B, S, H, D, stride_b, stride_s, stride_h, inverse);
    }
    PF_CHECK_LAUNCH();
    return 0;
  }
  long long blocks = (total + 255) / 256;
  if (blocks > cap) blocks = cap;
  PF_DISPATCH3(dtype, (after(rope_kernel<T>, (unsigned)blocks, 256, 0, st)(
      (const T*)x, (T*)out, (const float*)cos_t, (const float*)sin_t, B, S, H, D, stride_b,
      stride_s, stride_h, inverse)));
  PF_CHECK_LAUNCH();
  return 0;
}
