// Flash attention backward for sm_100a on tcgen05 tensor cores.
//
// Scores are computed transposed (rows = keys, columns = queries), so that the probabilities and
// their gradients come out in the layout the products over queries read as their A operand:
//     S^T  = K Q^T                      P^T  = exp2(S^T c - lse2)
//     dP^T = V dO^T                     dS^T = P^T (dP^T - delta) scale
//     dV += P^T dO     A = P^T straight from TMEM (16-bit), never in shared memory
//     dK += dS^T Q     A = dS^T in shared memory, K-major, or up to head dim 64 in the columns of dP^T
//     dQ  = dS K       A = the same dS^T tile, read as an MN-major operand
// Queries lie along the N side of the first two products and along the reduction of the next two,
// so a ragged last query tile costs what its rows cost, not a full tile; a ragged last key tile costs a
// full one.  One or two tokens beyond full tiles (ViT: 257 = 2 x 128 + the class token) are taken out of
// the tiles and handled by attn_bwd_edge_kernel.
//
// One CTA per SM walks over (key tile, head, batch) items; roles of its 16 warps:
//   warps 0-7    softmax side: thread <-> key row (TMEM lane), each warp half of the 128 queries
//   warps 8-11   drain: dQ tiles out of TMEM into the fp32 sums (TMA reduce-add through swizzled
//                boxes), and dK / dV at the end of an item while the next item is under way
//   warp 12      TMA producer      warp 13  MMA issuer, TMEM owner (14, 15: idle)
// What bounds it: per 128 x 128 tile pair 16384 exponentials (1024 cycles of the special-function
// units) against 5 products (1400 cycles at head dim 64, 2560 at 128), so the tensor core must
// never wait for the element-wise part.  Order of the MMA warp for tile i:
//   head dim <= 64   S(i+1) as soon as S(i) is in registers, dV(i), dK(i), dQ(i), dP(i+1), or with
//                    one key tile dP(i+1) before dK(i)
//   96               S(i+1) as soon as S(i) is in registers, dV(i), dQ(i), dK(i), dP(i+1)
//   128              dV(i), S(i+1) once dV(i) has read P^T, dQ(i), dK(i), dP(i+1)
// TMEM (512 columns): S^T 128, dP^T 128, P^T 64 (16-bit), dV, dK, dQ one head dim each.  At 96 dQ
// takes the columns of dP^T (dead once dS^T is in shared memory; the next dP^T waits until dQ is
// drained), at 128 P^T also takes the columns of S^T.
//
// Measured (B200, CUDA events, L2 flushed, with the pre- and post-pass), against one CTA per key
// tile that ran the five products and the element-wise part one after the other with scalar
// reductions into dQ: [4, 4096, 10, 64] 1330 -> 549 us, [2, 2048, 16, 128] 445 -> 222,
// causal [1, 2048, 32, 128] 302 -> 138, [24, 257, 16, 88] 192 -> 142.  Steps on the way at
// [4, 4096, 10, 64]: 877; 690 with one elected thread issuing the products (before, issuing the 28 of
// a tile pair took 4000 cycles); 590 with tile paths free of masks, barriers looked at together, the
// next 32 columns on their way while the last are worked on, and negated statistics; 549 with dS^T
// for dK in tensor memory.  At head dim 128: 261; 222 with S(i+1) issued under the dS^T of tile i and
// dQ leaving TMEM ahead of its boxes.
//
// Where a CTA takes all key tiles of a head (DQ_WHOLE), dQ needs neither clearing, adding in memory nor
// converting, and dK and dV leave through boxes (rotating inputs, everything included): [24, 257, 16, 88]
// 136 -> 107 us with its leftover token, [64, 257, 16, 64] 286 -> 163, [16, 256, 16, 64] 52 -> 42.5,
// [24, 400, 24, 32] 218 -> 167.  At head dim 88 the items of a head are bound by waits: dQ's way out through
// the columns of dP^T, and K and V, which have one place and arrive after the last product of the item before.
//
// A pre-pass writes per query tile the row statistics [128 x -lse2 | 128 x -delta scale] (-inf / 0
// beyond the last query, which makes the probabilities there zero without a test) and clears the fp32
// dQ sums; a post-pass converts them.  With one key tile the dQ tiles are complete and go straight to
// their 16-bit destination: no sums, no post-pass.
#include <climits>
#include <type_traits>
#include "attn_common.cuh"
#include "api.h"

namespace pf {

constexpr int BWD_LEFT_MAX = 2;       // leftover tokens of a head handled on CUDA cores (see bwd_plan)
constexpr int BWD_WHOLE_TILES = 8;    // most query tiles of a head that one CTA takes whole: its sums stay in L2

struct AttnBwdParams {
  int B, H, Sq, Sk, D;
  int causal;
  float scale;
  int fmt;              // 0 fp16, 1 bf16
  const float* stats;   // [B*H][query tiles][256]: -lse * log2(e), then -delta * scale
  void *dq, *dk, *dv;   // strides (batch, seq, head) in elements
  long long sdq[3], sdkv[3];
  int n_kt, n_qt;
  int* status;
  float4* part;         // DQ_WHOLE: per CTA the dQ of its head so far, [query tile][DP / 4][128 rows]
  // leftover rows (attn_bwd_edge_kernel): their number, their weights, and where q, k, dO begin
  int left;
  float* edge;          // [B*H][left][3][n_qt * 128]: P and dS of query n + t by key, dS of key n + t by query
  const void *q, *k, *dout;
  long long sq[3], sk[3];
};

// What becomes of a dQ tile.  DQ_SUMS: added to fp32 sums in memory, which a post-pass converts.
// DQ_DIRECT: one key tile, it is complete.  DQ_WHOLE: a CTA takes all key tiles of a head in turn, so the
// thread that drains a row of dQ keeps that row's sum, in a buffer of the CTA's own that never leaves L2,
// and writes 16 bits after the last one: nothing to clear, to add in memory or to convert.
// DQ_TILE: DQ_DIRECT for a few rows in one tile of either kind.  Its outputs leave by 16-byte stores, whose cost goes
// by the row, and not through boxes, each of which waits for the one before the last.  us over us with boxes and
// without, 1200 heads: head dim 64, 17 tokens 1.08, 64 1.03, 100 0.94; head dim 128, 17 1.10, 64 1.05, 77 0.96; 96 heads,
// which no other item follows: head dim 128, 33 tokens 1.04, 49 0.97, 64 0.92.
enum DqMode : int { DQ_SUMS = 0, DQ_DIRECT = 1, DQ_WHOLE = 2, DQ_TILE = 3 };
constexpr int BWD_TILE_ROWS = 192, BWD_TILE_ROWS_ONCE = 112;   // most rows of dQ, dK and dV of DQ_TILE

// One 8-lane group per (batch, padded query, head): delta = dO . O, statistics, cleared dQ sums.
template <typename T>
__global__ void __launch_bounds__(256)
attn_bwd_prep_kernel(const T* __restrict__ dout, const T* __restrict__ out,
                     const float* __restrict__ lse, float* __restrict__ stats,
                     float* __restrict__ dq_accum, int B, int S, int H, int D, int n_qt,
                     float scale) {
  after_previous();
  const int lane = threadIdx.x & 31, sub = lane & 7;
  const long long g = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * 4 + (lane >> 3);
  const int s_pad = n_qt * ATT_BM;
  const bool in = g < (long long)B * s_pad * H;
  const int h = in ? (int)(g % H) : 0;
  const long long bs = g / H;
  const int i = in ? (int)(bs % s_pad) : 0;
  const long long b = in ? bs / s_pad : 0;
  const bool live = in && i < S;
  const long long row = (b * S + i) * H + h;
  float s = 0.f;
  if (live) {
    const uint4* a = reinterpret_cast<const uint4*>(dout + row * D);
    const uint4* c = reinterpret_cast<const uint4*>(out + row * D);
    for (int v = sub; v < D / 8; v += 8) {
      const uint4 ua = __ldg(a + v), uc = __ldg(c + v);
      const T* ea = reinterpret_cast<const T*>(&ua);
      const T* ec = reinterpret_cast<const T*>(&uc);
#pragma unroll
      for (int j = 0; j < 8; ++j) s = fmaf(to_f32<T>(ea[j]), to_f32<T>(ec[j]), s);
      if (dq_accum) {
        float4* z = reinterpret_cast<float4*>(dq_accum + row * D) + 2 * v;
        z[0] = make_float4(0.f, 0.f, 0.f, 0.f);
        z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
  }
  s += __shfl_xor_sync(0xffffffffu, s, 4);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  if (in && sub == 0) {
    float* st = stats + (((b * H + h) * n_qt + i / ATT_BM) * 2) * ATT_BM + i % ATT_BM;
    st[0] = live ? -lse[(b * H + h) * S + i] * LOG2E : -INFINITY;
    st[ATT_BM] = live ? -s * scale : 0.f;
  }
}

// What the leftover rows of a head of n + left tokens (n a multiple of 128) take part in, on CUDA cores:
// one CTA per head walks over its tokens x once per leftover token r with
//     weights of query r by key x      P_r[x] = exp2(q_r k_x c - lse2_r),  dS_r[x] = P (dO_r v_x - delta_r) scale
//     weights of key r by query x      P[x], dS[x] likewise from q_x k_r, dO_x v_r
//     dQ_r = sum dS_r[x] k_x,  dV_r = sum P[x] dO_x,  dK_r = sum dS[x] q_x          (complete, written here)
// and leaves the weights that touch the other tokens to the kernel below (AttnBwdParams::edge), with the
// row statistics of the pre-pass, whose reads of O and dO it shares.
// Four lanes share a token: with 8 or 16 the sums over lanes and the reads of token r's values from shared
// memory bound it ([24, 257, 16, 88] 35 us, now 30).  A thread asks for its next token's five rows while it
// works on this one's, in slots of its own, so that the loop has no barrier.
template <int DP>
struct EdgeCfg {
  static constexpr int NV = DP / 32;                     // vectors of 8 columns per lane
  static constexpr int THREADS = 128, GROUPS = THREADS / 4;
  // per SM: shared memory bounds it above head dim 64, registers below.  Four there gain where heads fill
  // them ([64, 257, 16, 64] 154 -> 150 us with the tiles, [32, 129, 16, 64] 44 -> 40) and lose 1 to 2 %
  // where they do not ([8, 257, 12, 64] 27.1 -> 27.6).
  static constexpr int CTAS = NV > 3 ? 2 : 3, CTAS_MANY = NV > 2 ? CTAS : 4;
  static constexpr int RING = 2 * 5 * NV * THREADS * 16;
  static constexpr int OFF_VECS = RING, OFF_LSE = OFF_VECS + 4 * DP * 4;
  static constexpr int SMEM = OFF_LSE + (BWD_WHOLE_TILES * ATT_BM + BWD_LEFT_MAX) * 4;
  static_assert(4 * 3 * DP * 4 <= RING, "the warps' sums lie over the ring");
};

template <typename T, int DP, int CTAS>
__global__ void __launch_bounds__(EdgeCfg<DP>::THREADS, CTAS)
attn_bwd_edge_kernel(const AttnBwdParams p, const T* __restrict__ v, const T* __restrict__ out,
                     const float* __restrict__ lse, float* __restrict__ stats, const long long sv0,
                     const long long sv1, const long long sv2) {
  after_previous();
  using C = EdgeCfg<DP>;
  constexpr int NV = C::NV, THREADS = C::THREADS, GROUPS = C::GROUPS;
  extern __shared__ __align__(16) uint8_t edge_smem[];
  uint4* ring = reinterpret_cast<uint4*>(edge_smem) + threadIdx.x;              // [2][5][NV][THREADS]
  float* vecs = reinterpret_cast<float*>(edge_smem + C::OFF_VECS);              // q, k, v, dO of token r
  float* nlse = reinterpret_cast<float*>(edge_smem + C::OFF_LSE);
  float (*red)[3][DP] = reinterpret_cast<float (*)[3][DP]>(edge_smem);          // after the loop
  const int h = blockIdx.x, b = blockIdx.y, n = p.Sq, S = n + p.left;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & 3, grp = threadIdx.x >> 2;
  const long long bh = (long long)b * p.H + h;
  const float c2 = p.scale * LOG2E;
  // rows of q, k, v, dO, O; this lane's columns are vectors sub, sub + 4, ...
  const T* base[5] = {reinterpret_cast<const T*>(p.q) + b * p.sq[0] + h * p.sq[2],
                      reinterpret_cast<const T*>(p.k) + b * p.sk[0] + h * p.sk[2],
                      v + b * sv0 + h * sv2,
                      reinterpret_cast<const T*>(p.dout) + (b * (long long)S * p.H + h) * p.D,
                      out + (b * (long long)S * p.H + h) * p.D};
  const long long so = (long long)p.H * p.D;
  const long long stride[5] = {p.sq[1], p.sk[1], sv1, so, so};
  auto in = [&](int i) { return (sub + 4 * i) * 8 < p.D; };
  for (int x = threadIdx.x; x < S; x += THREADS) nlse[x] = -lse[bh * S + x] * LOG2E;
  const int trips = (S + GROUPS - 1) / GROUPS;           // the same for every lane
  auto fetch = [&](int trip) {
    const int x = min(trip * GROUPS + grp, S - 1);
    uint4* slot = ring + (trip & 1) * 5 * NV * THREADS;
    if (trip < trips) {
#pragma unroll
      for (int a = 0; a < 5; ++a)
#pragma unroll
        for (int i = 0; i < NV; ++i)
          if (in(i)) cp_async16(slot + (a * NV + i) * THREADS, base[a] + x * stride[a] + (sub + 4 * i) * 8);
    }
    cp_async_commit();
  };
  auto widen = [](const uint4& u, float* f) {
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = to_f32<T>(reinterpret_cast<const T*>(&u)[j]);
  };
  auto dot = [](const float (&a)[8 * NV], const float (&c)[8 * NV]) {
    float s[NV] = {};
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int i = 0; i < NV; ++i) s[i] = fmaf(a[i * 8 + j], c[i * 8 + j], s[i]);
    float r = s[0];
#pragma unroll
    for (int i = 1; i < NV; ++i) r += s[i];
    return r;
  };
  auto over_lanes = [](float s) {      // whole warps take part, whichever of their tokens exist
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    return s + __shfl_xor_sync(0xffffffffu, s, 1);
  };
  for (int t = 0; t < p.left; ++t) {
    const int r = n + t;
#pragma unroll
    for (int i = 0; i < 2 * 5 * NV; ++i)                 // columns beyond D count as zeros
      if (!in(i % NV)) ring[i * THREADS] = make_uint4(0, 0, 0, 0);
    fetch(0);
    if (threadIdx.x < DP)
#pragma unroll
      for (int a = 0; a < 4; ++a)
        vecs[a * DP + threadIdx.x] =
            (int)threadIdx.x < p.D ? to_f32<T>(base[a][r * stride[a] + threadIdx.x]) : 0.f;
    float f[8 * NV], g[8 * NV], w[8 * NV], dq[8 * NV] = {}, dk[8 * NV] = {}, dv[8 * NV] = {};
    auto own = [&](const T* row, float (&to)[8 * NV]) {
#pragma unroll
      for (int i = 0; i < NV; ++i)
        widen(in(i) ? __ldg(reinterpret_cast<const uint4*>(row) + sub + 4 * i) : make_uint4(0, 0, 0, 0),
              to + i * 8);
    };
    own(base[3] + r * so, g);
    own(base[4] + r * so, f);
    const float delta_r = over_lanes(dot(g, f));
    __syncthreads();
    const float nlse_r = nlse[r];
    auto vec = [&](int a, float (&to)[8 * NV]) {
#pragma unroll
      for (int i = 0; i < NV; ++i)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const float4 q = *reinterpret_cast<const float4*>(vecs + a * DP + (sub + 4 * i) * 8 + u * 4);
          float* o = to + i * 8 + u * 4;
          o[0] = q.x; o[1] = q.y; o[2] = q.z; o[3] = q.w;
        }
    };
    float* e = p.edge + (bh * p.left + t) * 3 * n;
    for (int trip = 0; trip < trips; ++trip) {
      fetch(trip + 1);
      cp_async_wait<1>();
      const int x = trip * GROUPS + grp;
      const bool live = x < S;          // the others hold a copy of the last token and take no part
      const uint4* slot = ring + (trip & 1) * 5 * NV * THREADS;
      auto row = [&](int a, float (&to)[8 * NV]) {
#pragma unroll
        for (int i = 0; i < NV; ++i) widen(slot[(a * NV + i) * THREADS], to + i * 8);
      };
      const float nlse_x = nlse[min(x, S - 1)];
      row(3, g);
      row(4, f);
      const float delta_x = over_lanes(dot(g, f));
      vec(2, w);
      const float dp_x = over_lanes(dot(g, w));           // dO_x v_r
      row(2, f);
      vec(3, w);
      const float dp_r = over_lanes(dot(f, w));           // dO_r v_x
      row(1, f);
      vec(0, w);
      const float s_r = over_lanes(dot(f, w));
      const float p_r = exp2f(fmaf(s_r, c2, nlse_r));
      const float ds_r = p_r * (dp_r - delta_r) * p.scale;
      if (live) {
#pragma unroll
        for (int j = 0; j < 8 * NV; ++j) dq[j] = fmaf(ds_r, f[j], dq[j]);
      }
      row(0, f);
      vec(1, w);
      const float s_x = over_lanes(dot(f, w));
      const float p_x = exp2f(fmaf(s_x, c2, nlse_x));
      const float ds_x = p_x * (dp_x - delta_x) * p.scale;
      if (live) {
#pragma unroll
        for (int j = 0; j < 8 * NV; ++j) {
          dk[j] = fmaf(ds_x, f[j], dk[j]);
          dv[j] = fmaf(p_x, g[j], dv[j]);
        }
      }
      if (sub == 0 && x < n) {
        e[x] = p_r;
        e[n + x] = ds_r;
        e[2 * n + x] = ds_x;
        if (t == 0) {
          float* st = stats + ((bh * p.n_qt + x / ATT_BM) * 2) * ATT_BM + x % ATT_BM;
          st[0] = nlse_x;
          st[ATT_BM] = -delta_x * p.scale;
        }
      }
    }
    cp_async_wait<0>();
    __syncthreads();
    // over the eight groups of a warp, then over the warps
#pragma unroll
    for (int j = 0; j < 8 * NV; ++j) {
#pragma unroll
      for (int m = 4; m < 32; m <<= 1) {
        dq[j] += __shfl_xor_sync(0xffffffffu, dq[j], m);
        dk[j] += __shfl_xor_sync(0xffffffffu, dk[j], m);
        dv[j] += __shfl_xor_sync(0xffffffffu, dv[j], m);
      }
      if (lane < 4) {
        const int d = (sub + 4 * (j / 8)) * 8 + j % 8;
        red[warp][0][d] = dq[j];
        red[warp][1][d] = dk[j];
        red[warp][2][d] = dv[j];
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 3 * DP; i += THREADS) {
      const int a = i / DP, d = i - a * DP;
      if (d < p.D) {
        const float s = (red[0][a][d] + red[1][a][d]) + (red[2][a][d] + red[3][a][d]);
        T* dst = a == 0 ? reinterpret_cast<T*>(p.dq) + b * p.sdq[0] + r * p.sdq[1] + h * p.sdq[2]
                        : reinterpret_cast<T*>(a == 1 ? p.dk : p.dv) + b * p.sdkv[0] +
                              r * p.sdkv[1] + h * p.sdkv[2];
        dst[d] = from_f32<T>(s);
      }
    }
    __syncthreads();
  }
}

// dq[b, i, h, :] (strided) = convert(acc[b, i, h, :]) ; acc is contiguous [B*Sq*H, D]
template <typename T>
__global__ void __launch_bounds__(256)
attn_dq_convert_kernel(const float* __restrict__ acc, T* __restrict__ dq, long long rows, int D,
                       int Sq, int H, long long sb, long long ss, long long sh) {
  after_previous();
  const int dv = D / 8;
  const long long total = rows * dv;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const long long row = i / dv;
    const int c = (int)(i - row * dv);
    const int h = (int)(row % H);
    const long long bs = row / H;
    const int si = (int)(bs % Sq);
    const long long b = bs / Sq;
    const float4 a0 = reinterpret_cast<const float4*>(acc + row * D)[2 * c];
    const float4 a1 = reinterpret_cast<const float4*>(acc + row * D)[2 * c + 1];
    uint4 q;
    q.x = pack2<T>(a0.x, a0.y); q.y = pack2<T>(a0.z, a0.w);
    q.z = pack2<T>(a1.x, a1.y); q.w = pack2<T>(a1.z, a1.w);
    reinterpret_cast<uint4*>(dq + b * sb + (long long)si * ss + (long long)h * sh)[c] = q;
  }
}

template <int DP, bool DS_TMEM>
struct BwdCfg {
  static constexpr int NBLK = (DP + 63) / 64;
  static constexpr int TILE = NBLK * ATT_BLK;
  static constexpr bool ALIAS_P = DP > 96;     // P^T in the columns of S^T
  static constexpr bool ALIAS_DQ = DP > 64;    // dQ in the columns of dP^T
  static constexpr int DOST = NBLK == 1 ? 2 : 1;   // dO stages (Q always has two)
  static constexpr int NDS = NBLK == 1 ? 2 : 1;    // dS^T buffers
  static constexpr int DS_BYTES = 2 * ATT_BLK;
  static constexpr int OFF_V = TILE;
  static constexpr int OFF_Q = 2 * TILE;
  static constexpr int OFF_DO = OFF_Q + 2 * TILE;
  static constexpr int OFF_DS = OFF_DO + DOST * TILE;
  static constexpr int OFF_STG = OFF_DS + NDS * DS_BYTES;   // 4 warps x 2 boxes of 4 KB
  static constexpr int OFF_STAT = OFF_STG + 4 * 2 * 4096;   // 2 stages x 1 KB
  static constexpr int OFF_BAR = OFF_STAT + 2 * 1024;
  static constexpr int SMEM = OFF_BAR + 256;
  static constexpr int T_S = 0, T_DP = 128;
  static constexpr int T_P = ALIAS_P ? 0 : 256;
  static constexpr int P_HALF = ALIAS_P ? 64 : 32;   // column distance of P^T's query halves
  static constexpr int T_DV = ALIAS_P ? 256 : 320;
  static constexpr int T_DK = T_DV + DP;
  static constexpr int T_DQ = ALIAS_DQ ? T_DP : T_DK + DP;
  // four warpgroups of 128 registers a thread at launch
  static constexpr int THREADS = 512;
  static constexpr int REGS_SOFTMAX = DS_TMEM ? 160 : 152, REGS_DRAIN = 104;
  static constexpr int REGS_OTHER = DS_TMEM ? 88 : 104;
  static_assert(!(DS_TMEM && ALIAS_DQ), "dS^T and dQ would share columns");
  static_assert(2 * REGS_SOFTMAX + REGS_DRAIN + REGS_OTHER <= 4 * 128, "registers of the block");
  static_assert(SMEM <= 232448, "shared memory per CTA");
  static_assert((ALIAS_DQ ? T_DK : T_DQ) + DP <= 512, "TMEM columns");
};

struct BwdItem {
  int kt, k0, h, b, q_begin, n;    // key tile, its first key, first visible query tile, query tiles
};
// Items of round `r`.  Causal key tiles see fewer queries the later they start: the long ones are
// dealt first (all heads of a key tile next to each other) and every other round runs backwards,
// so that a CTA with a long item in one round gets a short one in the next.  Otherwise the key
// tiles of a head are neighbours, which lets them share its Q / dO in L2.
__device__ __forceinline__ int bwd_index(int r) {
  const int slot = (r & 1) ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x;
  return r * (int)gridDim.x + slot;
}
// In DQ_WHOLE the items are heads and their key tiles rounds of their own.
template <int MODE>
__device__ __forceinline__ int bwd_rounds(const AttnBwdParams& p, int n_items) {
  const int rounds = (n_items + (int)gridDim.x - 1) / (int)gridDim.x;
  return MODE == DQ_WHOLE ? rounds * p.n_kt : rounds;
}
// the item of round `r`; false when this CTA has none
template <int MODE>
__device__ __forceinline__ bool bwd_item(const AttnBwdParams& p, int r, int n_items, BwdItem& it) {
  int kt, bh;
  if (MODE == DQ_WHOLE) {
    const int head = r / p.n_kt;
    kt = r - head * p.n_kt;
    bh = bwd_index(head);
    if (bh >= n_items) return false;
  } else {
    const int w = bwd_index(r);
    if (w >= n_items) return false;
    if (p.causal) { kt = w / (p.B * p.H); bh = w - kt * (p.B * p.H); }
    else { bh = w / p.n_kt; kt = w - bh * p.n_kt; }
  }
  it.kt = kt;
  it.k0 = kt * ATT_BN;
  it.h = bh % p.H;
  it.b = bh / p.H;
  it.q_begin = p.causal ? max(0, it.k0 - (p.Sk - p.Sq)) / ATT_BM : 0;
  it.n = max(0, p.n_qt - it.q_begin);
  return true;
}

// acc[0..31] += w * (columns c0 .. c0 + 31 of a 16-bit row of D values); every lane reads the same row
template <typename T>
__device__ __forceinline__ void axpy_row32(uint32_t (&acc)[32], float w, const T* row, int c0, int D) {
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    if (c0 + v * 8 < D) {
      const uint4 u = __ldg(reinterpret_cast<const uint4*>(row + c0) + v);
      const T* e = reinterpret_cast<const T*>(&u);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        acc[v * 8 + j] = __float_as_uint(fmaf(w, to_f32<T>(e[j]), __uint_as_float(acc[v * 8 + j])));
    }
  }
}

// Probabilities of 32 queries for this thread's key: kept in fp32, packed to 16 bits in the columns
// of P^T.  Queries below `lim` do not see the key.
template <typename T, bool MASKED>
__device__ __forceinline__ void bwd_probs(const uint32_t (&s)[32], float* pr, const float* nlse2,
                                          uint64_t c2v, int lim, uint32_t t_p) {
  uint32_t pk[16];
#pragma unroll
  for (int j = 0; j < 32; j += 4) {
    const float4 l4 = *reinterpret_cast<const float4*>(nlse2 + j);
    float x[4];
    f2_unpack(fma2(f2_pack(__uint_as_float(s[j]), __uint_as_float(s[j + 1])), c2v,
                   f2_pack(l4.x, l4.y)), x[0], x[1]);
    f2_unpack(fma2(f2_pack(__uint_as_float(s[j + 2]), __uint_as_float(s[j + 3])), c2v,
                   f2_pack(l4.z, l4.w)), x[2], x[3]);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float e = exp2f(x[u]);
      pr[j + u] = (MASKED && j + u < lim) ? 0.f : e;
    }
    pk[j / 2] = pack2<T>(pr[j], pr[j + 1]);
    pk[j / 2 + 1] = pack2<T>(pr[j + 2], pr[j + 3]);
  }
  tmem_st16(t_p, pk);
}

// dS^T of the same 32 queries: 16-bit, into this key's row of the swizzled tile from its 16-byte
// chunk `c0` on, and with TMEM also to the columns at `t_ds`, whose dP^T has been read
template <typename T, bool TMEM>
__device__ __forceinline__ void bwd_ds(const uint32_t (&s)[32], const float* pr, const float* ndlt,
                                       uint64_t scv, uint8_t* ds_row, int row, int c0,
                                       uint32_t t_ds) {
  uint32_t pk[16];
#pragma unroll
  for (int j = 0; j < 32; j += 8) {
    uint32_t* o = pk + j / 2;
#pragma unroll
    for (int u = 0; u < 8; u += 4) {
      const float4 d4 = *reinterpret_cast<const float4*>(ndlt + j + u);
      float a, b;
      f2_unpack(mul2(f2_pack(pr[j + u], pr[j + u + 1]),
                     fma2(f2_pack(__uint_as_float(s[j + u]), __uint_as_float(s[j + u + 1])), scv,
                          f2_pack(d4.x, d4.y))), a, b);
      o[u / 2] = pack2<T>(a, b);
      f2_unpack(mul2(f2_pack(pr[j + u + 2], pr[j + u + 3]),
                     fma2(f2_pack(__uint_as_float(s[j + u + 2]), __uint_as_float(s[j + u + 3])), scv,
                          f2_pack(d4.z, d4.w))), a, b);
      o[u / 2 + 1] = pack2<T>(a, b);
    }
    *reinterpret_cast<uint4*>(ds_row + (((c0 + j / 8) ^ (row & 7)) << 4)) =
        make_uint4(o[0], o[1], o[2], o[3]);
  }
  if (TMEM) tmem_st16(t_ds, pk);
}

// DS_TMEM: dK reads dS^T from tensor memory: 256 of the 3100 cycles' worth of shared-memory accesses of a
// tile pair less ([4, 4096, 10, 64] 579 -> 549 us).  dP(i+1) then waits for dK(i), which costs more
// than that where one key tile holds every key ([4, 1024, 20, 64] with 77 keys: 35 -> 37 us).
template <typename T, int DP, int MODE, bool DS_TMEM>
__global__ void __launch_bounds__(BwdCfg<DP, DS_TMEM>::THREADS, 1)
attn_bwd_ws_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                   const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tdo,
                   const __grid_constant__ CUtensorMap tdq, const __grid_constant__ CUtensorMap tdk,
                   const __grid_constant__ CUtensorMap tdv, const AttnBwdParams p,
                   const int n_items) {
  using C = BwdCfg<DP, DS_TMEM>;
  constexpr int NBLK = C::NBLK, TILE = C::TILE;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint64_t* kv_full = bars;          // K and V of the item
  uint64_t* kv_empty = bars + 1;     // every product of the item has completed
  uint64_t* q_full = bars + 2;       // [2] Q tile and its row statistics
  uint64_t* q_empty = bars + 4;      // [2] dK has read Q (1), the softmax warps the statistics (8)
  uint64_t* do_full = bars + 6;      // [2]
  uint64_t* do_empty = bars + 8;     // [2] dV has read dO
  uint64_t* s_full = bars + 10;
  uint64_t* s_empty = bars + 11;     // S^T is in registers (used when P^T has its own columns)
  uint64_t* p_ready = bars + 12;
  uint64_t* dv_done = bars + 13;     // dV(i) has read P^T
  uint64_t* dp_full = bars + 14;
  uint64_t* ds_ready = bars + 15;
  uint64_t* ds_empty = bars + 16;    // [2] dK and dQ have read dS^T
  uint64_t* dq_full = bars + 18;
  uint64_t* dq_empty = bars + 19;
  uint64_t* acc_full = bars + 20;    // dK / dV of the item are complete
  uint64_t* acc_empty = bars + 21;
  uint64_t* dk_done = bars + 22;     // dK(i) has read dS^T from the columns of dP^T (head dim <= 64)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 23);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // the 128-byte swizzle works on absolute shared-memory addresses
  if ((smem_u32(smem) & 1023u) != 0u) {
    if (tid == 0) report(p.status, PF_ERR_BAD_ARG);
    return;
  }
  if (tid == 0) {
    tma_prefetch_desc(&tq); tma_prefetch_desc(&tk); tma_prefetch_desc(&tv);
    tma_prefetch_desc(&tdo); tma_prefetch_desc(&tdq); tma_prefetch_desc(&tdk); tma_prefetch_desc(&tdv);
    for (int i = 0; i < 23; ++i) mbar_init(&bars[i], 1);
    for (int i = 0; i < 2; ++i) mbar_init(&q_empty[i], 1 + 8);
    mbar_init(s_empty, 8);
    mbar_init(p_ready, 8);
    mbar_init(ds_ready, 8);
    mbar_init(dq_empty, 4);
    mbar_init(acc_empty, 4);
    mbar_fence_init();
  }
  if (warp == 13) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_of(tmem_slot);
  after_previous();
  const int shift = p.Sk - p.Sq, rounds = bwd_rounds<MODE>(p, n_items);
  // one split per warpgroup: its four warps execute the same instruction
  if (warp >= 12) {
    regs_dec<C::REGS_OTHER>();
    if (warp == 12) {
      // ---------------------------------------------------------------- TMA producer
      if (elect_one()) {
        uint32_t g = 0, items = 0;
        bool ok = true;
        for (int r = 0; ok && r < rounds; ++r) {
          BwdItem it;
          if (!bwd_item<MODE>(p, r, n_items, it) || it.n == 0) continue;
          for (int i = 0; i < it.n && ok; ++i, ++g) {
            const int q0 = (it.q_begin + i) * ATT_BM, st = g & 1, ds = g % C::DOST;
            ok = mbar_wait(&q_empty[st], ((g >> 1) & 1) ^ 1, p.status, PF_ERR_TIMEOUT_EMPTY);
            if (!ok) break;
            mbar_expect_tx(&q_full[st], TILE + 1024);
#pragma unroll
            for (int c = 0; c < NBLK; ++c)
              tma_load_4d(smem + C::OFF_Q + st * TILE + c * ATT_BLK, &tq, &q_full[st], c * 64, it.h,
                          q0, it.b);
            bulk_load(smem + C::OFF_STAT + st * 1024,
                      p.stats + ((long long)(it.b * p.H + it.h) * p.n_qt + it.q_begin + i) * 256,
                      1024, &q_full[st]);
            if (i == 0) {
              ok = mbar_wait(kv_empty, (items & 1) ^ 1, p.status, PF_ERR_TIMEOUT_EMPTY);
              if (!ok) break;
              mbar_expect_tx(kv_full, 2 * TILE);
#pragma unroll
              for (int c = 0; c < NBLK; ++c) {
                tma_load_4d(smem + c * ATT_BLK, &tk, kv_full, c * 64, it.h, it.k0, it.b);
                tma_load_4d(smem + C::OFF_V + c * ATT_BLK, &tv, kv_full, c * 64, it.h, it.k0, it.b);
              }
            }
            ok = mbar_wait(&do_empty[ds], ((g / C::DOST) & 1) ^ 1, p.status, PF_ERR_TIMEOUT_EMPTY);
            if (!ok) break;
            mbar_expect_tx(&do_full[ds], TILE);
#pragma unroll
            for (int c = 0; c < NBLK; ++c)
              tma_load_4d(smem + C::OFF_DO + ds * TILE + c * ATT_BLK, &tdo, &do_full[ds], c * 64,
                          it.h, q0, it.b);
          }
          ++items;
        }
      }
      __syncwarp();
    } else if (warp == 13) {
      // ---------------------------------------------------------------- MMA issuer
      if (elect_one()) {
        const uint32_t sK = smem_u32(smem), sV = smem_u32(smem + C::OFF_V);
        const uint32_t sQ = smem_u32(smem + C::OFF_Q), sdO = smem_u32(smem + C::OFF_DO);
        const uint32_t sdS = smem_u32(smem + C::OFF_DS);
        const uint32_t id_kd = make_idesc_f16(128, DP, p.fmt, 0, 1);   // P^T dO, dS^T Q
        const uint32_t id_dq = make_idesc_f16(128, DP, p.fmt, 1, 1);   // dS K
        uint32_t g = 0, items = 0;
        bool ok = true;
        auto cols_of = [&](int qt) { return (min(ATT_BM, p.Sq - qt * ATT_BM) + 15) / 16 * 16; };
        // S^T of query tile `qt`, global tile number gg.  The columns of S^T must be free: either
        // the softmax warps hold the previous scores in registers, or (P^T in the same columns) the
        // previous dV has read its probabilities.
        auto issue_s = [&](uint32_t gg, int qt) -> bool {
          const int st = gg & 1;
          if (!mbar_wait(&q_full[st], (gg >> 1) & 1, p.status, PF_ERR_TIMEOUT_FULL)) return false;
          if (gg > 0 && !mbar_wait(C::ALIAS_P ? dv_done : s_empty, (gg - 1) & 1, p.status,
                                   PF_ERR_TIMEOUT_TMEM_EMPTY))
            return false;
          tc_fence_after();
          mma_kk<DP / 16>(tmem + C::T_S, sK, sQ + st * TILE,
                          make_idesc_f16(128, cols_of(qt), p.fmt, 0, 0));
          tc_commit(s_full);
          return true;
        };
        // dP^T; its columns are free once the previous dK has read dS^T there, or when dQ shares them,
        // once that has been drained
        auto issue_dp = [&](uint32_t gg, int qt) -> bool {
          const int st = gg % C::DOST;
          if (!mbar_wait(&do_full[st], (gg / C::DOST) & 1, p.status, PF_ERR_TIMEOUT_FULL))
            return false;
          if ((C::ALIAS_DQ || DS_TMEM) && gg > 0 &&
              !mbar_wait(C::ALIAS_DQ ? dq_empty : dk_done, (gg - 1) & 1, p.status,
                         PF_ERR_TIMEOUT_TMEM_EMPTY))
            return false;
          tc_fence_after();
          mma_kk<DP / 16>(tmem + C::T_DP, sV, sdO + st * TILE,
                          make_idesc_f16(128, cols_of(qt), p.fmt, 0, 0));
          tc_commit(dp_full);
          return true;
        };
        for (int r = 0; ok && r < rounds; ++r) {
          BwdItem it;
          if (!bwd_item<MODE>(p, r, n_items, it) || it.n == 0) continue;
          const int k_steps = (min(ATT_BN, p.Sk - it.k0) + 15) / 16;
          ok = mbar_wait(kv_full, items & 1, p.status, PF_ERR_TIMEOUT_FULL) &&
               issue_s(g, it.q_begin) && issue_dp(g, it.q_begin);
          for (int i = 0; i < it.n && ok; ++i, ++g) {
            const int qt = it.q_begin + i, st = g & 1, dst = g % C::DOST, dsb = g % C::NDS;
            const int q_steps = cols_of(qt) / 16;
            const bool more = i + 1 < it.n;
            if (!C::ALIAS_P && more && !(ok = issue_s(g + 1, qt + 1))) break;
            // ---- dV
            ok = mbar_wait(p_ready, g & 1, p.status, PF_ERR_TIMEOUT_FULL);
            if (ok && i == 0)
              ok = mbar_wait(acc_empty, (items & 1) ^ 1, p.status, PF_ERR_TIMEOUT_TMEM_EMPTY);
            if (!ok) break;
            tc_fence_after();
            mma_t_mn(tmem + C::T_DV, tmem + C::T_P, C::P_HALF, sdO + dst * TILE, id_kd, i > 0, q_steps);
            tc_commit(&do_empty[dst]);
            tc_commit(dv_done);
            if (C::ALIAS_P && more && !(ok = issue_s(g + 1, qt + 1))) break;
            ok = mbar_wait(ds_ready, g & 1, p.status, PF_ERR_TIMEOUT_FULL);
            if (!ok) break;
            const uint32_t ds_tile = sdS + dsb * C::DS_BYTES;
            auto issue_dk = [&]() {
              tc_fence_after();
              if (DS_TMEM)
                mma_t_mn(tmem + C::T_DK, tmem + C::T_DP, 64, sQ + st * TILE, id_kd, i > 0, q_steps);
              else
                mma_k_mn(tmem + C::T_DK, ds_tile, sQ + st * TILE, id_kd, i > 0, q_steps);
              tc_commit(&q_empty[st]);
              if (DS_TMEM) tc_commit(dk_done);
            };
            auto issue_dq = [&]() {
              tc_fence_after();
              mma_mn_mn(tmem + C::T_DQ, ds_tile, sK, id_dq, k_steps);
              tc_commit(dq_full);
            };
            if (C::ALIAS_DQ) {
              issue_dq();
              issue_dk();
              tc_commit(&ds_empty[dsb]);
              if (more && !(ok = issue_dp(g + 1, qt + 1))) break;
            } else {
              if (!DS_TMEM && more && !(ok = issue_dp(g + 1, qt + 1))) break;
              issue_dk();
              if (g > 0) ok = mbar_wait(dq_empty, (g - 1) & 1, p.status, PF_ERR_TIMEOUT_TMEM_EMPTY);
              if (!ok) break;
              issue_dq();
              tc_commit(&ds_empty[dsb]);
              if (DS_TMEM && more && !(ok = issue_dp(g + 1, qt + 1))) break;
            }
            if (!more) { tc_commit(acc_full); tc_commit(kv_empty); }
          }
          ++items;
        }
      }
      __syncwarp();
    }
  } else if (warp >= 8) {
    // ---------------------------------------------------------------- drain (4 warps)
    regs_dec<C::REGS_DRAIN>();
    const int quad = warp & 3;
    const uint32_t lane_off = uint32_t(quad * 32) << 16;
    uint8_t* boxes = smem + C::OFF_STG + quad * 8192;
    const int n_pad = p.n_qt * ATT_BM;
    float4* part = p.part + (long long)blockIdx.x * n_pad * (DP / 4);
    uint32_t g = 0, items = 0, box = 0;
    bool ok = true;
    // two boxes per warp: the store that last used this one must have read it
    auto next_box = [&]() -> uint8_t* {
      if (lane == 0 && box >= 2) tma_store_wait_read_but_one();
      __syncwarp();
      return boxes + (box++ & 1) * 4096;
    };
    for (int r = 0; ok && r < rounds; ++r) {
      BwdItem it;
      if (!bwd_item<MODE>(p, r, n_items, it)) continue;
      const int kj = it.k0 + quad * 32 + lane;
      const long long off_kv = (long long)it.b * p.sdkv[0] + (long long)kj * p.sdkv[1] +
                               (long long)it.h * p.sdkv[2];
      T* dkp = reinterpret_cast<T*>(p.dk) + off_kv;
      T* dvp = reinterpret_cast<T*>(p.dv) + off_kv;
      if (it.n == 0) {             // no query sees this key tile: its gradients are zero
        if (kj < p.Sk)
          for (int c = 0; c < p.D / 8; ++c) {
            reinterpret_cast<uint4*>(dkp)[c] = make_uint4(0, 0, 0, 0);
            reinterpret_cast<uint4*>(dvp)[c] = make_uint4(0, 0, 0, 0);
          }
        continue;
      }
      const float* edge = p.edge + (long long)(it.b * p.H + it.h) * p.left * 3 * n_pad;
      for (int i = 0; i < it.n && ok; ++i, ++g) {
        const int q0 = (it.q_begin + i) * ATT_BM + quad * 32;   // first query row of this warp
        // DQ_WHOLE: the last key tile that this query tile sees
        const int last_kt =
            p.causal ? min(p.n_kt - 1, ((it.q_begin + i + 1) * ATT_BM - 1 + shift) / ATT_BN) : p.n_kt - 1;
        ok = mbar_wait(dq_full, g & 1, p.status, PF_ERR_TIMEOUT_TMEM_FULL);
        if (!ok) break;
        tc_fence_after();
        // two chunks of 32 columns at a time: the columns of dQ are free as soon as the last pair is
        // in registers, whatever the boxes wait for
#pragma unroll
        for (int c0 = 0; c0 < DP / 32; c0 += 2) {
          uint32_t raw[2][32];
          tmem_ld32(tmem + C::T_DQ + lane_off + c0 * 32, raw[0]);
          if (c0 + 1 < DP / 32) tmem_ld32(tmem + C::T_DQ + lane_off + c0 * 32 + 32, raw[1]);
          tmem_ld_wait_for(raw[0]);
          if (c0 + 1 < DP / 32) tmem_ld_wait_for(raw[1]);
          if (c0 + 2 >= DP / 32) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(dq_empty);
          }
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int c = c0 + u;
            if (c >= DP / 32) continue;
            if (MODE == DQ_WHOLE) {
              const int qi = q0 + lane;
              float4* sum = part + ((it.q_begin + i) * (DP / 4) + c * 8) * ATT_BM + quad * 32 + lane;
              if (it.kt > 0) {
#pragma unroll
                for (int v = 0; v < 8; ++v) {
                  const float4 s = sum[v * ATT_BM];
                  raw[u][v * 4] = __float_as_uint(__uint_as_float(raw[u][v * 4]) + s.x);
                  raw[u][v * 4 + 1] = __float_as_uint(__uint_as_float(raw[u][v * 4 + 1]) + s.y);
                  raw[u][v * 4 + 2] = __float_as_uint(__uint_as_float(raw[u][v * 4 + 2]) + s.z);
                  raw[u][v * 4 + 3] = __float_as_uint(__uint_as_float(raw[u][v * 4 + 3]) + s.w);
                }
              }
              if (it.kt < last_kt) {
#pragma unroll
                for (int v = 0; v < 8; ++v)
                  sum[v * ATT_BM] = make_float4(
                      __uint_as_float(raw[u][v * 4]), __uint_as_float(raw[u][v * 4 + 1]),
                      __uint_as_float(raw[u][v * 4 + 2]), __uint_as_float(raw[u][v * 4 + 3]));
                continue;
              }
              for (int t = 0; t < p.left; ++t)         // the leftover keys' part
                axpy_row32<T>(raw[u], edge[(t * 3 + 2) * n_pad + qi],
                              reinterpret_cast<const T*>(p.k) + (long long)it.b * p.sk[0] +
                                  (long long)(p.Sk + t) * p.sk[1] + (long long)it.h * p.sk[2],
                              c * 32, p.D);
            }
            if (MODE == DQ_TILE) {
              if (q0 + lane < p.Sq) {
                T* dst = reinterpret_cast<T*>(p.dq) + (long long)it.b * p.sdq[0] +
                         (long long)(q0 + lane) * p.sdq[1] + (long long)it.h * p.sdq[2] + c * 32;
#pragma unroll
                for (int v = 0; v < 4; ++v)
                  if (c * 32 + v * 8 < p.D) reinterpret_cast<uint4*>(dst)[v] = pack8<T>(raw[u] + v * 8);
              }
              continue;
            }
            uint8_t* bx = next_box();
            if (MODE == DQ_SUMS) {
#pragma unroll
              for (int v = 0; v < 8; ++v)
                *reinterpret_cast<uint4*>(bx + lane * 128 + ((v ^ (lane & 7)) << 4)) = make_uint4(
                    raw[u][v * 4], raw[u][v * 4 + 1], raw[u][v * 4 + 2], raw[u][v * 4 + 3]);
            } else {
              box_row16<T>(bx, lane, raw[u]);
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) {
              // rows beyond the last query / columns beyond D are clipped by the TMA itself
              if (q0 < p.Sq) {
                if (MODE == DQ_SUMS) tma_reduce_add_4d(&tdq, bx, c * 32, it.h, q0, it.b);
                else tma_store_4d(&tdq, bx, c * 32, it.h, q0, it.b);
              }
              tma_store_commit();
            }
          }
        }
      }
      if (!ok) break;
      ok = mbar_wait(acc_full, items & 1, p.status, PF_ERR_TIMEOUT_TMEM_FULL);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < DP / 32; ++c) {
        uint32_t rk[32], rv[32];
        tmem_ld32(tmem + C::T_DK + lane_off + c * 32, rk);
        tmem_ld32(tmem + C::T_DV + lane_off + c * 32, rv);
        tmem_ld_wait_for(rk);
        tmem_ld_wait_for(rv);
        if (c == DP / 32 - 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc_empty);
        }
        if constexpr (MODE == DQ_SUMS || MODE == DQ_TILE) {
          if (kj < p.Sk) {
#pragma unroll
            for (int v = 0; v < 4; ++v)
              if (c * 32 + v * 8 < p.D) {
                reinterpret_cast<uint4*>(dkp)[c * 4 + v] = pack8<T>(rk + v * 8);
                reinterpret_cast<uint4*>(dvp)[c * 4 + v] = pack8<T>(rv + v * 8);
              }
          }
        } else {
          // A row's 16 bytes per thread take some 6800 cycles to leave at head dim 88, more than the products
          // of a short item: they go through boxes.  Among the boxes of DQ_SUMS they would only wait
          // ([12, 513, 25, 64] 181 -> 200 us).
          for (int t = 0; t < p.left; ++t) {       // the leftover queries' part
            const long long r = p.Sq + t;
            axpy_row32<T>(rk, edge[(t * 3 + 1) * n_pad + kj],
                          reinterpret_cast<const T*>(p.q) + (long long)it.b * p.sq[0] + r * p.sq[1] +
                              (long long)it.h * p.sq[2],
                          c * 32, p.D);
            axpy_row32<T>(rv, edge[t * 3 * n_pad + kj],
                          reinterpret_cast<const T*>(p.dout) +
                              (((long long)it.b * (p.Sq + p.left) + r) * p.H + it.h) * p.D,
                          c * 32, p.D);
          }
          uint8_t* bx = next_box();                // half a box each
          box_row16<T>(bx, lane, rk);
          box_row16<T>(bx + 2048, lane, rv);
          fence_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (it.k0 + quad * 32 < p.Sk) {
              tma_store_4d(&tdk, bx, c * 32, it.h, it.k0 + quad * 32, it.b);
              tma_store_4d(&tdv, bx + 2048, c * 32, it.h, it.k0 + quad * 32, it.b);
            }
            tma_store_commit();
          }
        }
      }
      ++items;
    }
    if (lane == 0) tma_store_wait_all();
  } else {
    // ---------------------------------------------------------------- softmax side (8 warps)
    regs_inc<C::REGS_SOFTMAX>();
    const int quad = warp & 3, half = warp >> 2;
    const int row = quad * 32 + lane;
    const uint32_t lane_off = uint32_t(quad * 32) << 16;
    const float c2 = p.scale * LOG2E;
    const uint64_t c2v = f2_pack(c2, c2), scv = f2_pack(p.scale, p.scale);
    uint32_t g = 0;
    bool ok = true;
    for (int r = 0; ok && r < rounds; ++r) {
      BwdItem it;
      if (!bwd_item<MODE>(p, r, n_items, it)) continue;
      const bool ragged = it.k0 + ATT_BN > p.Sk;
      const int kj = it.k0 + row;
      // a warp all of whose keys lie beyond the last one (rounded to the reduction steps of dQ)
      // has nothing to contribute: those rows of dK / dV are not stored, dQ does not read them
      const bool warp_live = it.k0 + quad * 32 < (p.Sk + 15) / 16 * 16;
      for (int i = 0; i < it.n && ok; ++i, ++g) {
        const int q0 = (it.q_begin + i) * ATT_BM, st = g & 1, dsb = g % C::NDS;
        const int cols = (min(ATT_BM, p.Sq - q0) + 15) / 16 * 16;
        const float* nlse2 =
            reinterpret_cast<const float*>(smem + C::OFF_STAT + st * 1024) + half * 64;
        const float* ndlt = nlse2 + 128;
        const bool masked = ragged || (p.causal && it.k0 + ATT_BN - 1 > q0 + shift);
        // queries of this half below `lim` do not see the key of this row
        int lim = p.causal ? kj - shift - q0 - half * 64 : -1;
        if (kj >= p.Sk) lim = ATT_BM;
        // A wait that is satisfied still takes some 130 cycles: all barriers are looked at together
        // first.  (The columns of P^T must have been read by dV of the previous tile.)
        const bool chk_dv = !C::ALIAS_P && g > 0;
        const bool seen_q = mbar_test(&q_full[st], (g >> 1) & 1), seen_s = mbar_test(s_full, g & 1);
        const bool seen_v = !chk_dv || mbar_test(dv_done, (g - 1) & 1);
        if (!(seen_q && seen_s && seen_v)) {
          ok = mbar_wait(&q_full[st], (g >> 1) & 1, p.status, PF_ERR_TIMEOUT_FULL) &&
               mbar_wait(s_full, g & 1, p.status, PF_ERR_TIMEOUT_TMEM_FULL);
          if (chk_dv && ok) ok = mbar_wait(dv_done, (g - 1) & 1, p.status, PF_ERR_TIMEOUT_TMEM_EMPTY);
        }
        if (!ok) break;
        tc_fence_after();
        float pr[64];
        const uint32_t t_p = tmem + C::T_P + lane_off + half * C::P_HALF;
        const uint32_t t_s = tmem + C::T_S + lane_off + half * 64;
        const uint32_t t_dp = tmem + C::T_DP + lane_off + half * 64;
        // the usual tile: nothing masked, all of this warp's columns and rows exist
        const bool whole = warp_live && !masked && half * 64 + 64 <= cols;
        if (whole) {
          uint32_t s0[32], s1[32];
          tmem_ld32(t_s, s0);
          tmem_ld_wait_for(s0);
          tmem_ld32(t_s + 32, s1);          // travels while the first half is worked on
          bwd_probs<T, false>(s0, pr, nlse2, c2v, 0, t_p);
          tmem_ld_wait_for(s1);
          if (!C::ALIAS_P) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(s_empty);
          }
          bwd_probs<T, false>(s1, pr + 32, nlse2 + 32, c2v, 0, t_p + 16);
        } else {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const bool work = warp_live && half * 64 + c * 32 < cols;     // warp-uniform
            uint32_t s[32];
            if (work) {
              tmem_ld32(t_s + c * 32, s);
              tmem_ld_wait_for(s);
            }
            if (!C::ALIAS_P && c == 1) {
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(s_empty);
            }
            if (work)
              bwd_probs<T, true>(s, pr + c * 32, nlse2 + c * 32, c2v, lim - c * 32, t_p + c * 16);
          }
        }
        const bool seen_dp = mbar_test(dp_full, g & 1);
        const bool seen_ds = mbar_test(&ds_empty[dsb], ((g / C::NDS) & 1) ^ 1);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_ready);
        // ---- dS^T
        if (!(seen_dp && seen_ds))
          ok = mbar_wait(dp_full, g & 1, p.status, PF_ERR_TIMEOUT_TMEM_FULL) &&
               mbar_wait(&ds_empty[dsb], ((g / C::NDS) & 1) ^ 1, p.status, PF_ERR_TIMEOUT_EMPTY);
        if (!ok) break;
        tc_fence_after();
        uint8_t* ds_row = smem + C::OFF_DS + dsb * C::DS_BYTES + half * ATT_BLK + row * 128;
        if (whole) {
          uint32_t s0[32], s1[32];
          tmem_ld32(t_dp, s0);
          tmem_ld_wait_for(s0);
          tmem_ld32(t_dp + 32, s1);
          bwd_ds<T, DS_TMEM>(s0, pr, ndlt, scv, ds_row, row, 0, t_dp);
          tmem_ld_wait_for(s1);
          bwd_ds<T, DS_TMEM>(s1, pr + 32, ndlt + 32, scv, ds_row, row, 4, t_dp + 16);
        } else {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            if (warp_live && half * 64 + c * 32 < cols) {
              uint32_t s[32];
              tmem_ld32(t_dp + c * 32, s);
              tmem_ld_wait_for(s);
              bwd_ds<T, DS_TMEM>(s, pr + c * 32, ndlt + c * 32, scv, ds_row, row, c * 4,
                                 t_dp + c * 16);
            }
          }
        }
        fence_async_smem();
        if (DS_TMEM) tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) { mbar_arrive(ds_ready); mbar_arrive(&q_empty[st]); }
      }
    }
  }

  // teardown: every role reaches this point (all waits are bounded)
  tc_fence_before();
  __syncthreads();
  if (warp == 13) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// ------------------------------------------------------------------------------- host side
// fp32 [B, Sq, H, D] contiguous sums; box = 32 x 1 x 32 x 1 in the 128-byte swizzle
static int make_tmap_dq(CUtensorMap* map, const void* base, int B, int S, int H, int D) {
  EncodeTiledFn enc = attn_get_encode();
  if (!enc) return -100;
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)S, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)D * 4, (cuuint64_t)H * D * 4, (cuuint64_t)S * H * D * 4};
  cuuint32_t box[4] = {32, 1, 32, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<void*>(base), dims, strides,
                   box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -(1000 + (int)r);
}

template <typename T, int DP>
static int launch_bwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                      const CUtensorMap& tdo, const CUtensorMap& tdq, const CUtensorMap& tdk,
                      const CUtensorMap& tdv, const AttnBwdParams& p, int mode, cudaStream_t st) {
  const int n_items = (mode == DQ_WHOLE ? 1 : p.n_kt) * p.H * p.B, sms = attn_sm_count();
  const int grid = n_items < sms ? n_items : sms;
  auto run = [&](auto m, auto ds_tmem) -> int {
    using C = BwdCfg<DP, decltype(ds_tmem)::value>;
    auto kern = attn_bwd_ws_kernel<T, DP, decltype(m)::value, decltype(ds_tmem)::value>;
    static bool done[64] = {};       // one per instantiation of this lambda
    const int r = set_smem(kern, C::SMEM, done);
    if (r) return r;
    after(kern, grid, C::THREADS, C::SMEM, st)(tq, tk, tv, tdo, tdq, tdk, tdv, p, n_items);
    PF_CHECK_LAUNCH();
    return 0;
  };
  std::integral_constant<int, DQ_SUMS> sums;
  std::integral_constant<int, DQ_DIRECT> direct;
  std::integral_constant<int, DQ_WHOLE> whole;
  constexpr std::bool_constant<(DP <= 64)> in_tmem{};
  constexpr std::false_type in_smem{};
  if (mode == DQ_SUMS) return run(sums, in_tmem);
  if (mode == DQ_DIRECT) return run(direct, in_smem);
  if (mode == DQ_TILE) return run(std::integral_constant<int, DQ_TILE>(), in_smem);
  return p.n_kt > 1 ? run(whole, in_tmem) : run(whole, in_smem);
}

template <typename T, int DP>
static int launch_edge(const AttnBwdParams& p, const void* v, const void* out, const void* lse, void* stats,
                       const long long* sv, cudaStream_t st) {
  using C = EdgeCfg<DP>;
  static bool done[2][64] = {};
  const bool many = C::CTAS_MANY > C::CTAS && (long long)p.H * p.B > (long long)C::CTAS * attn_sm_count();
  auto kern = many ? attn_bwd_edge_kernel<T, DP, C::CTAS_MANY> : attn_bwd_edge_kernel<T, DP, C::CTAS>;
  const int r = set_smem(kern, C::SMEM, done[many]);
  if (r) return r;
  after(kern, dim3(p.H, p.B), C::THREADS, C::SMEM, st)(
      p, (const T*)v, (const T*)out, (const float*)lse, (float*)stats, sv[0], sv[1], sv[2]);
  PF_CHECK_LAUNCH();
  return 0;
}

// one key tile that every query tile visits: its dQ tiles need no summation
static bool bwd_direct(int Sq, int Sk, int causal) {
  return Sk <= ATT_BN && (!causal || Sk >= Sq);
}

struct BwdPlan {
  int mode, left, n_kt, n_qt;
  long long part, edge;               // floats of scratch: dQ so far (or the fp32 sums), leftover weights
};
// Heads are taken whole where that takes no more rounds of key tiles than dealing the key tiles one by one, and
// while a head's sums of dQ (512 bytes per query tile and column) are small: a CTA reads and writes them once
// per key tile, and past 200 KB, or 320 with two key tiles, that costs more than adding in memory.  us, dealt and
// whole, 144 heads: head dim 64, 256 tokens 25.8 21.8, 768 99.9 99.8, 1024 156 176, 1024 queries of 200 keys 1.17
// times as fast whole; head dim 128, 256 tokens 37.5 32.3, 384 59.8 58.9, 512 86.8 101, 1024 243 409.
// Under a causal mask a head visits half the pairs of tiles and whole heads gain for longer (head dim 128, 294
// heads of 512 168 126, of 1024 1.07 times), but dealing, longest first, fills a single round better (head dim
// 128, 144 heads of 640 1.05 times, of 768 0.98; head dim 32, 132 heads of 898 0.95), and a last tile of a few
// rows costs it next to nothing (head dim 88, 432 heads of 898 0.92, of 1024 1.03).
static bool whole_pays(int causal, int dp, int Sq, int n_kt, long long heads, long long sms) {
  const long long rounds = (heads + sms - 1) / sms, apart = (heads * n_kt + sms - 1) / sms;
  const int n_qt = (Sq + ATT_BM - 1) / ATT_BM, size = n_qt * dp;
  if (n_qt > BWD_WHOLE_TILES || rounds * n_kt > apart) return false;
  if (!causal)
    return size <= (n_kt == 2 ? 640 : n_kt == 3 && dp <= 96 ? 512 : n_kt <= 4 || dp <= 96 ? 384 : 256);
  const bool few_rows = Sq % ATT_BM > 0 && Sq % ATT_BM <= 32;
  if (rounds == 1) return size <= (few_rows ? 512 : 640) && (n_qt <= 6 || 20 * heads >= 19 * sms);
  return dp <= 64 || !few_rows || size <= 640;
}
// Whether the leftover tokens are taken out of the tiles, which saves a key tile and a query tile per head and
// costs a pass over the head per token.  `rounds` are of heads, of n_kt key tiles without the leftovers.  The pass
// takes the place of the one that clears and of the one that converts, so that one token pays without a saved
// round up to head dim 64, and for a fifth of the rounds at 96 and a quarter at 128; two tokens pay for nearly
// half of them at head dim 64, or for a quarter where the tiles cannot be taken whole, and want several rounds of
// heads over which the pass spreads.  us, dealt, whole and so: [10, 257, 16, 64] 46.9 54.1 42.5, [24, 257, 16, 88]
// 114.7 113.7 103.4, [10, 257, 16, 88] 60.1 73.6 67.7, [24, 257, 16, 128] 129.5 127.4 130.1, [3, 129, 19, 64] 13.2
// 15.0 14.4, [3, 130, 19, 64] 13.3 15.1 20.0, [24, 258, 16, 64] 90.8 87.2 86.0, [16, 386, 19, 32] 106 111 92.5.
static bool leftover_pays(int left, int dp, int n_qt, int n_kt, long long rounds, long long apart) {
  const long long r = rounds * n_kt;
  if (n_qt > BWD_WHOLE_TILES || n_qt * dp > 384) return false;
  if (left == 1) {
    const int percent = dp <= 64 ? 100 : dp <= 96 ? 122 : 133;
    return r * percent <= apart * 100 && (r < apart || n_kt > 1);
  }
  if (dp <= 32) return r < apart || (r == apart && rounds > 1);
  return rounds > 1 && (8 * r <= 5 * apart || (n_kt > 1 && 4 * r <= 3 * apart && rounds * (n_kt + 1) > apart));
}
static BwdPlan bwd_plan(int B, int H, int Sq, int Sk, int D, int causal) {
  const long long heads = (long long)B * H, sms = attn_sm_count();
  auto tiles = [](int n) { return (n + ATT_BN - 1) / ATT_BN; };
  BwdPlan g = {bwd_direct(Sq, Sk, causal) ? DQ_DIRECT : DQ_SUMS, 0, tiles(Sk), tiles(Sq), 0, 0};
  if (g.mode == DQ_DIRECT && g.n_qt == 1 && Sq + 2 * Sk <= (heads > sms ? BWD_TILE_ROWS : BWD_TILE_ROWS_ONCE))
    g.mode = DQ_TILE;
  const int dp = (D + 31) / 32 * 32;
  const long long rounds = (heads + sms - 1) / sms, apart = (heads * g.n_kt + sms - 1) / sms;
  if (g.mode == DQ_SUMS && (!causal || Sk >= Sq)) {
    const int left = !causal && Sq == Sk && Sq > ATT_BM ? Sq % ATT_BM : 0;
    if (left > 0 && left <= (D > 64 ? 1 : BWD_LEFT_MAX) &&
        leftover_pays(left, dp, g.n_qt - 1, g.n_kt - 1, rounds, apart)) {
      g.mode = DQ_WHOLE;
      g.left = left;
      --g.n_kt;
      --g.n_qt;
    } else if (whole_pays(causal, dp, Sq, g.n_kt, heads, sms)) {
      g.mode = DQ_WHOLE;
    }
  }
  if (g.mode == DQ_WHOLE) {
    g.part = (heads < sms ? heads : sms) * g.n_qt * ATT_BM * dp;
    g.edge = heads * g.left * 3 * g.n_qt * ATT_BM;
  } else if (g.mode == DQ_SUMS) {
    g.part = heads * Sq * D;
  }
  return g;
}

}  // namespace pf

using namespace pf;

// KiB of scratch that pf_attn_bwd needs on the current device (0: none)
PF_API int pf_attn_bwd_scratch(int B, int H, int Sq, int Sk, int D, int causal) {
  const BwdPlan g = bwd_plan(B, H, Sq, Sk, D, causal);
  return (int)((g.part + g.edge + 255) / 256);
}

// dout / out: [B, Sq, H, D] contiguous.  stats: fp32 scratch [B, H, ceil(Sq / 128), 256]; scratch: of
// pf_attn_bwd_scratch KiB; both 16-byte aligned.
PF_API int pf_attn_bwd(const void* dout, const void* q, const void* k, const void* v,
                       const void* out, const void* lse, void* stats, void* scratch, void* dq,
                       void* dk, void* dv, int B, int H, int Sq, int Sk, int D,
                       const long long* sq, const long long* sk, const long long* sv,
                       const long long* sdq, const long long* sdkv, int causal,
                       float scale, int dtype, int* status, int sm_count, void* stream) {
  if (dtype != PF_F16 && dtype != PF_BF16) return -1;
  if (D % 8 || D > 128) return -3;
  const BwdPlan plan = bwd_plan(B, H, Sq, Sk, D, causal);
  if (!strides_ok(q, sq[0], sq[1], sq[2]) || !strides_ok(k, sk[0], sk[1], sk[2]) ||
      !strides_ok(v, sv[0], sv[1], sv[2]) || (reinterpret_cast<uintptr_t>(dout) & 15) ||
      (reinterpret_cast<uintptr_t>(out) & 15) || (reinterpret_cast<uintptr_t>(stats) & 15) ||
      (plan.part && (!scratch || (reinterpret_cast<uintptr_t>(scratch) & 15))) ||
      !strides_ok(dq, sdq[0], sdq[1], sdq[2]) || !strides_ok(dk, sdkv[0], sdkv[1], sdkv[2]) ||
      !strides_ok(dv, sdkv[0], sdkv[1], sdkv[2]))
    return -2;
  const int fmt = dtype == PF_BF16;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  AttnBwdParams p = {};
  // with leftover rows the tensor-core kernel sees the tokens before them
  p.B = B; p.H = H; p.Sq = Sq - plan.left; p.Sk = Sk - plan.left; p.D = D; p.causal = causal;
  p.scale = scale; p.fmt = fmt; p.stats = (const float*)stats; p.dq = dq; p.dk = dk; p.dv = dv;
  p.status = status; p.n_kt = plan.n_kt; p.n_qt = plan.n_qt;
  p.part = (float4*)scratch; p.left = plan.left; p.edge = (float*)scratch + plan.part;
  p.q = q; p.k = k; p.dout = dout;
  for (int i = 0; i < 3; ++i) {
    p.sdq[i] = sdq[i]; p.sdkv[i] = sdkv[i]; p.sq[i] = sq[i]; p.sk[i] = sk[i];
  }
  CUtensorMap tq, tk, tv, tdo, tdq, tdk, tdv;
  int r;
  if ((r = make_tmap_bshd(&tq, q, fmt, B, Sq, H, D, sq[0], sq[1], sq[2]))) return r;
  if ((r = make_tmap_bshd(&tk, k, fmt, B, Sk, H, D, sk[0], sk[1], sk[2]))) return r;
  if ((r = make_tmap_bshd(&tv, v, fmt, B, Sk, H, D, sv[0], sv[1], sv[2]))) return r;
  if ((r = make_tmap_bshd(&tdo, dout, fmt, B, Sq, H, D, (long long)Sq * H * D, (long long)H * D,
                          D)))
    return r;
  float* sums = plan.mode == DQ_SUMS ? (float*)scratch : nullptr;
  if ((r = sums ? make_tmap_dq(&tdq, sums, B, Sq, H, D)
                : make_tmap_box32(&tdq, dq, fmt, B, Sq, H, D, sdq)) ||
      (r = make_tmap_box32(&tdk, dk, fmt, B, Sk, H, D, sdkv)) ||
      (r = make_tmap_box32(&tdv, dv, fmt, B, Sk, H, D, sdkv)))
    return r;
  if (plan.left) {
    auto run = [&]() -> int { PF_ATTN_DISPATCH(launch_edge, p, v, out, lse, stats, sv, st); };
    if ((r = run())) return r;
  } else {
    const long long pad_rows = (long long)B * p.n_qt * ATT_BM * H;
    const unsigned prep = (unsigned)((pad_rows + 31) / 32);
    if (dtype == PF_F16)
      after(attn_bwd_prep_kernel<__half>, prep, 256, 0, st)((const __half*)dout, (const __half*)out,
          (const float*)lse, (float*)stats, sums, B, Sq, H, D, p.n_qt, scale);
    else
      after(attn_bwd_prep_kernel<__nv_bfloat16>, prep, 256, 0, st)((const __nv_bfloat16*)dout,
          (const __nv_bfloat16*)out, (const float*)lse, (float*)stats, sums, B, Sq, H, D, p.n_qt,
          scale);
  }
  PF_CHECK_LAUNCH();
  {
    auto run = [&]() -> int { PF_ATTN_DISPATCH(launch_bwd, tq, tk, tv, tdo, tdq, tdk, tdv, p, plan.mode, st); };
    if ((r = run())) return r;
  }
  if (!sums) return 0;
  const long long rows = (long long)B * Sq * H, n = rows * (D / 8);
  long long blocks = (n + 255) / 256;
  const long long cap = (long long)(sm_count > 0 ? sm_count : 148) * 8;
  if (blocks > cap) blocks = cap;
  if (dtype == PF_F16)
    after(attn_dq_convert_kernel<__half>, (unsigned)blocks, 256, 0, st)(
        sums, (__half*)dq, rows, D, Sq, H, sdq[0], sdq[1], sdq[2]);
  else
    after(attn_dq_convert_kernel<__nv_bfloat16>, (unsigned)blocks, 256, 0, st)(
        sums, (__nv_bfloat16*)dq, rows, D, Sq, H, sdq[0], sdq[1], sdq[2]);
  PF_CHECK_LAUNCH();
  return 0;
}
