// Flash attention forward for sm_100a on tcgen05 tensor cores (the backward: attn_bwd_sm100.cu).
//
// Layout: q [B, Sq, H, D], k/v [B, Sk, H, D] with arbitrary (16-byte aligned) batch / sequence /
// head strides and a unit inner stride, so the three slices of a fused QKV projection are
// consumed in place through 4-D TMA tensor maps.  Head dims up to 128, any multiple of 8
// (88 for ViT-g/14 runs as 96 with zero-filled tails: the tensor map's inner extent is D, so
// the tail of the last 64-element block is filled with zeros by TMA, never with the next head).
//
// A persistent kernel, one CTA per SM, walks over items of up to 256 query rows of one (head,
// batch): two query tiles of 128 that share every K / V tile it loads (or, where pairs would leave
// SMs idle, one tile whose keys are shared out: see FwdItem).  Its warps:
//   warps 0-3 / 4-7   softmax of side 0 / 1, thread <-> query row <-> TMEM lane
//   warp 8            TMA producer (K and V rings; runs ahead, across item boundaries too)
//   warp 9            MMA issuer (warp 10: of side 1, where each has its own), TMEM owner
//   warp 11           idle
// Per query tile t and key tile j:
//     S_t = Q_t K_j^T   tcgen05.mma, shared memory x shared memory -> TMEM
//     online softmax    S_t read once into registers, base-2 exponent, running maximum and sum
//     P_t -> TMEM       16-bit, read by the next product as its A operand; P never touches
//                       shared memory
//     O_t += P_t V_j    accumulated in TMEM and rescaled there only when the row maximum grew by
//                       more than 2^8 since it was last set (P stays below 2^8, which both 16-bit
//                       formats hold, and most tiles need no rescaling)
// What bounds it: 16384 exponentials per tile, 1024 cycles of the special-function units, against
// 8 x head dim cycles of tensor core (512 at head dim 64; at 128 both take 1024).  Two tiles in
// flight keep one tile's products under the other's exponentials.
// Measured (B200, CUDA events, cold L2), against one query tile per CTA with P in shared
// memory: [4, 4096, 10, 64] 402 -> 236 us, causal [1, 2048, 32, 128] 87 -> 48, causal [6, 1782, 21, 32]
// 200 -> 101, 77 keys [4, 1024, 20, 64] 32 -> 17.7, [24, 257, 16, 88] 62 -> 39.  Steps on the way at
// [4, 4096, 10, 64]: 346 with two query tiles per CTA, 305 with one elected thread issuing the products,
// 292 with the maximum found in the pass over the exponentials, 273 with the pairs beyond whole rounds
// split, 266 with O leaving through boxes, 249 with an issuing thread per query tile, 236 with the split
// pairs' launch beside the other.  The two sides
// of a CTA run in step, so that the 1000 of a step's 3100 cycles in which a side waits, loads and
// stores find nobody at the exponentials: held half a step apart, a step takes 2770, but they drift back.
// TMEM (512 columns): S_0, S_1 128 each, O_0, O_1 one head dim each.  Up to head dim 64 P_0, P_1
// have 64 columns of their own, so S of the next key tile is issued as soon as this one's scores
// are in registers; above, P_t takes the columns of S_t and the next S_t waits until P_t V has
// read it.
//
// Short tails.  A sequence length just above a multiple of 128 (ViT: 257 = 2 x 128 + the class
// token) would spend a whole item on a few rows.  When at most ATT_TAIL_MAX rows are left over, the
// tensor-core tiles cover only the full multiples and a small CUDA-core kernel computes the
// leftover query rows (see attn_fwd_tail_kernel).
#include "attn_common.cuh"
#include "api.h"

namespace pf {

constexpr int ATT_TAIL_MAX = 4;      // leftover rows handled on CUDA cores
constexpr int ATT_TAIL_SEQ_MAX = 2048;  // most keys of a leftover row

struct AttnParams {
  int B, H, Sq, Sk, D;
  int causal;
  float scale;
  int fmt;              // 0 fp16, 1 bf16
  void* o;              // [B,Sq,H,D] contiguous
  float* lse;           // [B,H,Sq]
  int* status;
  int q_rows;           // query rows of the tensor-core kernel; the others are leftover rows
  int q_pairs;          // pairs of query tiles per head: ceil(q_rows / 256)
  int n_pair;           // the first items are pairs, the others split tiles (see FwdItem)
  int item0;            // first item of this launch
  int q_tail;           // leftover rows
  // A call's launches need nothing of one another, so that the next one's CTAs start on the SMs that the
  // last round leaves idle (a CTA of the tensor-core kernel holds an SM to itself).  They find the inputs
  // complete, which the first launch has waited for, and read them through L2 only.
  int not_first, not_last;
  // raw views for the leftover rows (element strides: batch, seq, head)
  const void* q; const void* k; const void* v;
  long long sq[3], sk[3], sv[3];
};

// One leftover query row per CTA, on CUDA cores.  Four lanes share a key (8 columns to a lane at a time) and
// fold the keys they meet into a maximum, a sum and an output of their own; the 32 groups are joined at the
// end.  Bound by memory: a thread asks for the keys and values of its next two tokens while it works on
// one, in slots of its own, so that the loop has no barrier ([64, 257, 16, 64] 90 -> 72 us with the tiles,
// causal [1, 2049, 32, 128] 95 -> 78, against one thread per key and staged scores).
template <int DP>
struct TailCfg {
  static constexpr int NV = DP / 32;                     // vectors of 8 columns per lane
  static constexpr int THREADS = 128, GROUPS = THREADS / 4, DEPTH = 3;
  static constexpr int RING = DEPTH * 2 * NV * THREADS * 16;
  static constexpr int SMEM = RING > 4 * (DP + 2) * 4 ? RING : 4 * (DP + 2) * 4;
};
template <typename T, int DP>
__global__ void __launch_bounds__(TailCfg<DP>::THREADS)
attn_fwd_tail_kernel(const AttnParams p) {       // never a call's first launch
  using C = TailCfg<DP>;
  constexpr int NV = C::NV, THREADS = C::THREADS, GROUPS = C::GROUPS, DEPTH = C::DEPTH;
  extern __shared__ __align__(16) uint8_t tail_smem[];
  uint4* ring = reinterpret_cast<uint4*>(tail_smem) + threadIdx.x;     // [DEPTH][K, V][NV][THREADS]
  float* warps = reinterpret_cast<float*>(tail_smem);                  // after the loop: [4][DP + 2]
  const int qi = p.q_rows + (int)blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & 3, grp = threadIdx.x >> 2;
  const T* qrow = reinterpret_cast<const T*>(p.q) + b * p.sq[0] + (long long)qi * p.sq[1] + h * p.sq[2];
  const T* kb = reinterpret_cast<const T*>(p.k) + b * p.sk[0] + h * p.sk[2];
  const T* vb = reinterpret_cast<const T*>(p.v) + b * p.sv[0] + h * p.sv[2];
  const float c2 = p.scale * LOG2E;
  const int keys = p.causal ? max(0, min(p.Sk, qi + p.Sk - p.Sq + 1)) : p.Sk;   // visible to this row
  const int trips = (keys + GROUPS - 1) / GROUPS;                      // the same for every lane
  auto in = [&](int i) { return (sub + 4 * i) * 8 < p.D; };
  auto fetch = [&](int trip) {
    if (trip < trips) {
      const long long x = min(trip * GROUPS + grp, keys - 1);
      uint4* slot = ring + (trip % DEPTH) * 2 * NV * THREADS;
#pragma unroll
      for (int i = 0; i < NV; ++i)
        if (in(i)) {
          cp_async16(slot + i * THREADS, kb + x * p.sk[1] + (sub + 4 * i) * 8);
          cp_async16(slot + (NV + i) * THREADS, vb + x * p.sv[1] + (sub + 4 * i) * 8);
        }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int i = 0; i < DEPTH * 2 * NV; ++i)                             // columns beyond D count as zeros
    if (!in(i % NV)) ring[i * THREADS] = make_uint4(0, 0, 0, 0);
  for (int i = 0; i < DEPTH - 1; ++i) fetch(i);
  float q[8 * NV], acc[8 * NV] = {}, m = -INFINITY, l = 0.f;
  auto widen = [](const uint4& u, float* f) {
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = to_f32<T>(reinterpret_cast<const T*>(&u)[j]);
  };
#pragma unroll
  for (int i = 0; i < NV; ++i)
    widen(in(i) ? __ldcg(reinterpret_cast<const uint4*>(qrow) + sub + 4 * i) : make_uint4(0, 0, 0, 0),
          q + i * 8);
  for (int trip = 0; trip < trips; ++trip) {
    fetch(trip + DEPTH - 1);
    cp_async_wait<DEPTH - 1>();
    uint4* slot = ring + (trip % DEPTH) * 2 * NV * THREADS;
    // Beyond the last key lies a copy of its value, which a weight of zero does not take out if it is infinite.
    const bool live = trip * GROUPS + grp < keys;
    if (!live) {
#pragma unroll
      for (int i = 0; i < NV; ++i) slot[(NV + i) * THREADS] = make_uint4(0, 0, 0, 0);
    }
    float f[8], s = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      widen(slot[i * THREADS], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) s = fmaf(f[j], q[i * 8 + j], s);
    }
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s = live ? s * c2 : -INFINITY;
    if (s > m) {                                                       // also the first finite score
      const float alpha = exp2f(m - s);
      l *= alpha;
#pragma unroll
      for (int j = 0; j < 8 * NV; ++j) acc[j] *= alpha;
      m = s;
    }
    const float w = s == -INFINITY ? 0.f : exp2f(s - m);               // a NaN stays one
    l += w;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      widen(slot[(NV + i) * THREADS], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i * 8 + j] = fmaf(w, f[j], acc[i * 8 + j]);
    }
  }
  cp_async_wait<0>();
  // the eight groups of a warp, then the warps
  float mw = m;
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) mw = fmaxf(mw, __shfl_xor_sync(0xffffffffu, mw, o));
  const float mine = mw == -INFINITY ? 0.f : exp2f(m - mw);
  l *= mine;
#pragma unroll
  for (int j = 0; j < 8 * NV; ++j) acc[j] *= mine;
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    l += __shfl_xor_sync(0xffffffffu, l, o);
#pragma unroll
    for (int j = 0; j < 8 * NV; ++j) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
  }
  __syncthreads();                                                     // `warps` lies over the ring
  float* w = warps + warp * (DP + 2);
  if (lane < 4) {
#pragma unroll
    for (int j = 0; j < 8 * NV; ++j) w[(sub + 4 * (j / 8)) * 8 + j % 8] = acc[j];
  }
  if (lane == 0) { w[DP] = mw; w[DP + 1] = l; }
  __syncthreads();
  float mx = -INFINITY, sum = 0.f, o = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) mx = fmaxf(mx, warps[i * (DP + 2) + DP]);
  const int d = threadIdx.x;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float* wi = warps + i * (DP + 2);
    const float e = mx == -INFINITY ? 0.f : exp2f(wi[DP] - mx);
    sum = fmaf(e, wi[DP + 1], sum);
    if (d < DP) o = fmaf(e, wi[d], o);
  }
  if (d < p.D)
    (reinterpret_cast<T*>(p.o) + (((long long)b * p.Sq + qi) * p.H + h) * p.D)[d] =
        from_f32<T>(sum == 0.f ? 0.f : o / sum);
  if (d == 0)
    p.lse[((long long)b * p.H + h) * p.Sq + qi] = (sum > 0.f) ? (mx + log2f(sum)) * LN2 : -INFINITY;
  if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) after_previous();
}

template <int DP>
struct FwdCfg {
  static constexpr int NBLK = (DP + 63) / 64;
  static constexpr int TILE = NBLK * ATT_BLK;
  static constexpr bool ALIAS_P = DP > 64;
  static constexpr int ST = NBLK >= 2 ? 2 : 4;          // K/V ring stages
  static constexpr int OFF_K = 2 * TILE;
  static constexpr int OFF_V = OFF_K + ST * TILE;
  static constexpr int OFF_SIDE = OFF_V + ST * TILE;     // maxima and sums of a split tile's side 1
  static constexpr int OFF_BOX = OFF_SIDE + 2 * ATT_BM * 4;   // 8 warps x 2 boxes of 32 rows x 32 columns of O
  static constexpr int OFF_BAR = OFF_BOX + 8 * 2 * 2048;
  static constexpr int SMEM = OFF_BAR + 256;
  static constexpr int T_O = 256;                        // + t * DP
  static constexpr int T_P = ALIAS_P ? 0 : 256 + 2 * DP;
  static constexpr int P_TILE = ALIAS_P ? 128 : 64;      // column distance of P_0 and P_1
  // three warpgroups of 168 registers a thread at launch; the softmax ones hold a row of scores
  static constexpr int THREADS = 384;
  static constexpr int REGS_SOFTMAX = 216, REGS_OTHER = 72;
  static_assert(2 * REGS_SOFTMAX + REGS_OTHER <= 3 * 168, "registers of the block");
  static_assert(SMEM <= 232448, "shared memory per CTA");
  static_assert((ALIAS_P ? T_O + 2 * DP : T_P + 128) <= 512, "TMEM columns");
};

// An item is a pair of query tiles that read the same key tiles or, when the pairs left over after
// whole rounds of the SMs are no more than half of those, one query tile whose key tiles are dealt to
// the two sides in turn; each side then has the maximum, sum and output of its own keys, which side 0
// joins at the end.  A split tile takes half the steps of a pair; it is always its CTA's last item.
// Head dim 128, 2048 tokens: 8 heads (64 pairs) 45 us as pairs, 28 split; 20 heads (160 pairs) 89
// and 72.  Head dim 64, [1, 2048, 8, 64]: 38 and 24 us.
struct FwdItem {
  int q0, h, b, n[2];    // first query row; key tiles seen by the two query tiles
};
__device__ __forceinline__ FwdItem fwd_item(const AttnParams& p, int w) {
  FwdItem it;
  int qp, bh;
  if (p.causal) {
    // later queries see more keys: the long items of every head are dealt first
    qp = w / (p.B * p.H);
    bh = w - qp * (p.B * p.H);
    qp = p.q_pairs - 1 - qp;
  } else {
    bh = w / p.q_pairs;
    qp = w - bh * p.q_pairs;
  }
  it.q0 = qp * 2 * ATT_BM;
  it.h = bh % p.H;
  it.b = bh / p.H;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int q0 = it.q0 + t * ATT_BM;
    int kv_end = p.Sk;
    if (p.causal) kv_end = min(p.Sk, q0 + ATT_BM + (p.Sk - p.Sq));
    it.n[t] = (q0 < p.q_rows && kv_end > 0) ? (kv_end + ATT_BN - 1) / ATT_BN : 0;
  }
  return it;
}
// item `w` of a kernel whose items from n_pair on are split tiles (`split` says whether this one is)
__device__ __forceinline__ FwdItem fwd_item(const AttnParams& p, int w, bool& split) {
  w += p.item0;
  split = w >= p.n_pair;
  if (!split) return fwd_item(p, w);
  const int u = w - p.n_pair, t = u & 1;
  FwdItem it = fwd_item(p, p.n_pair + (u >> 1));
  const int n = t ? it.n[1] : it.n[0];
  it.q0 += t * ATT_BM;
  it.n[0] = (n + 1) / 2;
  it.n[1] = n / 2;
  return it;
}
// rounds run alternately forwards and backwards over the CTAs, so that a CTA with a long item in
// one round gets a short one in the next
__device__ __forceinline__ int fwd_index(int r) {
  const int slot = (r & 1) ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x;
  return r * (int)gridDim.x + slot;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Probabilities of one row under the maximum `m_sub`, packed to 16 bits and stored to the columns of P
// chunk by chunk; returns their fp32 sum (of the unrounded values).  With MAX the largest score is
// found on the way: its comparisons go to another unit than the exponentials that bound the loop.
template <typename T, bool MASKED, bool MAX>
__device__ __forceinline__ float probs(const uint32_t (&s)[4][32], uint32_t t_p, float c2, float m_sub,
                                       int n_chunks, int lim, float& mx) {
  const uint64_t c2v = f2_pack(c2, c2), nm = f2_pack(-m_sub, -m_sub);
  uint64_t r01 = 0, r23 = 0;                  // pairs of fp32 sums
  float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if (!MASKED || c < n_chunks) {
      uint32_t pk[16];
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        float x[4], e[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = __uint_as_float(s[c][i + u]);
        if (MAX) {
          m0 = max3(m0, x[0], x[1]);
          m1 = max3(m1, x[2], x[3]);
        }
        f2_unpack(fma2(f2_pack(x[0], x[1]), c2v, nm), e[0], e[1]);
        f2_unpack(fma2(f2_pack(x[2], x[3]), c2v, nm), e[2], e[3]);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          e[u] = exp2f(e[u]);
          if (MASKED && c * 32 + i + u >= lim) e[u] = 0.f;
        }
        r01 = add2(r01, f2_pack(e[0], e[1]));
        r23 = add2(r23, f2_pack(e[2], e[3]));
        pk[i / 2] = pack2<T>(e[0], e[1]);
        pk[i / 2 + 1] = pack2<T>(e[2], e[3]);
      }
      tmem_st16(t_p + c * 16, pk);
    }
  }
  if (MAX) mx = fmaxf(m0, m1);
  float a, b, d, e;
  f2_unpack(r01, a, b);
  f2_unpack(r23, d, e);
  return (a + b) + (d + e);
}

template <typename T, int DP, bool SPLIT, bool ONE_ISSUER>
__global__ void __launch_bounds__(FwdCfg<DP>::THREADS, 1)
attn_fwd_ws_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                   const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap to,
                   const AttnParams p, const int n_items) {
  using C = FwdCfg<DP>;
  constexpr int NBLK = C::NBLK, TILE = C::TILE, ST = C::ST;
  // Pairs with P in columns of its own: a thread per side issues its products, where one thread for both held
  // a side's products back until the other's were due ([4, 4096, 10, 64] 266 -> 249 us, 77 keys
  // [4, 1024, 20, 64] 17.7 -> 16.7).  With P in the columns of S that order is what keeps the sides half a step
  // apart (head dim 128: 176 us so, 208 with two threads), and the form with split tiles lost, too
  // ([1, 8192, 10, 64] 264 and 290); see also one_issues.
  constexpr bool TWO_ISSUERS = !C::ALIAS_P && !SPLIT && !ONE_ISSUER;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint64_t* q_full = bars;               // [2] by query tile
  uint64_t* q_empty = bars + 2;          // [2] the item's last S product of that tile is done
  uint64_t* s_full = bars + 4;           // [2]
  uint64_t* s_empty = bars + 6;          // [2] scores are in registers (P in columns of its own)
  uint64_t* p_full = bars + 8;           // [2] P is in TMEM (and O rescaled)
  uint64_t* pv_done = bars + 10;         // [2] P V has completed
  uint64_t* k_full = bars + 12;          // [ST]
  uint64_t* k_empty = k_full + ST;
  uint64_t* v_full = k_empty + ST;
  uint64_t* v_empty = v_full + ST;
  uint64_t* joined = v_empty + ST;       // side 1 of a split tile has left its maxima and sums
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(joined + 1);
  constexpr int N_BARS = 13 + 4 * ST;
  float* side1 = reinterpret_cast<float*>(smem + C::OFF_SIDE);   // [2][128]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // the 128-byte swizzle works on absolute shared-memory addresses
  if ((smem_u32(smem) & 1023u) != 0u) {
    if (tid == 0) report(p.status, PF_ERR_BAD_ARG);
    return;
  }
  if (tid == 0) {
    tma_prefetch_desc(&tq); tma_prefetch_desc(&tk); tma_prefetch_desc(&tv);
    tma_prefetch_desc(&to);
    for (int i = 0; i < N_BARS; ++i) mbar_init(&bars[i], 1);
    for (int t = 0; t < 2; ++t) { mbar_init(&s_empty[t], 4); mbar_init(&p_full[t], 4); }
    mbar_init(joined, 4);
    if (TWO_ISSUERS)                     // both sides free a tile, in either order
      for (int i = 0; i < ST; ++i) { mbar_init(&k_empty[i], 2); mbar_init(&v_empty[i], 2); }
    mbar_fence_init();
  }
  if (warp == 9) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_of(tmem_slot);
  if (!p.not_first) after_previous();
  if (p.not_last && tid == 0) let_next_start();

  // one split per warpgroup: its four warps execute the same instruction
  if (warp >= 8) {
    regs_dec<C::REGS_OTHER>();
    if (warp == 8) {
      // ---------------------------------------------------------------- TMA producer
      if (elect_one()) {
        uint32_t g = 0, qc[2] = {0, 0};
        bool ok = true;
        for (int r = 0; ok && r * (int)gridDim.x < n_items; ++r) {
          const int w = fwd_index(r);
          if (w >= n_items) continue;
          bool split = false;
          const FwdItem it = SPLIT ? fwd_item(p, w, split) : fwd_item(p, w);
          const int nmax = split ? it.n[0] + it.n[1] : max(it.n[0], it.n[1]);
          for (int j = 0; j < nmax && ok; ++j, ++g) {
            const int st = g % ST;
            if (j == 0 && it.n[0] > 0) {
              ok = mbar_wait(&q_empty[0], (qc[0] & 1) ^ 1, p.status, PF_ERR_TIMEOUT_EMPTY);
              if (!ok) break;
              load_tile<NBLK>(smem, &tq, &q_full[0], it.h, it.q0, it.b);
              ++qc[0];
            }
            ok = mbar_wait(&k_empty[st], ((g / ST) & 1) ^ 1, p.status, PF_ERR_TIMEOUT_EMPTY);
            if (!ok) break;
            load_tile<NBLK>(smem + C::OFF_K + st * TILE, &tk, &k_full[st], it.h, j * ATT_BN, it.b);
            if (j == 0 && it.n[1] > 0) {
              ok = mbar_wait(&q_empty[1], (qc[1] & 1) ^ 1, p.status, PF_ERR_TIMEOUT_EMPTY);
              if (!ok) break;
              load_tile<NBLK>(smem + TILE, &tq, &q_full[1], it.h,
                              split ? it.q0 : it.q0 + ATT_BM, it.b);
              ++qc[1];
            }
            ok = mbar_wait(&v_empty[st], ((g / ST) & 1) ^ 1, p.status, PF_ERR_TIMEOUT_EMPTY);
            if (!ok) break;
            load_tile<NBLK>(smem + C::OFF_V + st * TILE, &tv, &v_full[st], it.h, j * ATT_BN, it.b);
          }
        }
      }
      __syncwarp();
    } else if (TWO_ISSUERS && (warp == 9 || warp == 10)) {
      // ---------------------------------------------------------------- MMA issuers, one per side
      if (elect_one()) {
        const int t = warp - 9;
        const uint32_t id_o = make_idesc_f16(128, DP, p.fmt, 0, 1);
        const uint32_t t_s = tmem + t * 128, t_o = tmem + C::T_O + t * DP, t_p = tmem + C::T_P + t * C::P_TILE;
        const uint32_t sQ = smem_u32(smem + t * TILE);
        uint32_t g = 0, items = 0, cnt = 0;      // ring position; items and steps of this side so far
        bool ok = true;
        for (int r = 0; ok && r * (int)gridDim.x < n_items; ++r) {
          const int w = fwd_index(r);
          if (w >= n_items) continue;
          const FwdItem it = fwd_item(p, w);
          const int n = t ? it.n[1] : it.n[0], other = t ? it.n[0] : it.n[1];
          auto keys = [&](int j) { return (min(ATT_BN, p.Sk - j * ATT_BN) + 15) / 16 * 16; };
          // a tile is free when both sides have read it; one that the other does not read counts twice
          auto free_tile = [&](uint64_t* bar, int j) {
            tc_commit(bar);
            if (j >= other) tc_commit(bar);
          };
          // S of step j, once the previous scores are in registers
          auto issue_s = [&](int j) -> bool {
            const int st = (g + j) % ST;
            if (!mbar_wait(&k_full[st], ((g + j) / ST) & 1, p.status, PF_ERR_TIMEOUT_FULL)) return false;
            if (cnt > 0 && !mbar_wait(&s_empty[t], (cnt - 1) & 1, p.status, PF_ERR_TIMEOUT_TMEM_EMPTY))
              return false;
            tc_fence_after();
            mma_kk<DP / 16>(t_s, sQ, smem_u32(smem + C::OFF_K + st * TILE),
                            make_idesc_f16(128, keys(j), p.fmt, 0, 0));
            tc_commit(&s_full[t]);
            free_tile(&k_empty[st], j);
            if (j == n - 1) tc_commit(&q_empty[t]);
            ++cnt;
            return true;
          };
          if (n > 0) {
            ok = mbar_wait(&q_full[t], items & 1, p.status, PF_ERR_TIMEOUT_FULL) && issue_s(0);
            ++items;
          }
          for (int j = 0; j < n && ok; ++j) {
            const uint32_t c = cnt - 1;          // step j
            if (j + 1 < n && !(ok = issue_s(j + 1))) break;
            const int st = (g + j) % ST;
            ok = mbar_wait(&v_full[st], ((g + j) / ST) & 1, p.status, PF_ERR_TIMEOUT_FULL) &&
                 mbar_wait(&p_full[t], c & 1, p.status, PF_ERR_TIMEOUT_FULL);
            if (!ok) break;
            tc_fence_after();
            mma_t_mn(t_o, t_p, 32, smem_u32(smem + C::OFF_V + st * TILE), id_o, j > 0, keys(j) / 16);
            tc_commit(&pv_done[t]);
            free_tile(&v_empty[st], j);
          }
          g += max(n, other);
        }
      }
      __syncwarp();
    } else if (!TWO_ISSUERS && warp == 9) {
      // ---------------------------------------------------------------- MMA issuer
      if (elect_one()) {
        const uint32_t id_s = make_idesc_f16(128, 128, p.fmt, 0, 0);
        const uint32_t id_o = make_idesc_f16(128, DP, p.fmt, 0, 1);
        uint32_t g = 0, qc[2] = {0, 0}, cnt[2] = {0, 0};    // cnt: S tiles issued per side
        bool ok = true;
        // S of step j of side t: key tile kt (ring position gg).  Its columns must be free: the
        // previous scores are in registers, or (P in the same columns) the previous P V has read
        // its probabilities.
        auto issue_s = [&](int t, uint32_t gg, int j, int kt, int n, bool last_of_tile) -> bool {
          const int st = gg % ST;
          if (j == 0) {
            if (!mbar_wait(&q_full[t], qc[t] & 1, p.status, PF_ERR_TIMEOUT_FULL)) return false;
            ++qc[t];
          }
          if (!mbar_wait(&k_full[st], (gg / ST) & 1, p.status, PF_ERR_TIMEOUT_FULL))
            return false;
          if (cnt[t] > 0 && !mbar_wait(C::ALIAS_P ? &pv_done[t] : &s_empty[t],
                                            (cnt[t] - 1) & 1, p.status,
                                            PF_ERR_TIMEOUT_TMEM_EMPTY))
            return false;
          tc_fence_after();
          const int rem = min(ATT_BN, p.Sk - kt * ATT_BN);
          const int n_mma = (rem + 15) / 16 * 16;
          const uint32_t id = n_mma == ATT_BN ? id_s : make_idesc_f16(128, n_mma, p.fmt, 0, 0);
          mma_kk<DP / 16>(tmem + t * 128, smem_u32(smem + t * TILE),
                       smem_u32(smem + C::OFF_K + st * TILE), id);
          if (last_of_tile) tc_commit(&k_empty[st]);
          tc_commit(&s_full[t]);
          if (j == n - 1) tc_commit(&q_empty[t]);
          ++cnt[t];
          return true;
        };
        for (int r = 0; ok && r * (int)gridDim.x < n_items; ++r) {
          const int w = fwd_index(r);
          if (w >= n_items) continue;
          bool split = false;
          const FwdItem it = SPLIT ? fwd_item(p, w, split) : fwd_item(p, w);
          const int nmax = max(it.n[0], it.n[1]);
          // in a pair, tile 1 reads every key tile that tile 0 reads, and after it
          auto last_reader = [&](int t, int j) {
            return (SPLIT && split) || t == 1 || j >= it.n[1];
          };
          // key tile of step j of side t
          auto key = [&](int t, int j) { return (SPLIT && split) ? 2 * j + t : j; };
#pragma unroll
          for (int t = 0; t < 2; ++t)
            if (ok && it.n[t] > 0)
              ok = issue_s(t, g + key(t, 0), 0, key(t, 0), it.n[t], last_reader(t, 0));
          for (int j = 0; j < nmax && ok; ++j) {
            if (!C::ALIAS_P) {
#pragma unroll
              for (int t = 0; t < 2; ++t)
                if (ok && j + 1 < it.n[t])
                  ok = issue_s(t, g + key(t, j + 1), j + 1, key(t, j + 1), it.n[t],
                               last_reader(t, j + 1));
              if (!ok) break;
            }
            if (!SPLIT) {        // one V tile for both sides
              ok = mbar_wait(&v_full[(g + j) % ST], ((g + j) / ST) & 1, p.status,
                                  PF_ERR_TIMEOUT_FULL);
              if (!ok) break;
            }
#pragma unroll
            for (int t = 0; t < 2; ++t) {
              if (!ok || j >= it.n[t]) continue;
              const uint32_t gg = g + key(t, j);
              const int st = gg % ST;
              if (SPLIT)
                ok = mbar_wait(&v_full[st], (gg / ST) & 1, p.status, PF_ERR_TIMEOUT_FULL);
              const int k_steps = (min(ATT_BN, p.Sk - key(t, j) * ATT_BN) + 15) / 16;
              // the probabilities waited for are those of the step before any S issued above
              const uint32_t c = cnt[t] - 1 - ((!C::ALIAS_P && j + 1 < it.n[t]) ? 1u : 0u);
              ok = ok && mbar_wait(&p_full[t], c & 1, p.status, PF_ERR_TIMEOUT_FULL);
              if (!ok) continue;
              tc_fence_after();
              const uint32_t sV = smem_u32(smem + C::OFF_V + st * TILE);
              const uint32_t t_p = tmem + C::T_P + t * C::P_TILE;
              mma_t_mn(tmem + C::T_O + t * DP, t_p, 32, sV, id_o, j > 0, k_steps);
              if (last_reader(t, j)) tc_commit(&v_empty[st]);
              tc_commit(&pv_done[t]);
              if (C::ALIAS_P && j + 1 < it.n[t])
                ok = issue_s(t, g + key(t, j + 1), j + 1, key(t, j + 1), it.n[t],
                             last_reader(t, j + 1));
            }
          }
          g += (SPLIT && split) ? it.n[0] + it.n[1] : nmax;
        }
      }
      __syncwarp();
    }
  } else {
    // ---------------------------------------------------------------- softmax (2 x 4 warps)
    regs_inc<C::REGS_SOFTMAX>();
    const int t = warp >> 2, quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_off = uint32_t(quad * 32) << 16;
    const uint32_t t_s = tmem + t * 128 + lane_off;
    const uint32_t t_o = tmem + C::T_O + t * DP + lane_off;
    const uint32_t t_p = tmem + C::T_P + t * C::P_TILE + lane_off;
    const float c2 = p.scale * LOG2E;
    const int shift = p.Sk - p.Sq;
    uint8_t* boxes = smem + C::OFF_BOX + warp * 4096;
    uint32_t cnt = 0, box = 0;
    bool ok = true;
    for (int r = 0; ok && r * (int)gridDim.x < n_items; ++r) {
      const int w = fwd_index(r);
      if (w >= n_items) continue;
      bool split = false;
      const FwdItem it = SPLIT ? fwd_item(p, w, split) : fwd_item(p, w);
      const int q0 = it.q0 + (split ? 0 : t * ATT_BM), n_tiles = t ? it.n[1] : it.n[0];
      const int qi = q0 + row;
      if (q0 >= p.q_rows || (split && t && it.n[0] == 0)) continue;
      T* dst = reinterpret_cast<T*>(p.o) + (((long long)it.b * p.Sq + qi) * p.H + it.h) * p.D;
      float* lse_dst = p.lse + ((long long)it.b * p.H + it.h) * p.Sq + qi;
      if (n_tiles == 0 && !(split && t)) {      // no key is visible to this query tile
        if (qi < p.Sq) {
          for (int c = 0; c < p.D / 8; ++c)
            reinterpret_cast<uint4*>(dst)[c] = make_uint4(0, 0, 0, 0);
          *lse_dst = -INFINITY;
        }
        continue;
      }
      // a warp whose rows all lie beyond the last query only keeps the barriers going
      const bool warp_live = q0 + quad * 32 < p.Sq;
      float m_used = -INFINITY, l = 0.f;
      bool s_seen = false;                   // the scores of this step are known to be there
      for (int j = 0; j < n_tiles && ok; ++j, ++cnt) {
        const int k0 = (split ? 2 * j + t : j) * ATT_BN;
        const int rem = min(ATT_BN, p.Sk - k0);
        const int n_chunks = ((rem + 15) / 16 * 16 + 31) / 32;
        // a tile needs masks when it is ragged or crosses the causal diagonal of this q tile
        const bool masked = rem < ATT_BN || (p.causal && k0 + ATT_BN - 1 > q0 + shift);
        if (!s_seen) ok = mbar_wait(&s_full[t], cnt & 1, p.status, PF_ERR_TIMEOUT_TMEM_FULL);
        if (!ok) break;
        tc_fence_after();
        // looked at here, needed below: even a wait that is satisfied takes some 130 cycles
        const bool pv_seen = C::ALIAS_P || j == 0 || mbar_test(&pv_done[t], (cnt - 1) & 1);
        uint32_t s[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32(t_s + c * 32, s[c]);
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_wait_for(s[c]);
        if (!C::ALIAS_P) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&s_empty[t]);
        }
        // keys of this tile below `lim` are visible to this row
        const int lim = p.causal ? min(p.Sk, qi + shift + 1) - k0 : p.Sk - k0;
        // P in columns of its own: the previous P V must have read its probabilities before they are
        // overwritten (that product ran while the scores were fetched), and O must hold every
        // earlier tile before it is rescaled.  The wait also keeps a warp without live rows from
        // arriving twice on one phase of p_full.  With P in the columns of S the scores were only
        // computed after that product.
        if (!pv_seen) ok = mbar_wait(&pv_done[t], (cnt - 1) & 1, p.status, PF_ERR_TIMEOUT_TMEM_FULL);
        if (!ok) break;
        tc_fence_after();
        if (warp_live) {
          // The maximum in use only moves when the row's grew by more than 2^8, which is rare after
          // the first tiles: the probabilities are computed under the old one while the new maximum
          // is looked for, and once more if a row of the warp turns out to need it.
          // (Two passes, maximum first, took 490 cycles of the 3470 of a step at head dim 64.)
          float mx = -INFINITY, rs = 0.f;
          bool again = j == 0 || masked;
          if (!again) {
            rs = probs<T, false, true>(s, t_p, c2, (m_used == -INFINITY) ? 0.f : m_used, 4, ATT_BN, mx);
            mx *= c2;                                 // c2 > 0; -inf stays -inf
            again = __any_sync(0xffffffffu, mx > m_used + 8.f);
            if (again) tmem_st_wait();
          } else if (!masked) {
            float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
#pragma unroll
              for (int i = 0; i < 32; i += 4) {
                m0 = max3(m0, __uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1]));
                m1 = max3(m1, __uint_as_float(s[c][i + 2]), __uint_as_float(s[c][i + 3]));
              }
            }
            mx = fmaxf(m0, m1) * c2;
          } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              if (c < n_chunks) {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                  if (c * 32 + i < lim) mx = fmaxf(mx, __uint_as_float(s[c][i]));
              }
            }
            mx *= c2;
          }
          if (again) {
            float alpha = 1.f;
            if (j == 0) {
              m_used = mx;
            } else if (mx > m_used + 8.f) {           // also true when m_used is still -inf
              alpha = exp2f(m_used - mx);             // exp2(-inf) = 0: nothing had accumulated
              m_used = mx;
            }
            const float m_sub = (m_used == -INFINITY) ? 0.f : m_used;
            rs = masked ? probs<T, true, false>(s, t_p, c2, m_sub, n_chunks, lim, mx)
                        : probs<T, false, false>(s, t_p, c2, m_sub, 4, ATT_BN, mx);
            if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
              l *= alpha;
#pragma unroll
              for (int c = 0; c < DP / 32; ++c) {
                uint32_t o[32];
                tmem_ld32(t_o + c * 32, o);
                tmem_ld_wait_for(o);
#pragma unroll
                for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                tmem_st32(t_o + c * 32, o);
              }
            }
          }
          l += rs;
          if (!C::ALIAS_P) s_seen = j + 1 < n_tiles && mbar_test(&s_full[t], (cnt + 1) & 1);
          tmem_st_wait();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[t]);
      }
      if (!ok) break;
      // ---- epilogue of the tile: O / l
      if (!SPLIT || n_tiles > 0) {
        ok = mbar_wait(&pv_done[t], (cnt - 1) & 1, p.status, PF_ERR_TIMEOUT_TMEM_FULL);
        if (!ok) break;
        tc_fence_after();
      }
      float w0 = 1.f, w1 = 0.f;              // weights of the two sides' outputs
      if (split) {
        if (t) {                             // the thread of this row on side 0 finishes it
          side1[row] = m_used;
          side1[ATT_BM + row] = l;
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(joined);
          continue;
        }
        ok = mbar_wait(joined, 0, p.status, PF_ERR_TIMEOUT_TMEM_FULL);
        if (!ok) break;
        tc_fence_after();
        const float m1 = side1[row], m = fmaxf(m_used, m1), m_sub = (m == -INFINITY) ? 0.f : m;
        w0 = exp2f(m_used - m_sub);
        w1 = exp2f(m1 - m_sub);
        l = l * w0 + side1[ATT_BM + row] * w1;
        m_used = m;
      }
      if (warp_live) {
        const float inv = l > 0.f ? 1.f / l : 0.f;
        w0 *= inv;
        w1 *= inv;
#pragma unroll
        for (int c = 0; c < DP / 32; ++c) {
          uint32_t o[32];
          tmem_ld32(t_o + c * 32, o);
          tmem_ld_wait_for(o);
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * w0);
          if (split && it.n[1] > 0) {     // the same row of the other side's columns
            uint32_t o1[32];
            tmem_ld32(t_o + DP + c * 32, o1);
            tmem_ld_wait_for(o1);
#pragma unroll
            for (int i = 0; i < 32; ++i)
              o[i] = __float_as_uint(fmaf(__uint_as_float(o1[i]), w1, __uint_as_float(o[i])));
          }
          // Through boxes: 16 bytes of a row per thread and store take longer to leave than a key tile's
          // products (at head dim 88 8000 cycles from item to item, 3600 between key tiles).  The store
          // that last used this box must have read it; rows and columns that do not exist are clipped.
          uint8_t* bx = boxes + (box & 1) * 2048;
          if (lane == 0 && box >= 2) tma_store_wait_read_but_one();
          __syncwarp();
          box_row16<T>(bx, lane, o);
          fence_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_4d(&to, bx, c * 32, it.h, q0 + quad * 32, it.b);
            tma_store_commit();
          }
          ++box;
        }
        if (qi < p.Sq) *lse_dst = (l > 0.f) ? (m_used + log2f(l)) * LN2 : -INFINITY;
      }
      // the reads of O above have completed (tcgen05.wait::ld); the next item's first P V of this
      // tile, which overwrites O, is ordered after them by this warp's next arrival on p_full
      tc_fence_before();
    }
    if (lane == 0) tma_store_wait_all();
  }

  // teardown: every role reaches this point (all waits are bounded)
  tc_fence_before();
  __syncthreads();
  if (warp == 9) { tc_fence_after(); tmem_dealloc(tmem, 512); }
  if (p.not_first && blockIdx.x == 0) after_previous();
}

// Whether one thread issues the products of both sides of pairs up to head dim 64.  Where the tiles of a head are
// odd, a side that has none to itself goes ahead to the next item, and with a ragged key tile the two then
// keep fetching one another's instructions out: half of the time of a step goes there.  Held together by one
// thread they do not ([19, 640, 19, 64] over 612 keys 118 us with two, 101 with one; over 640 keys 84 and 90).
// The more key tiles, the rarer the ragged one, and the more pairs to a head, the rarer the odd tile; four or
// eight pairs to a head put the shorter items on the same SMs; and over few rounds the sides are never far apart.
// Two threads against one, us over us, by heads, query tiles and keys: 361, 3 and 172 1.08, 356 1.14, 612 1.15,
// 868 1.06, 996 1.03; 361, 5 and 172 1.16, 356 1.31, 740 1.11, 996 0.99; 190 (3.9 rounds), 5 and 172 0.99, 356 1.15,
// 868 0.95; 200, 7 and 300 1.10, 428 0.97; 200, 11 and 356 1.12, 556 1.04, 868 1.00; 100 (4.7), 13 and 356 1.08,
// 556 1.00; 498 (20), 11 and 708 1.11; 130 (1.8), 3 and 356 0.95.  Under a causal mask the sides of a pair
// differ by a masked tile, and over many rounds of long rows they come as far apart: head dim 64, 460 heads of 640
// 0.90, 896 0.99, 1024 1.08, 1280 1.10, 300 (8.1 rounds) of 931 0.98, 1024 1.02, 150 (5.1) of 1280 1.00; head dim 32,
// 576 heads of 1024 0.97, 1280 1.03.
static bool one_issues(const AttnParams& p, int Sk) {
  const int q_tiles = (p.q_rows + ATT_BM - 1) / ATT_BM, n_kt = (Sk + ATT_BN - 1) / ATT_BN;
  const int pairs = p.q_pairs;
  const long long tenths = 10ll * pairs * p.H * p.B / attn_sm_count();          // of rounds
  if (p.causal) return n_kt >= 8 && n_kt * tenths >= (p.D <= 32 ? 1500 : Sk % ATT_BN ? 900 : 550);
  if (q_tiles % 2 == 0 || q_tiles == 1 || Sk % ATT_BN == 0) return false;
  const int least = tenths >= (pairs == 2 ? 35 : 60) ? 2 : 3;
  const int most = pairs % 4 == 0 ? 3 : pairs == 2 || tenths >= (pairs <= 5 ? 60 : pairs <= 8 ? 170 : 20 * pairs) ? 7
                   : pairs <= 5 || tenths >= 80 ? 5 : 3;
  return tenths >= (pairs == 2 ? 26 : 35) && n_kt >= least && n_kt <= most;
}

template <typename T, int DP>
static int launch_fwd_ws(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                         const CUtensorMap& to, const AttnParams& p, bool two_launches, bool one_issuer,
                         cudaStream_t st) {
  using C = FwdCfg<DP>;
  const int pairs = p.q_pairs * p.H * p.B, tiles = 2 * (pairs - p.n_pair);
  static bool done[3][64] = {};
  auto run = [&](const AttnParams& q, bool split, int n) -> int {
    if (n <= 0) return 0;
    auto kern = split ? attn_fwd_ws_kernel<T, DP, true, false> : attn_fwd_ws_kernel<T, DP, false, false>;
    const bool one = DP <= 64 && !split && one_issuer;
    if (one) kern = attn_fwd_ws_kernel<T, DP, false, DP <= 64>;
    const int r = set_smem(kern, C::SMEM, done[split ? 1 : one ? 2 : 0]), sms = attn_sm_count();
    if (r) return r;
    after(kern, n < sms ? n : sms, C::THREADS, C::SMEM, st)(tq, tk, tv, to, q, n);
    PF_CHECK_LAUNCH();
    return 0;
  };
  int r;
  AttnParams first = p;
  first.not_last = two_launches || p.q_tail > 0;
  if (two_launches) {
    AttnParams rest = p;
    rest.item0 = p.n_pair;
    rest.not_first = 1;
    rest.not_last = p.q_tail > 0;
    if ((r = run(first, false, p.n_pair)) || (r = run(rest, true, tiles))) return r;
  } else if ((r = run(first, tiles > 0, p.n_pair + tiles))) {
    return r;
  }
  if (p.q_tail > 0) {
    static bool tail_done[64] = {};
    using Tail = TailCfg<DP>;
    // The leftover rows start on the SMs that the last round leaves idle.  No SM may take many more than
    // its share of them, or the others would wait for it: shared memory that nobody uses sees to that.
    // us, after the tiles' end, at once with all that fit on an SM, and with this many: [24, 257, 16, 88]
    // 42.2, 43.5, 39.1; [64, 257, 16, 64] 66.5, 63.8, 63.8; [16, 513, 16, 64] 54.0, 62.0, 53.4; causal
    // [4, 1025, 16, 128] 50.8, 55.6, 45.0; [24, 258, 16, 88] 49.1, 47.3, 45.9; [8, 641, 16, 64] 51.3,
    // 46.9, 44.8.
    const long long share = (long long)p.q_tail * p.H * p.B / attn_sm_count();
    const int per_sm = share < 2 ? 2 : share < 8 ? (int)share : 8, room = 228 * 1024 / per_sm - 2048;
    if ((r = set_smem(attn_fwd_tail_kernel<T, DP>, 112 * 1024, tail_done))) return r;
    after(attn_fwd_tail_kernel<T, DP>, dim3(p.q_tail, p.H, p.B), Tail::THREADS,
          room > Tail::SMEM ? room : Tail::SMEM, st)(p);
    PF_CHECK_LAUNCH();
  }
  return 0;
}

}  // namespace pf

using namespace pf;

// strides are in elements, order (batch, seq, head) for each of q, k, v
PF_API int pf_attn_fwd(const void* q, const void* k, const void* v, void* o, void* lse, int B,
                       int H, int Sq, int Sk, int D, const long long* sq, const long long* sk,
                       const long long* sv, int causal, float scale, int dtype, int* status,
                       void* stream) {
  if (dtype != PF_F16 && dtype != PF_BF16) return -1;
  if (D % 8 || D > 128) return -3;
  if (!strides_ok(q, sq[0], sq[1], sq[2]) || !strides_ok(k, sk[0], sk[1], sk[2]) ||
      !strides_ok(v, sv[0], sv[1], sv[2]) || (reinterpret_cast<uintptr_t>(o) & 15))
    return -2;
  const int fmt = dtype == PF_BF16;
  CUtensorMap tq, tk, tv, to;
  int r;
  if ((r = make_tmap_bshd(&tq, q, fmt, B, Sq, H, D, sq[0], sq[1], sq[2]))) return r;
  if ((r = make_tmap_bshd(&tk, k, fmt, B, Sk, H, D, sk[0], sk[1], sk[2]))) return r;
  if ((r = make_tmap_bshd(&tv, v, fmt, B, Sk, H, D, sv[0], sv[1], sv[2]))) return r;
  const long long so[3] = {(long long)Sq * H * D, (long long)H * D, D};
  if ((r = make_tmap_box32(&to, o, fmt, B, Sq, H, D, so))) return r;
  AttnParams p = {};
  p.B = B; p.H = H; p.Sq = Sq; p.Sk = Sk; p.D = D; p.causal = causal; p.scale = scale;
  p.fmt = fmt; p.o = o; p.lse = (float*)lse; p.status = status;
  p.q = q; p.k = k; p.v = v;
  for (int i = 0; i < 3; ++i) { p.sq[i] = sq[i]; p.sk[i] = sk[i]; p.sv[i] = sv[i]; }
  // A short leftover (at most ATT_TAIL_MAX rows after at least one full tile) goes to the CUDA-core
  // kernel, whose time grows with the keys; otherwise the last tile is ragged.
  const int left = Sq % ATT_BM;
  p.q_tail = (Sq > ATT_BM && left > 0 && left <= ATT_TAIL_MAX && Sk <= ATT_TAIL_SEQ_MAX) ? left : 0;
  p.q_rows = Sq - p.q_tail;
  p.q_pairs = (p.q_rows + 2 * ATT_BM - 1) / (2 * ATT_BM);
  // Pairs left over after whole rounds are split into tiles when these fit one round (FwdItem).  The
  // form of the kernel that can do both takes 4 to 9 % longer over a pair: up to three rounds it gains
  // all the same ([4, 1024, 20, 64] 56 us whole, 48 split, [2, 2048, 20, 128] 116 and 103), after more
  // it does not.  There the whole rounds go to the form without and the tiles to a second launch, whose
  // CTAs start where the first one's leave.  us, by pairs of head dim 64 and key tiles, in one launch and
  // in two: 640 and 4 51.2 51.5, 8 85.5 79.6, 16 146 133, 32 255 238; 664 and 8 86.5 84.2; 900 and 8 113
  // 105.5, 16 201 181; 1500 and 8 170 167; head dim 32 alike.  In three rounds: 468 and 8 64.0 62.2, 500 and
  // 8 63.8 65.7, 464 and 16 107.7 103.5, 496 and 16 109 108.  At head dim 128: 640 and 8 99.5 106, 16 177
  // 176; 900 and 8 134 141, 16 243 240.  Causal items differ in length and are dealt by it: there only a
  // call without a whole round is split.
  const int pairs = p.q_pairs * H * B, left_over = pairs % attn_sm_count();
  const int rounds = pairs / attn_sm_count();
  const bool fits = left_over > 0 && 2 * left_over <= attn_sm_count();
  const int two_from = D > 64 ? (rounds > 3 ? 12 : INT_MAX) : rounds > 3 ? 8 : rounds == 3 ? 16 : INT_MAX;
  const bool two_launches = fits && !causal && (Sk + ATT_BN - 1) / ATT_BN >= two_from;
  // One tile per head is no pair to begin with: its keys are shared out from the third key tile on
  // ([1, 128, 4, 128] 7.2 us whole, 7.8 split).
  const bool split = two_launches ||
                     (fits && rounds <= (causal ? 0 : 3) &&
                      (p.q_rows > ATT_BM || Sk > 2 * ATT_BN));
  p.n_pair = split ? pairs - left_over : pairs;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const bool one_issuer = one_issues(p, Sk);
  PF_ATTN_DISPATCH(launch_fwd_ws, tq, tk, tv, to, p, two_launches, one_issuer, st);
}
