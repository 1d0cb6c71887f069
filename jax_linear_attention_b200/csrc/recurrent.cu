// fp32 token-scan kernels: the exact path of the library (JLA_PATH_RECURRENT).
//
// They walk the tokens in the order of the reference's scan step (src/jla/ops/reference.py:140-157):
// reset, decay, delta write, read; with cu_seqlens every sequence is a row with its own initial and
// final state (reference.py:170-203). Arithmetic is fp32 FMA on CUDA cores whatever the storage dtype,
// so this path serves the fp32 configuration (relative L2 error <= 1e-5 against the fp32 reference) and
// is the on-device cross-check of the tensor-core kernels.
//
// The walks are bound by latency: one token's chain is decay -> key dot product -> write, and it repeats for every
// token of a row. So a walk does nothing but its chain. The columns of the state are independent recurrences: a warp
// owns 32 / KL columns with the key channels over KL lanes (16 channels a thread), so the key reduction is log2(KL)
// shuffles and no barrier; a CTA of four warps stages eight tokens at a time in shared memory, the next eight already on
// their way to registers. The backward has two such walks that need nothing of each other and run side by side in one
// launch: the forward state with a checkpoint every TB tokens, and the state gradient, which never reads the state
// (dS_t = decay (dS_{t+1} + ...), du_t = k_t dS), with its own checkpoints. Everything that needs both, the gradients
// of q, k and the gates, is then computed for all blocks of TB tokens at once from the two checkpoints of a block.
//
// fp32 B1 T512 H4 K = V = 64 forward + backward: 119 + 145 + 16 us of kernels (walk, two walks, block gradients); the
// one-CTA-per-head scan with barriers in every token and the gradient reductions inside the walk took 410 + 2718 us.
// A token of a walk is 108 instructions of one warp, 240 ns: its chain and the waits of a warp that is alone on its
// scheduler.
#include <stdio.h>

#include <type_traits>

#include "common.cuh"
#include "profile.cuh"

namespace jla {
namespace {

constexpr int TB = 16;        // tokens between two checkpoints = tokens of a block of block_grads_kernel
constexpr int SB = 8;         // tokens that a walk stages at a time
constexpr int NW = 4;         // warps of a walk's CTA
constexpr int KPT = 16;       // key channels of a thread in the walks
constexpr int GT = 256;       // threads of block_grads_kernel
constexpr int CT = 64;        // its channel tile
constexpr int VT = 32;        // its tile of value columns
constexpr int VTS = VT + 4;   // (stride of a staged state row: 16-byte reads of 8 neighbouring rows hit 8 bank groups)

struct RecParams {
  Rows rows;
  int H, Hk, K, V;
  int head0, heads;  // the value heads of this launch
  int gate;  // 0 none, 1 scalar, 2 per key channel
  int delta, l2norm;
  float scale;
  const void *q, *k, *v;
  const void* k_read;  // optional [B*T, H, K]: the recall reads the state with it (k still writes); nullptr = k
  const float *g, *beta, *h0;
  void* o;
  float* final_state;
  const void* d_o;
  const float* d_final;
  float *dq_acc, *dk_acc;  // [B*T, H, K] f32
  float* dkr_acc;          // [B*T, H, K] f32: gradient of k_read (with k_read only)
  void* dv;
  float *dg, *dbeta, *dh0;
  // [heads][slots][K*V]: the state entering every block of a row; the state gradient coming from behind every block. Slot of
  // block b of a row: slot0(row) + b.
  float *s_ckpt, *ds_ckpt;
  float *resid, *du;  // [B*T, H, V] f32: v_t - r_t and the gradient of the written value u_t
  int* slot_row;      // [slots]: the row of a slot (unwritten slots hold anything: the reader checks)
  long slots;

  __device__ __forceinline__ long slot0(int r, int tok0) const { return tok0 / TB + r; }
};

template <int KL>
__device__ __forceinline__ float key_sum(float x) {  // over the KL neighbouring lanes of a column
#pragma unroll
  for (int off = KL / 2; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
  return x;
}

__device__ __forceinline__ float warp_sum(float x) { return key_sum<32>(x); }

// ---- staging of the walks --------------------------------------------------------------------------
template <int KL>
struct WalkSmem {
  static constexpr int KP = KL * KPT;        // channels, padded with zeros
  static constexpr int NC = NW * (32 / KL);  // value columns of the CTA
  float q[SB][KP], k[SB][KP], kr[SB][KP], e[SB][KP];
  float x[SB][NC];  // v, or the upstream gradient
  float es[SB], bs[SB];
  int rs[SB], any_reset;
};

// One batch of SB tokens on its way from global memory to shared memory. Warp w carries tokens w and w + NW whole, so
// the L2 norm of q and k (reference.py:128-129) is a warp reduction. Tokens behind the end of the row are staged as
// tokens that change nothing (zero vectors, decay 1).
template <typename T, int KL>
struct Stage {
  static constexpr int M = KL / 2 > 0 ? KL / 2 : 1;            // channels of a lane
  static constexpr int NC = WalkSmem<KL>::NC;
  static constexpr int NX = SB * NC / (NW * 32) > 0 ? SB * NC / (NW * 32) : 1;
  T q[SB / NW][M], k[SB / NW][M], kr[SB / NW][M], x[NX];
  float g[SB / NW][M], gs, beta;
  int seg_reset;

  __device__ __forceinline__ void load(const RecParams& p, const T* xs, bool want_q, int tok, int nb, int row_tok0, int h,
                                       int hk, int v0) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int n = 0; n < SB / NW; ++n) {
      const int j = warp + n * NW;
      const long key = ((long)(tok + j) * p.Hk + hk) * p.K, val = ((long)(tok + j) * p.H + h) * p.K;
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int c = lane + 32 * m;
        const bool ok = j < nb && c < p.K;
        q[n][m] = ok && want_q ? static_cast<const T*>(p.q)[key + c] : from_f32<T>(0.f);
        k[n][m] = ok ? static_cast<const T*>(p.k)[key + c] : from_f32<T>(0.f);
        if (p.k_read) kr[n][m] = ok ? static_cast<const T*>(p.k_read)[val + c] : from_f32<T>(0.f);
        if (p.gate == 2) g[n][m] = ok ? p.g[val + c] : 0.f;
      }
    }
#pragma unroll
    for (int m = 0; m < NX; ++m) {
      const int idx = threadIdx.x + m * NW * 32, j = idx / NC, c = idx - j * NC;
      x[m] = j < nb && v0 + c < p.V ? xs[((long)(tok + j) * p.H + h) * p.V + v0 + c] : from_f32<T>(0.f);
    }
    gs = 0.f, beta = 0.f, seg_reset = 0;
    if (threadIdx.x < nb) {
      const long t = (long)(tok + threadIdx.x) * p.H + h;
      if (p.gate == 1) gs = p.g[t];
      beta = p.delta ? p.beta[t] : 1.f;
      seg_reset = p.rows.resets(tok + threadIdx.x, row_tok0) ? 1 : 0;
    }
  }

  __device__ __forceinline__ void commit(const RecParams& p, WalkSmem<KL>& s, bool want_q, int nb) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int n = 0; n < SB / NW; ++n) {
      const int j = warp + n * NW;
      float qf[M], kf[M];
      float sq = 0.f, sk = 0.f;
#pragma unroll
      for (int m = 0; m < M; ++m) {
        qf[m] = to_f32(q[n][m]), kf[m] = to_f32(k[n][m]);
        sq += qf[m] * qf[m], sk += kf[m] * kf[m];
      }
      if (p.l2norm) {  // the reference rounds the normalised tensors to the input dtype (reference.py:69)
        const float iq = rsqrtf(warp_sum(sq) + 1e-6f), ik = rsqrtf(warp_sum(sk) + 1e-6f);
#pragma unroll
        for (int m = 0; m < M; ++m) {
          qf[m] = to_f32(from_f32<T>(qf[m] * iq));
          kf[m] = to_f32(from_f32<T>(kf[m] * ik));
        }
      }
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int c = lane + 32 * m;
        if (c >= WalkSmem<KL>::KP) break;
        if (want_q) s.q[j][c] = qf[m];
        s.k[j][c] = kf[m];
        if (p.k_read) s.kr[j][c] = to_f32(kr[n][m]);
        if (p.gate == 2) s.e[j][c] = expf(g[n][m]);
      }
    }
#pragma unroll
    for (int m = 0; m < NX; ++m) {
      const int idx = threadIdx.x + m * NW * 32;
      if (idx < SB * NC) s.x[idx / NC][idx % NC] = to_f32(x[m]);
    }
    if (threadIdx.x < 32) {
      const unsigned any = __ballot_sync(0xffffffffu, seg_reset);
      if (threadIdx.x < SB) {
        s.es[threadIdx.x] = p.gate == 1 && threadIdx.x < nb ? expf(gs) : 1.f;
        s.bs[threadIdx.x] = beta;
        s.rs[threadIdx.x] = seg_reset;
      }
      if (threadIdx.x == 0) s.any_reset = any != 0;
    }
  }
};

// (packed: the walks issue half the arithmetic instructions, which is what is left of a token next to its chain)
constexpr int KP2 = KPT / 2;
typedef f32x2 Chan[KP2];  // the channels of a thread

__device__ __forceinline__ float dot(const Chan& a, const Chan& b) {
  f32x2 s[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) s[i] = mul2(a[i], b[i]);
#pragma unroll
  for (int i = 4; i < KP2; ++i) s[i & 3] = fma2(a[i], b[i], s[i & 3]);
  const float2 x = unpack2f(add2(add2(s[0], s[1]), add2(s[2], s[3])));
  return x.x + x.y;
}
__device__ __forceinline__ void axpy(Chan& S, const Chan& a, float u) {
  const f32x2 uu = pack2f(u, u);
#pragma unroll
  for (int i = 0; i < KP2; ++i) S[i] = fma2(a[i], uu, S[i]);
}
__device__ __forceinline__ void scale_by(Chan& S, float e) {
  const f32x2 ee = pack2f(e, e);
#pragma unroll
  for (int i = 0; i < KP2; ++i) S[i] = mul2(S[i], ee);
}
__device__ __forceinline__ void scale_by(Chan& S, const Chan& e) {
#pragma unroll
  for (int i = 0; i < KP2; ++i) S[i] = mul2(S[i], e[i]);
}
__device__ __forceinline__ void clear(Chan& S) {
#pragma unroll
  for (int i = 0; i < KP2; ++i) S[i] = 0;
}

// A thread's place in a walk: key lane kl of column v; channel of its entry i (16-byte shared-memory reads of the KL
// lanes are neighbours).
template <int KL>
struct Lane {
  int kl, col, v;
  bool active;
  __device__ __forceinline__ Lane(int v0, int V) {
    const int lane = threadIdx.x & 31;
    kl = lane % KL;
    col = (threadIdx.x >> 5) * (32 / KL) + lane / KL;
    v = v0 + col;
    active = v < V;
  }
  __device__ __forceinline__ int channel(int i) const { return (i >> 2) * (4 * KL) + kl * 4 + (i & 3); }
  __device__ __forceinline__ void read(const float* src, Chan& dst) const {
#pragma unroll
    for (int i = 0; i < KPT; i += 4) {
      const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(src + channel(i));
      dst[i / 2] = x.x, dst[i / 2 + 1] = x.y;
    }
  }
  __device__ __forceinline__ void load_state(const float* src, int K, int V, Chan& S) const {
#pragma unroll
    for (int i = 0; i < KPT; i += 2) {
      const bool ok = src && active && channel(i) < K;  // (K is even)
      const float* at = src + (long)channel(i) * V + v;
      S[i / 2] = ok ? pack2f(at[0], at[V]) : 0;
    }
  }
  __device__ __forceinline__ void store_state(float* dst, int K, int V, const Chan& S) const {
#pragma unroll
    for (int i = 0; i < KPT; i += 2) {
      if (!active || channel(i) >= K) continue;
      float* at = dst + (long)channel(i) * V + v;
      const float2 x = unpack2f(S[i / 2]);
      at[0] = x.x, at[V] = x.y;
    }
  }
};

// What a walk does per token, fixed at compile time so that the eight staged tokens are one straight line of code (the
// key vectors of a token are then read while the token before it waits for its shuffles; with run-time branches in the
// token body the fp32 walk of K = V = 64 took 326 ns a token).
enum { kHeadDecay = 0, kHeadDelta = 1, kChannelDelta = 2 };  // scalar (or no) gate; with the delta rule; per key channel
template <int MODE>
struct Walk {
  static constexpr bool delta = MODE != kHeadDecay, channels = MODE == kChannelDelta;
};

// Forward walk of one row, head and block of value columns. OP: writes o and the final state; otherwise the checkpoints
// and the residuals v_t - r_t that the gradients start from.
template <typename T, int KL, int MODE, bool OP>
__device__ __forceinline__ void forward_walk(const RecParams& p, WalkSmem<KL>& s, int r, int h, int v0) {
  using W = Walk<MODE>;
  const int K = p.K, V = p.V, hk = h / (p.H / p.Hk);
  int tok0, len;
  p.rows.range(r, tok0, len);
  const Lane<KL> me(v0, V);
  Chan S;
  me.load_state(p.h0 ? p.h0 + ((long)r * p.H + h) * K * V : nullptr, K, V, S);
  float* ckpt = nullptr;
  if (!OP) {
    const long slot = p.slot0(r, tok0);
    ckpt = p.s_ckpt + ((long)(h - p.head0) * p.slots + slot) * K * V;
    if (h == p.head0 && v0 == 0) {
      for (int b = threadIdx.x; b * TB < len; b += NW * 32) p.slot_row[slot + b] = r;
    }
  }
  const float(*read_key)[WalkSmem<KL>::KP] = p.k_read ? s.kr : s.k;
  Stage<T, KL> st;
  st.load(p, static_cast<const T*>(p.v), OP, tok0, min(SB, len), tok0, h, hk, v0);
  for (int t0 = 0; t0 < len; t0 += SB) {
    const int nb = min(SB, len - t0);
    __syncthreads();
    st.commit(p, s, OP, nb);
    __syncthreads();
    if (t0 + SB < len) {
      st.load(p, static_cast<const T*>(p.v), OP, tok0 + t0 + SB, min(SB, len - t0 - SB), tok0, h, hk, v0);
    }
    if (!OP && t0 % TB == 0) me.store_state(ckpt + (long)(t0 / TB) * K * V, K, V, S);
    float out[SB];  // this thread's share of q_t S_t, or v_t - r_t
    Chan e, w, k, q, e1, w1, k1, q1;  // this token's vectors and the next one's, read a token ahead of their use
    auto fetch = [&](int j, Chan& e, Chan& w, Chan& k, Chan& q) {
      if (W::channels) me.read(s.e[j], e);
      if (W::delta) me.read(read_key[j], w);
      me.read(s.k[j], k);
      if (OP) me.read(s.q[j], q);
    };
    auto token = [&](int j, bool resets, Chan& e, Chan& w, Chan& k, Chan& q) {
      if (resets && s.rs[j]) clear(S);
      if (W::channels) scale_by(S, e);
      else scale_by(S, s.es[j]);
      float u = s.x[j][me.col];
      if (W::delta) {
        u -= key_sum<KL>(dot(w, S));
        if (!OP) out[j] = u;
        u *= s.bs[j];
      }
      axpy(S, k, u);
      if (OP) out[j] = dot(q, S);
    };
    auto tokens = [&](auto with_resets) {
      fetch(0, e, w, k, q);
#pragma unroll
      for (int j = 0; j < SB; j += 2) {
        fetch(j + 1, e1, w1, k1, q1);
        token(j, decltype(with_resets)::value, e, w, k, q);
        if (j + 2 < SB) fetch(j + 2, e, w, k, q);
        token(j + 1, decltype(with_resets)::value, e1, w1, k1, q1);
      }
    };
    if (s.any_reset) tokens(std::true_type{});
    else tokens(std::false_type{});
    const long at = ((long)(tok0 + t0) * p.H + h) * V + me.v, next = (long)p.H * V;
    if (OP) {
#pragma unroll
      for (int j = 0; j < SB; ++j) out[j] = key_sum<KL>(out[j]);
    }
    if ((OP || W::delta) && me.kl == 0 && me.active) {
#pragma unroll
      for (int j = 0; j < SB; ++j) {
        if (j < nb) {
          if (OP) static_cast<T*>(p.o)[at + j * next] = from_f32<T>(p.scale * out[j]);
          else p.resid[at + j * next] = out[j];
        }
      }
    }
  }
  if (OP && p.final_state) me.store_state(p.final_state + ((long)r * p.H + h) * K * V, K, V, S);
}

// Reverse walk of the state gradient, with a checkpoint of what comes from behind every block:
//   dS += scale q_t^T do_t;  du_t = k_t dS;  dv_t = beta_t du_t, dr_t = -beta_t du_t;
//   dS_{t-1} = exp(g_t) (dS + k_t^T dr_t)  (zero across a reset).
template <typename T, int KL, int MODE>
__device__ __forceinline__ void reverse_walk(const RecParams& p, WalkSmem<KL>& s, int r, int h, int v0) {
  using W = Walk<MODE>;
  const int K = p.K, V = p.V, hk = h / (p.H / p.Hk);
  int tok0, len;
  p.rows.range(r, tok0, len);
  const Lane<KL> me(v0, V);
  Chan dS;
  me.load_state(p.d_final ? p.d_final + ((long)r * p.H + h) * K * V : nullptr, K, V, dS);
  float* ckpt = p.ds_ckpt + ((long)(h - p.head0) * p.slots + p.slot0(r, tok0)) * K * V;
  const float(*read_key)[WalkSmem<KL>::KP] = p.k_read ? s.kr : s.k;
  Stage<T, KL> st;
  const int last = len > 0 ? (len - 1) / SB * SB : -SB;
  if (len > 0) st.load(p, static_cast<const T*>(p.d_o), true, tok0 + last, len - last, tok0, h, hk, v0);
  for (int t0 = last; t0 >= 0; t0 -= SB) {
    const int nb = min(SB, len - t0);
    __syncthreads();
    st.commit(p, s, true, nb);
    __syncthreads();
    if (t0 > 0) st.load(p, static_cast<const T*>(p.d_o), true, tok0 + t0 - SB, SB, tok0, h, hk, v0);
    if ((t0 + SB) % TB == 0 || t0 == last) me.store_state(ckpt + (long)(t0 / TB) * K * V, K, V, dS);
    float out[SB];  // du_t
    Chan e, w, k, q, e1, w1, k1, q1;
    auto fetch = [&](int j, Chan& e, Chan& w, Chan& k, Chan& q) {
      me.read(s.q[j], q);
      me.read(s.k[j], k);
      if (W::delta) me.read(read_key[j], w);
      if (W::channels) me.read(s.e[j], e);
    };
    auto token = [&](int j, bool resets, Chan& e, Chan& w, Chan& k, Chan& q) {
      axpy(dS, q, p.scale * s.x[j][me.col]);
      out[j] = key_sum<KL>(dot(k, dS));
      if (W::delta) axpy(dS, w, -s.bs[j] * out[j]);
      if (W::channels) scale_by(dS, e);
      else scale_by(dS, s.es[j]);
      if (resets && s.rs[j]) clear(dS);
    };
    auto tokens = [&](auto with_resets) {
      fetch(SB - 1, e, w, k, q);
#pragma unroll
      for (int j = SB - 1; j >= 0; j -= 2) {
        fetch(j - 1, e1, w1, k1, q1);
        token(j, decltype(with_resets)::value, e, w, k, q);
        if (j >= 2) fetch(j - 2, e, w, k, q);
        token(j - 1, decltype(with_resets)::value, e1, w1, k1, q1);
      }
    };
    if (s.any_reset) tokens(std::true_type{});
    else tokens(std::false_type{});
    if (me.kl == 0 && me.active) {
      const long at = ((long)(tok0 + t0) * p.H + h) * V + me.v, next = (long)p.H * V;
#pragma unroll
      for (int j = 0; j < SB; ++j) {
        if (j < nb) {
          static_cast<T*>(p.dv)[at + j * next] = from_f32<T>(W::delta ? s.bs[j] * out[j] : out[j]);
          if (W::delta) p.du[at + j * next] = out[j];
        }
      }
    }
  }
  if (p.dh0) me.store_state(p.dh0 + ((long)r * p.H + h) * K * V, K, V, dS);
}

// grid: (heads * column blocks, rows)
template <typename T, int KL, int MODE>
__global__ void __launch_bounds__(NW * 32) rec_fwd_kernel(RecParams p) {
  __shared__ __align__(16) WalkSmem<KL> s;
  const int h = p.head0 + blockIdx.x % p.heads, v0 = blockIdx.x / p.heads * WalkSmem<KL>::NC;
  forward_walk<T, KL, MODE, true>(p, s, blockIdx.y, h, v0);
}

// grid: (2 * heads * column blocks, rows); the two walks are independent of each other
template <typename T, int KL, int MODE>
__global__ void __launch_bounds__(NW * 32) rec_bwd_kernel(RecParams p) {
  __shared__ __align__(16) WalkSmem<KL> s;
  const int x = blockIdx.x >> 1, h = p.head0 + x % p.heads, v0 = x / p.heads * WalkSmem<KL>::NC;
  if (blockIdx.x & 1) reverse_walk<T, KL, MODE>(p, s, blockIdx.y, h, v0);
  else forward_walk<T, KL, MODE, false>(p, s, blockIdx.y, h, v0);
}

// Gradients of q, k (and the read key) and of the gates for the TB tokens of one block and one head, from the state S0
// entering the block, the state gradient dE coming from behind it and the per-token vectors do, dr = -beta du and
// u = beta (v - r). With e_t the decay of token t (the products below stop at a reset):
//   dq_t  = scale [ (prod_{s<=t} e_s) S0 do_t + sum_{j<=t} (prod_{j<s<=t} e_s) k_j (u_j . do_t) ]      (= scale S_t do_t)
//   dkr_t =         (prod_{s<=t} e_s) S0 dr_t + sum_{j<t}  (prod_{j<s<=t} e_s) k_j (u_j . dr_t)        (= S'_t dr_t)
//   dku_t = (prod_{s>t} e_s) dE u_t + sum_{i>=t} (prod_{t<s<=i} e_s) [scale q_i (do_i . u_t) + (i > t) kr_i (dr_i . u_t)]
//   dbeta_t = du_t . (v_t - r_t)
//   dg_t = <dS'_t, S'_t> = sum over the pairs j < t <= i of A_ji,
//          A_ji = (prod_{j<s<=i} e_s) k_j (scale q_i (u_j . do_i) + kr_i (u_j . dr_i))   per channel,
//          with S0 in the place of an earlier token's k_j u_j and dE in that of a later one's reads; summed over channels
//          for scalar gates
// Products of decays, never quotients, so any decay is safe, and dg as a sum of the terms that pass through token t: the
// running sum of q_t dq_t - k_t dku_t + kr_t dkr_t gives the same numbers from differences of terms that do not, which lost
// what a strong decay leaves of dg (relative error of its entries, median: 3e-4 where decays of e^-12 and e^-0.05
// alternate, against 2e-7). Latency hides behind the other blocks of the grid: (tokens / TB) * H CTAs where the walks have
// one CTA per columns block.
struct GradSmem {
  int K, V, vs;  // K padded to whole channel tiles; vs: row stride of the value vectors
  float *q, *k, *kr, *e, *d, *r, *u, *ts, *te, *ud, *ur, *udt, *urt, *es;
  float* dl;  // [4 token groups][TB][CT] shares of dg, over ts | te once a channel tile's products are formed
  __host__ __device__ static size_t floats(int K, int V) {
    const int kp = (K + CT - 1) / CT * CT;
    return 4 * TB * (size_t)kp + 3 * TB * (size_t)(V + 4) + 2 * CT * VTS + 4 * TB * TB + TB;
  }
  __device__ GradSmem(float* base, int k_dim, int v_dim) {
    const int kp = (k_dim + CT - 1) / CT * CT;
    K = kp, V = v_dim, vs = v_dim + 4;
    q = base, k = q + TB * kp, kr = k + TB * kp, e = kr + TB * kp;
    d = e + TB * kp, r = d + TB * vs, u = r + TB * vs;
    ts = u + TB * vs, te = ts + CT * VTS;
    ud = te + CT * VTS, ur = ud + TB * TB, udt = ur + TB * TB, urt = udt + TB * TB, es = urt + TB * TB;
    dl = ts;
    static_assert(4 * TB * CT <= 2 * CT * VTS, "the shares of dg fit over the staged states");
  }
};

template <typename T>
__global__ void __launch_bounds__(GT) block_grads_kernel(RecParams p) {
  extern __shared__ __align__(16) float smem_raw[];
  const int K = p.K, V = p.V, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int hl = blockIdx.x % p.heads, h = p.head0 + hl, hk = h / (p.H / p.Hk);
  const long slot = blockIdx.x / p.heads;
  const int row = p.slot_row[slot];
  if (row < 0 || row >= p.rows.count()) return;
  int tok0, len;
  p.rows.range(row, tok0, len);
  const long b = slot - p.slot0(row, tok0);
  if (b < 0 || b * TB >= len) return;
  const int n = min(TB, len - (int)b * TB), tok = tok0 + (int)b * TB;
  const GradSmem s(smem_raw, K, V);
  __shared__ unsigned resets_s;

  // ---- the block's vectors; tokens behind the row's end are zeros with decay 1
#pragma unroll 4
  for (int idx = tid; idx < TB * s.K; idx += GT) {
    const int t = idx / s.K, c = idx - t * s.K;
    const bool ok = t < n && c < K;
    const long key = ((long)(tok + t) * p.Hk + hk) * K + c, kv = ((long)(tok + t) * p.H + h) * K + c;
    const float k = ok ? to_f32(static_cast<const T*>(p.k)[key]) : 0.f;
    s.q[idx] = ok ? to_f32(static_cast<const T*>(p.q)[key]) : 0.f;
    s.k[idx] = k;
    s.e[idx] = ok && p.gate == 2 ? expf(p.g[kv]) : 1.f;
    s.kr[idx] = ok && p.k_read ? to_f32(static_cast<const T*>(p.k_read)[kv]) : k;
  }
#pragma unroll 4
  for (int idx = tid; idx < TB * V; idx += GT) {
    const int t = idx / V, c = idx - t * V, at = t * s.vs + c;
    const long src = ((long)(tok + t) * p.H + h) * V + c;
    s.d[at] = t < n ? to_f32(static_cast<const T*>(p.d_o)[src]) : 0.f;
    s.r[at] = t < n && p.delta ? p.du[src] : 0.f;
    s.u[at] = t >= n ? 0.f : p.delta ? p.resid[src] : to_f32(static_cast<const T*>(p.v)[src]);
  }
  if (warp == 0) {
    const bool in = lane < n;
    if (lane < TB) s.es[lane] = in && p.gate == 1 ? expf(p.g[(long)(tok + lane) * p.H + h]) : 1.f;
    const unsigned bits = __ballot_sync(0xffffffffu, in && p.rows.resets(tok + lane, tok0));
    if (lane == 0) resets_s = bits;
  }
  __syncthreads();
  if (p.l2norm || p.delta) {
    for (int t = warp; t < n; t += GT / 32) {
      if (p.l2norm) {  // the reference rounds the normalised tensors to the input dtype (reference.py:69)
        float sq = 0.f, sk = 0.f;
        for (int c = lane; c < s.K; c += 32) {
          const float q = s.q[t * s.K + c], k = s.k[t * s.K + c];
          sq += q * q, sk += k * k;
        }
        const float iq = rsqrtf(warp_sum(sq) + 1e-6f), ik = rsqrtf(warp_sum(sk) + 1e-6f);
        for (int c = lane; c < s.K; c += 32) {
          s.q[t * s.K + c] = to_f32(from_f32<T>(s.q[t * s.K + c] * iq));
          s.k[t * s.K + c] = to_f32(from_f32<T>(s.k[t * s.K + c] * ik));
          if (!p.k_read) s.kr[t * s.K + c] = s.k[t * s.K + c];
        }
      }
      if (p.delta) {  // du, v - r  ->  -beta du, beta (v - r), and their product's sum on the way
        const long th = (long)(tok + t) * p.H + h;
        const float beta = p.beta[th];
        float db = 0.f;
        for (int c = lane; c < V; c += 32) {
          const float du = s.r[t * s.vs + c], x = s.u[t * s.vs + c];
          s.r[t * s.vs + c] = -beta * du, s.u[t * s.vs + c] = beta * x;
          db += du * x;
        }
        db = warp_sum(db);
        if (lane == 0) p.dbeta[th] = db;
      }
    }
    __syncthreads();
  }
  const unsigned resets = resets_s;

  {  // u_j . do_t and u_j . dr_t, one pair (j, t) a thread
    const int j = tid / TB, t = tid % TB;
    float at = 0.f, ct = 0.f;
    for (int x0 = 0; x0 < V; x0 += VT / 2) {  // (sums of short sums: the rounding of a long chain would show in dq and dg)
      float a[4] = {}, c[4] = {};
#pragma unroll
      for (int x = x0; x < min(V, x0 + VT / 2); x += 4) {
        const float4 u = *reinterpret_cast<const float4*>(s.u + j * s.vs + x);
        const float4 d = *reinterpret_cast<const float4*>(s.d + t * s.vs + x);
        const float4 r = *reinterpret_cast<const float4*>(s.r + t * s.vs + x);
        a[0] += u.x * d.x, a[1] += u.y * d.y, a[2] += u.z * d.z, a[3] += u.w * d.w;
        c[0] += u.x * r.x, c[1] += u.y * r.y, c[2] += u.z * r.z, c[3] += u.w * r.w;
      }
      at += (a[0] + a[1]) + (a[2] + a[3]), ct += (c[0] + c[1]) + (c[2] + c[3]);
    }
    s.udt[t * TB + j] = s.ud[tid] = at;
    s.urt[t * TB + j] = s.ur[tid] = ct;
  }

  const float* S0 = p.s_ckpt + ((long)hl * p.slots + slot) * K * V;
  const float* dE = p.ds_ckpt + ((long)hl * p.slots + slot) * K * V;
  const int cl = tid % CT, tg = tid / CT, tq = 4 * tg;  // channel of the tile; this thread's tokens are tq .. tq + 3
  double gsum = 0.;                                     // scalar gates: a sixteenth of dg of token tid / 16
  for (int c0 = 0; c0 < K; c0 += CT) {
    // ---- S0 do_t, S0 dr_t, dE u_t for the tile's channels, and a quarter of <dE, S0>
    float ad[4] = {}, ar[4] = {}, au[4] = {}, en = 0.f;
    for (int x0 = 0; x0 < V; x0 += VT) {
      __syncthreads();
#pragma unroll
      for (int idx = tid; idx < CT * VT / 4; idx += GT) {
        const int c = idx / (VT / 4), x = idx % (VT / 4) * 4;
        const bool ok = c0 + c < K && x0 + x < V;
        const long at = (long)(c0 + c) * V + x0 + x;
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(s.ts + c * VTS + x) = ok ? *reinterpret_cast<const float4*>(S0 + at) : z;
        *reinterpret_cast<float4*>(s.te + c * VTS + x) = ok ? *reinterpret_cast<const float4*>(dE + at) : z;
      }
      __syncthreads();
      const int xe = min(VT, V - x0);
#pragma unroll
      for (int xh = 0; xh < VT; xh += VT / 2) {  // (short sums here too)
        float td[4] = {}, tr[4] = {}, tu[4] = {}, tn = 0.f;
#pragma unroll
        for (int x = xh; x < xh + VT / 2; x += 4) {
          if (x >= xe) break;
          const float4 a = *reinterpret_cast<const float4*>(s.ts + cl * VTS + x);
          const float4 g = *reinterpret_cast<const float4*>(s.te + cl * VTS + x);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int at = (tq + i) * s.vs + x0 + x;
            const float4 d = *reinterpret_cast<const float4*>(s.d + at);
            const float4 r = *reinterpret_cast<const float4*>(s.r + at);
            const float4 u = *reinterpret_cast<const float4*>(s.u + at);
            td[i] += (a.x * d.x + a.y * d.y) + (a.z * d.z + a.w * d.w);
            tr[i] += (a.x * r.x + a.y * r.y) + (a.z * r.z + a.w * r.w);
            tu[i] += (g.x * u.x + g.y * u.y) + (g.z * u.z + g.w * u.w);
          }
          if ((x / 4 & 3) == tg) tn += (g.x * a.x + g.y * a.y) + (g.z * a.z + g.w * a.w);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) ad[i] += td[i], ar[i] += tr[i], au[i] += tu[i];
        en += tn;
      }
    }
    // ---- the in-block terms of this thread's channel and four tokens; the products of decays grow one token at a time
    const int c = c0 + cl;
    float w[4] = {1.f, 1.f, 1.f, 1.f}, dq[4] = {}, dkr[4] = {}, dk[4] = {};
    // Of dg: A_ji of this thread's tokens i passes through the tokens j + 1 .. i. For the tokens up to tq that is all four i,
    // whose sum is kept per j; behind tq, token tq + m takes those of i >= m.
    float pairs[TB - 1], behind[4] = {}, qs[4], krs[4];
    float odd_q[4], odd_r[4];  // terms join dq and dkr two at a time: half the roundings of the growing sums
#pragma unroll
    for (int i = 0; i < 4; ++i) qs[i] = p.scale * s.q[(tq + i) * s.K + c], krs[i] = s.kr[(tq + i) * s.K + c];
    auto add_pairs = [&](const float (&a)[4]) {
      const float a23 = a[2] + a[3], a13 = a[1] + a23;
      behind[1] += a13, behind[2] += a23, behind[3] += a[3];
      return a[0] + a13;
    };
#pragma unroll
    for (int j = TB - 1; j >= 0; --j) {  // from token j's predecessor into tokens t >= j
      const float e = p.gate == 2 ? s.e[j * s.K + c] : s.es[j];
      const bool cut = resets >> j & 1;
      const float kp = j > 0 ? s.k[(j - 1) * s.K + c] : 0.f;
      const int at = (j > 0 ? j - 1 : 0) * TB + tq;
      const float4 x = *reinterpret_cast<const float4*>(s.ud + at), y = *reinterpret_cast<const float4*>(s.ur + at);
      const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
      float a[4] = {};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float xq = 0.f, xr = 0.f;
        if (tq + i >= j) {
          w[i] = cut ? 0.f : w[i] * e;
          if (j > 0 && w[i] != 0.f) {
            xq = w[i] * kp * xs[i], xr = w[i] * kp * ys[i];
            a[i] = qs[i] * xq + krs[i] * xr;
          }
        }
        if (j & 1) odd_q[i] = xq, odd_r[i] = xr;
        else dq[i] += odd_q[i] + xq, dkr[i] += odd_r[i] + xr;
      }
      if (j > 0) {  // (a predecessor among this thread's own tokens does not pass through those up to itself)
        const int own = j - 1 - tq;
        if (own < 0) {
          pairs[j - 1] = add_pairs(a);
        } else {
          pairs[j - 1] = 0.f;
          if (own < 1) behind[1] += a[1] + (a[2] + a[3]);
          if (own < 2) behind[2] += a[2] + a[3];
          if (own < 3) behind[3] += a[3];
        }
      }
    }
    const float w0 = w[0];
    float first[4] = {};  // the entering state
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (w[i] != 0.f) {
        const float xq = w[i] * ad[i], xr = w[i] * ar[i];
        dq[i] += xq, dkr[i] += xr;
        first[i] = qs[i] * xq + krs[i] * xr;
      }
      w[i] = 1.f;
    }
    float upto = add_pairs(first);  // dg of the tokens up to tq, from the block's first token on
#pragma unroll 4
    for (int j = 1; j < TB; ++j) {  // what tokens j > t read of token t's write
      const float e = p.gate == 2 ? s.e[j * s.K + c] : s.es[j];
      const bool cut = resets >> j & 1;
      const float qj = p.scale * s.q[j * s.K + c], rj = s.kr[j * s.K + c];
      const float4 x = *reinterpret_cast<const float4*>(s.udt + j * TB + tq);
      const float4 y = *reinterpret_cast<const float4*>(s.urt + j * TB + tq);
      const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (tq + i < j) {
          w[i] = cut ? 0.f : w[i] * e;
          if (w[i] != 0.f) dk[i] += w[i] * (qj * xs[i] + rj * ys[i]);
        }
      }
    }
    float through = w0 * w[0] != 0.f ? w0 * w[0] * en : 0.f;  // <dE, S0> passes through every token of the block
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = tq + i;
      const float q = s.q[t * s.K + c], k = s.k[t * s.K + c], own = s.ud[t * TB + t];
      const float x = w[i] != 0.f ? w[i] * au[i] : 0.f;
      dk[i] += x;
      behind[i] += through;
      through += k * x;  // (token t's write passes through the tokens behind t on its way out of the block)
      if (i == 0) upto += behind[0];
      if (t < n && c < K) {
        const long at = ((long)(tok + t) * p.H + h) * K + c;
        const float dku = dk[i] + p.scale * q * own;
        p.dq_acc[at] = p.scale * (dq[i] + k * own);
        p.dk_acc[at] = p.k_read ? dku : dku + dkr[i];
        if (p.k_read) p.dkr_acc[at] = dkr[i];
      }
    }
    if (p.gate == 0) continue;
    __syncthreads();  // every thread is done with the staged states
#pragma unroll
    for (int t = 0; t < TB; ++t) {
      if (t > 0 && t <= tq) upto += pairs[t - 1];
      s.dl[(tg * TB + t) * CT + cl] = t <= tq ? upto : t - tq < 4 ? behind[t & 3] : through;
    }
    __syncthreads();
    if (p.gate == 2) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int at = (tq + i) * CT + cl;
        const float x = (s.dl[at] + s.dl[at + TB * CT]) + (s.dl[at + 2 * TB * CT] + s.dl[at + 3 * TB * CT]);
        if (tq + i < n && c < K) p.dg[((long)(tok + tq + i) * p.H + h) * K + c] = x;
      }
    } else {
#pragma unroll
      for (int m = 0; m < 16; ++m) gsum += s.dl[((m & 3) * TB + tid / 16) * CT + (m >> 2) * 16 + tid % 16];
    }
  }
  if (p.gate == 1) {
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) gsum += __shfl_xor_sync(0xffffffffu, gsum, off);
    if (tid % 16 == 0 && tid / 16 < n) p.dg[(long)(tok + tid / 16) * p.H + h] = (float)gsum;
  }
}

// Head sizes of the path: V columns times slices of 1, 2, 4 .. 128 key channels in at most 512 threads, whole warps.
bool covered(int K, int V) {
  for (int slice = 1; slice <= 128; slice *= 2) {
    if (K % slice == 0 && (long)V * (K / slice) <= 512 && V * (K / slice) % 32 == 0) return true;
  }
  return false;
}

// Key lanes per column: 16 channels a thread.
int pick_key_lanes(int K) { return K <= 32 ? 2 : K <= 64 ? 4 : K <= 128 ? 8 : 16; }

RecParams base_params(const jla_problem& p) {
  RecParams r{};
  r.rows = make_rows(p);
  r.H = p.H; r.Hk = p.Hk; r.K = p.K; r.V = p.V;
  r.head0 = 0; r.heads = p.H;
  r.gate = p.kind == JLA_KIND_DELTANET ? 0 : (p.kind == JLA_KIND_KDA ? 2 : 1);
  r.delta = p.kind != JLA_KIND_SIMPLE_GLA;
  r.l2norm = (p.flags & JLA_FLAG_QK_L2NORM) != 0;
  r.scale = p.scale;
  r.q = p.q; r.k = p.k; r.v = p.v; r.g = p.g; r.beta = p.beta; r.h0 = p.h0;
  r.k_read = p.k_read;
  return r;
}

template <typename T, int KL>
int launch_walks(const RecParams& rp, bool bwd, int rows, cudaStream_t stream) {
  const int blocks = (rp.V + WalkSmem<KL>::NC - 1) / WalkSmem<KL>::NC;
  ProfScope ps(bwd ? kProfRecBwd : kProfRecFwd, stream);
  const dim3 grid((unsigned)(rp.heads * blocks * (bwd ? 2 : 1)), (unsigned)rows);
  auto run = [&](auto* fwd, auto* back) { (bwd ? back : fwd)<<<grid, NW * 32, 0, stream>>>(rp); };
  if (!rp.delta) run(rec_fwd_kernel<T, KL, kHeadDecay>, rec_bwd_kernel<T, KL, kHeadDecay>);
  else if (rp.gate == 2) run(rec_fwd_kernel<T, KL, kChannelDelta>, rec_bwd_kernel<T, KL, kChannelDelta>);
  else run(rec_fwd_kernel<T, KL, kHeadDelta>, rec_bwd_kernel<T, KL, kHeadDelta>);
  JLA_LAUNCH_OK();
  return JLA_OK;
}

template <typename T>
int launch_t(const RecParams& rp, bool bwd, int rows, cudaStream_t stream) {
  int rc;
  switch (pick_key_lanes(rp.K)) {
    case 2: rc = launch_walks<T, 2>(rp, bwd, rows, stream); break;
    case 4: rc = launch_walks<T, 4>(rp, bwd, rows, stream); break;
    case 8: rc = launch_walks<T, 8>(rp, bwd, rows, stream); break;
    default: rc = launch_walks<T, 16>(rp, bwd, rows, stream); break;
  }
  if (rc != JLA_OK || !bwd) return rc;
  const size_t smem = GradSmem::floats(rp.K, rp.V) * sizeof(float);
  JLA_CUDA_OK(cudaFuncSetAttribute(block_grads_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  ProfScope ps(kProfRecGrads, stream);
  block_grads_kernel<T><<<(unsigned)(rp.slots * rp.heads), GT, smem, stream>>>(rp);
  JLA_LAUNCH_OK();
  return JLA_OK;
}

int launch_dtype(const RecParams& rp, int dtype, bool bwd, int rows, cudaStream_t stream) {
  switch (dtype) {
    case JLA_DTYPE_BF16: return launch_t<__nv_bfloat16>(rp, bwd, rows, stream);
    case JLA_DTYPE_F16: return launch_t<__half>(rp, bwd, rows, stream);
    case JLA_DTYPE_F32: return launch_t<float>(rp, bwd, rows, stream);
  }
  set_error("unknown dtype %d", dtype);
  return JLA_ERR_BAD_ARGUMENT;
}

struct BwdScratch {
  float *dq_acc, *dk_acc, *dkr_acc, *s_ckpt, *ds_ckpt, *resid, *du;
  int* slot_row;
  long slots;
  int heads;
  size_t bytes;
};

// The two checkpoint sets take K V / 2 bytes a token and head (twice what one walk with one set took, eight kilobytes at
// K = V = 128), so very long calls run a slice of the heads at a time through the same buffers: heads are independent, and
// the slices follow each other on the stream. The limit leaves a call of 180 GB the room that it had with one set, and
// sends no call of ordinary size through slices, which are walks one after the other.
constexpr size_t kMaxCheckpointBytes = 32ull << 30;

BwdScratch carve_bwd(const jla_problem& p, void* base) {
  Carver c(base);
  BwdScratch s;
  const long tokens = (long)p.B * p.T;
  const int rows = p.cu_seqlens || p.num_seqs ? p.num_seqs : p.B;
  const bool delta = p.kind != JLA_KIND_SIMPLE_GLA;
  s.slots = tokens / TB + rows + 1;
  s.dq_acc = c.take<float>((size_t)tokens * p.H * p.K);
  s.dk_acc = c.take<float>((size_t)tokens * p.H * p.K);
  s.dkr_acc = c.take<float>(p.k_read ? (size_t)tokens * p.H * p.K : 0);
  const size_t per_head = (size_t)s.slots * p.K * p.V;  // of one set, in floats
  const size_t fit = kMaxCheckpointBytes / (2 * sizeof(float) * per_head);
  const int slices = fit >= (size_t)p.H ? 1 : fit > 0 ? (int)((p.H + fit - 1) / fit) : p.H;
  s.heads = (p.H + slices - 1) / slices;
  s.s_ckpt = c.take<float>(s.heads * per_head);
  s.ds_ckpt = c.take<float>(s.heads * per_head);
  s.resid = c.take<float>(delta ? (size_t)tokens * p.H * p.V : 0);
  s.du = c.take<float>(delta ? (size_t)tokens * p.H * p.V : 0);
  s.slot_row = c.take<int>((size_t)s.slots);
  s.bytes = c.bytes();
  return s;
}

}  // namespace

const char* recurrent_unsupported(const jla_problem& p) {
  if (p.K > 256 || p.V > 256 || p.K % 8) return "recurrent path: K must be a multiple of 8 and K, V <= 256";
  if (p.V < 8 || (p.V & (p.V - 1))) return "recurrent path: V must be a power of two in [8, 256]";
  if (!covered(p.K, p.V)) return "recurrent path: no thread layout for this K, V";
  return nullptr;
}

size_t recurrent_bwd_scratch_bytes(const jla_problem& p) { return carve_bwd(p, nullptr).bytes; }

int recurrent_fwd(const jla_problem& p, const jla_fwd_io& io, cudaStream_t stream) {
  RecParams rp = base_params(p);
  rp.o = io.o;
  rp.final_state = io.final_state;
  const int rows = p.cu_seqlens ? p.num_seqs : p.B;
  if (rows == 0 || p.H == 0) return JLA_OK;
  return launch_dtype(rp, p.dtype, false, rows, stream);
}

int recurrent_bwd(const jla_problem& p, const jla_bwd_io& io, cudaStream_t stream) {
  RecParams rp = base_params(p);
  const BwdScratch s = carve_bwd(p, io.scratch);
  if (io.scratch_bytes < s.bytes) {
    set_error("backward scratch too small: %zu < %zu bytes", io.scratch_bytes, s.bytes);
    return JLA_ERR_WORKSPACE;
  }
  rp.d_o = io.d_o; rp.d_final = io.d_final;
  rp.dq_acc = s.dq_acc; rp.dk_acc = s.dk_acc; rp.dkr_acc = s.dkr_acc;
  rp.dv = io.dv; rp.dg = io.dg; rp.dbeta = io.dbeta; rp.dh0 = io.dh0;
  rp.s_ckpt = s.s_ckpt; rp.ds_ckpt = s.ds_ckpt; rp.resid = s.resid; rp.du = s.du;
  rp.slot_row = s.slot_row; rp.slots = s.slots;
  const int rows = p.cu_seqlens ? p.num_seqs : p.B;
  const long tokens = (long)p.B * p.T;
  for (rp.head0 = 0; rows > 0 && rp.head0 < p.H; rp.head0 += s.heads) {
    rp.heads = p.H - rp.head0 < s.heads ? p.H - rp.head0 : s.heads;
    const int rc = launch_dtype(rp, p.dtype, true, rows, stream);
    if (rc != JLA_OK) return rc;
  }
  const bool l2 = (p.flags & JLA_FLAG_QK_L2NORM) != 0;
  int rc = finalize_key_grad(s.dq_acc, p.q, io.dq, p.dtype, tokens, p.H, p.Hk, p.K, l2, stream);
  if (rc != JLA_OK) return rc;
  if (p.k_read) {  // one row per value head, used as passed: no group sum, no norm to differentiate through
    rc = finalize_key_grad(s.dkr_acc, nullptr, io.dk_read, p.dtype, tokens, p.H, p.H, p.K, false, stream);
    if (rc != JLA_OK) return rc;
  }
  return finalize_key_grad(s.dk_acc, p.k, io.dk, p.dtype, tokens, p.H, p.Hk, p.K, l2, stream);
}

}  // namespace jla
