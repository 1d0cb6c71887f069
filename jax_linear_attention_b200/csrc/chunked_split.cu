// Training forms of the mma.sync scalar-gate kernels (head sizes other than K = V = 128), split by what is serial:
//
//   forward   state pass, one CTA per (row, head, block of value columns):  W = V - (cin Gamma)(K S);  Vn = Ag W;
//             S+ = keep gamma S + K^T (tail Gamma_r Vn), leaving h (the state entering every chunk) and Vn behind;
//             then all outputs at once: O = scale [(cin Gamma)(Q h) + ((Q K^T) D) Vn]
//   backward  all Z = scale P^T dO at once (delta rule); the reverse state pass dVn = (tail Gamma_r)(K dS+) + Z;
//             dW = dV = Ag^T dVn; dS = keep gamma dS+ + Q^T (scale cin Gamma dO) - K^T (cin Gamma dW), leaving dh
//             (without the delta rule dV needs no state of its own and is the gradient kernel's, chunked_bwd.cu)
//
// A state pass walks a row's chunks, so its time is the number of chunks times the length of one chunk's chain of
// dependent products; the forms that also computed scores and outputs inside the walk took 6.8 us a chunk (24 chains of
// B3 T1000 H8 K = V = 64) and, two CTAs to an SM, 6.9 us a chunk and SM (512 chains of Mamba-2's B8 T2048 H64 P64 N128).
// Here the walk holds only the chain: three products and three barriers a chunk with the delta rule, one product and one
// barrier without, on four warps; the value columns of a state are independent, so a call with few chains runs them in
// blocks of VB. What is read back for the outputs (h, Vn) the backward keeps anyway. Forwards that keep nothing run the
// fused kernel (chunked_fwd.cu): it is slower, but its scratch holds neither (see chunked_api.cu).
//
// Measured: the walks of the d = 64 shape 23 + 29 us (fused, with outputs and scores, 109 + 119), of the Mamba-2 shape 139 +
// 137 us and its outputs 150 us (fused 439 + 436); what bounds them now is the latency of a chunk's loads, barriers and
// products at one to four CTAs of four warps an SM.
//
// 16-bit operands, fp32 accumulation, the carried state in fp32, Z in fp32. The reverse walk rounds the weighted query
// fragments (the weighted dO once did); in f16 the weights are lifted to the chunk's largest one first, see state_kernel.
#include <type_traits>

#include "chunked.cuh"
#include "profile.cuh"
#include "mma.cuh"

namespace jla {
namespace {

constexpr int NT = 128;  // threads of every kernel here: four warps, 16 token rows each

// ---------------------------------------------------------------------------------------------------------
// state passes
struct StateParams {
  const ChunkMeta* meta;
  const int2* row_chunks;
  const float* gates;
  const unsigned char* runs;
  const void *q, *k, *x, *ag;  // x: v, or the upstream gradient (backward)
  const float* z;              // [chunk slot, H, 64, V] f32 (backward, delta rule)
  const float* first;          // the state a row starts from (h0, or d_final), or nullptr
  float* last;                 // the state a row ends with (final_state, or dh0), or nullptr
  void* h;                     // [chunk slot, H, K, V]: the state entering a chunk (backward: dS+ coming from behind it)
  void* vn;                    // [chunk slot, H, 64, V]: Vn (backward: dVn); delta rule
  void* dv;                    // [tokens, H, V] (backward, delta rule)
  int H, Hk, V;
  float scale;
};

template <typename T, int K, int VB, bool DELTA, bool BWD>
struct StateSmem {
  static constexpr int LDK = K + 8, LDV = VB + 8, LDC = 72;
  static constexpr bool kQ = BWD, kK = DELTA || !BWD;  // tiles a stage holds
  static constexpr int kStageElems = ((kQ ? 1 : 0) + (kK ? 1 : 0)) * 64 * LDK + 64 * LDV + (DELTA ? 64 * LDC : 0);
  static constexpr int kStageBytes = kStageElems * 2 + 512 + 64;  // + gates (128 f32) + runs (64 u8)
  static constexpr int kTiles = DELTA ? K * LDV + 3 * 64 * LDV : 0;
  static constexpr int kBytes = 2 * kStageBytes + kTiles * 2;
};

template <typename T, int K, int VB, bool DELTA, bool BWD>
__global__ void __launch_bounds__(NT) state_kernel(StateParams p) {
  using L = StateSmem<T, K, VB, DELTA, BWD>;
  constexpr int LDK = L::LDK, LDV = L::LDV, LDC = L::LDC;
  constexpr int NTV = VB / 8;   // n-tiles across the value columns
  constexpr int MT = K / 64;    // 16-row tiles of the state per warp
  // f16 backward: the weights scale (cin Gamma) of a chunk that starts behind a strong decay would push the weighted query
  // fragments below the type's normal range (unit rows behind e^-8: the chunk's share of dS off by 8e-3). They are carried
  // relative to the power of two above the largest one, which the fp32 accumulators take out again.
  constexpr bool kLift = BWD && std::is_same<T, __half>::value;
  const int vblocks = p.V / VB;
  const int v0 = (blockIdx.x % vblocks) * VB, rh = blockIdx.x / vblocks;
  const int row = rh / p.H, h = rh - row * p.H, hk = h / (p.H / p.Hk);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int r0 = 16 * warp, sr0 = 16 * MT * warp;
  const int2 rc = p.row_chunks[row];

  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto stage = [&](int s) { return reinterpret_cast<T*>(smem_raw + s * L::kStageBytes); };
  auto stage_q = [&](int s) { return stage(s); };
  auto stage_k = [&](int s) { return stage(s) + (L::kQ ? 64 * LDK : 0); };
  auto stage_x = [&](int s) { return stage_k(s) + (L::kK ? 64 * LDK : 0); };
  auto stage_ag = [&](int s) { return stage_x(s) + 64 * LDV; };
  auto stage_g = [&](int s) { return reinterpret_cast<float*>(smem_raw + s * L::kStageBytes + L::kStageElems * 2); };
  auto stage_runs = [&](int s) { return reinterpret_cast<unsigned char*>(stage_g(s) + 128); };
  T* Sb = reinterpret_cast<T*>(smem_raw + 2 * L::kStageBytes);  // 16-bit copy of the carried state
  T* A1 = Sb + K * LDV;    // W; backward -(cin Gamma) dW
  T* A2 = A1 + 64 * LDV;   // Vn, dVn
  T* A3 = A2 + 64 * LDV;   // (tail Gamma_r) Vn

  auto issue_load = [&](int ci, int s, const ChunkMeta& m) {
    const int c = rc.x + ci;
    const long key = ((long)m.tok0 * p.Hk + hk) * K;
    if (L::kQ) load_tile_async<T, 64, K>(stage_q(s), LDK, static_cast<const T*>(p.q) + key, (long)p.Hk * K, m.len, tid, NT);
    if (L::kK) load_tile_async<T, 64, K>(stage_k(s), LDK, static_cast<const T*>(p.k) + key, (long)p.Hk * K, m.len, tid, NT);
    load_tile_async<T, 64, VB>(stage_x(s), LDV, static_cast<const T*>(p.x) + ((long)m.tok0 * p.H + h) * p.V + v0,
                               (long)p.H * p.V, m.len, tid, NT);
    if (DELTA) {
      load_tile_async<T, 64, 64>(stage_ag(s), LDC, static_cast<const T*>(p.ag) + ((long)c * p.H + h) * 4096, 64, 64, tid, NT);
    }
    if (tid < 32) cp_async16(stage_g(s) + tid * 4, p.gates + ((long)c * p.H + h) * 128 + tid * 4);
    if (tid >= 32 && tid < 36) cp_async16(stage_runs(s) + (tid - 32) * 16, p.runs + (long)c * 64 + (tid - 32) * 16);
    cp_async_commit();
  };
  float z[BWD && DELTA ? NTV : 1][4];  // Z of the next chunk to come, in accumulator fragments
  auto load_z = [&](int ci) {
    const float* src = p.z + ((long)(rc.x + ci) * p.H + h) * 64 * p.V + (long)(r0 + g) * p.V + v0 + 2 * t;
#pragma unroll
    for (int nt = 0; nt < (BWD && DELTA ? NTV : 0); ++nt) {
      const float2 lo = *reinterpret_cast<const float2*>(src + nt * 8);
      const float2 hi = *reinterpret_cast<const float2*>(src + 8 * p.V + nt * 8);
      z[nt][0] = lo.x, z[nt][1] = lo.y, z[nt][2] = hi.x, z[nt][3] = hi.y;
    }
  };

  float acc[MT][NTV][4];  // the carried state: rows sr0 + 16 mt + g (+8), columns 8 nt + 2t (+1) of the block
  const float* first = p.first ? p.first + ((long)row * p.H + h) * K * p.V + v0 : nullptr;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
    for (int nt = 0; nt < NTV; ++nt) {
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        float2 x = make_float2(0.f, 0.f);
        if (first) x = *reinterpret_cast<const float2*>(first + (long)(sr0 + 16 * mt + g + 8 * hh) * p.V + nt * 8 + 2 * t);
        acc[mt][nt][2 * hh] = x.x, acc[mt][nt][2 * hh + 1] = x.y;
      }
    }
    if (DELTA) store_acc<T, NTV>(Sb, LDV, sr0 + 16 * mt, 0, acc[mt], lane);
  }
  const int n = rc.y;
  auto chunk_at = [&](int it) { return BWD ? n - 1 - it : it; };
  // table entries of this chunk, of the next one (whose loads it addresses) and of the one after, read a chunk ahead
  ChunkMeta m{}, m1{}, m2{};
  if (n > 0) m1 = p.meta[rc.x + chunk_at(0)];
  if (n > 1) m2 = p.meta[rc.x + chunk_at(1)];
  if (n > 0) {
    issue_load(chunk_at(0), 0, m1);
    if (BWD && DELTA) load_z(chunk_at(0));
  }

  for (int it = 0; it < n; ++it) {
    const int s = it & 1, c = rc.x + chunk_at(it);
    cp_async_wait<0>();
    __syncthreads();  // the stage has landed, Sb holds the state, the other stage is free
    m = m1, m1 = m2;
    if (it + 1 < n) issue_load(chunk_at(it + 1), s ^ 1, m1);
    if (it + 2 < n) m2 = p.meta[rc.x + chunk_at(it + 2)];
    const float* Gs = stage_g(s);
    const unsigned char* runs = stage_runs(s);
    const float kg = keep_gamma(Gs, runs, m.flags);
    T* hout = static_cast<T*>(p.h) + ((long)c * p.H + h) * K * p.V + v0;
    // the per-token weight of the update that is applied to the key or query fragments, in the (here unused) beta half
    // of the gate vectors: tail Gamma_r forward, scale (cin Gamma) backward; a barrier follows before its readers
    float lift = 1.f, unlift = 1.f;
    if (kLift) {
      const float a = p.scale * row_scalars(Gs, runs, m.flags, lane).gam;
      const float b = p.scale * row_scalars(Gs, runs, m.flags, lane + 32).gam;
      const unsigned e = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(fabsf(a), fabsf(b)))) >> 23;
      if (e > 0 && e < 253) lift = __uint_as_float((253 - e) << 23), unlift = __uint_as_float((e + 1) << 23);
    }
    if ((BWD || !DELTA) && tid < 64) {
      const RowScalars r = row_scalars(Gs, runs, m.flags, tid);
      stage_g(s)[64 + tid] = BWD ? p.scale * r.gam * lift : r.gamr;
    }
    if (DELTA) {
      store_tile<T, VB>(hout, p.V, Sb, LDV, K, tid, NT);
      const RowScalars rs0 = row_scalars(Gs, runs, m.flags, r0 + g);
      const RowScalars rs1 = row_scalars(Gs, runs, m.flags, r0 + g + 8);
      float x[NTV][4];
      zero_acc(x);
      warp_gemm<T, NTV, K / 16, A_ROW, B_KN>(x, stage_k(s) + r0 * LDK, LDK, Sb, LDV, lane);  // K S
      if (!BWD) {
#pragma unroll
        for (int nt = 0; nt < NTV; ++nt) {
          const T* v = stage_x(s) + (r0 + g) * LDV + nt * 8 + 2 * t;
          const float2 a = unpack2<T>(*reinterpret_cast<const uint32_t*>(v));
          const float2 b = unpack2<T>(*reinterpret_cast<const uint32_t*>(v + 8 * LDV));
          x[nt][0] = a.x - rs0.gam * x[nt][0], x[nt][1] = a.y - rs0.gam * x[nt][1];
          x[nt][2] = b.x - rs1.gam * x[nt][2], x[nt][3] = b.y - rs1.gam * x[nt][3];
        }
        store_acc<T, NTV>(A1, LDV, r0, 0, x, lane);  // W
        __syncthreads();
        zero_acc(x);
        warp_gemm<T, NTV, 4, A_ROW, B_KN>(x, stage_ag(s) + r0 * LDC, LDC, A1, LDV, lane);  // Vn = Ag W
        store_acc<T, NTV>(A2, LDV, r0, 0, x, lane);
        store_acc<T, NTV>(A3, LDV, r0, 0, x, lane, rs0.gamr, rs1.gamr);
        __syncthreads();
        store_tile<T, VB>(static_cast<T*>(p.vn) + ((long)c * p.H + h) * 64 * p.V + v0, p.V, A2, LDV, 64, tid, NT);
      } else {
#pragma unroll
        for (int nt = 0; nt < NTV; ++nt) {
          x[nt][0] = x[nt][0] * rs0.gamr + z[nt][0], x[nt][1] = x[nt][1] * rs0.gamr + z[nt][1];
          x[nt][2] = x[nt][2] * rs1.gamr + z[nt][2], x[nt][3] = x[nt][3] * rs1.gamr + z[nt][3];
        }
        store_acc<T, NTV>(A2, LDV, r0, 0, x, lane);  // dVn
        if (it + 1 < n) load_z(chunk_at(it + 1));
        __syncthreads();
        store_tile<T, VB>(static_cast<T*>(p.vn) + ((long)c * p.H + h) * 64 * p.V + v0, p.V, A2, LDV, 64, tid, NT);
        zero_acc(x);
        warp_gemm<T, NTV, 4, A_COL, B_KN>(x, stage_ag(s) + r0, LDC, A2, LDV, lane);  // dW = dV = Ag^T dVn
        store_acc<T, NTV>(A1, LDV, r0, 0, x, lane, -rs0.gam, -rs1.gam);
        store_acc_wide<T, NTV>(static_cast<T*>(p.dv) + ((long)(m.tok0 + r0) * p.H + h) * p.V + v0, (long)p.H * p.V, x, lane,
                               m.len - r0);
      }
    } else {
      __syncthreads();
      // straight from the accumulators: a 16-bit copy in shared memory would leave room for one CTA less on an SM
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        store_acc_wide<T, NTV>(hout + (long)(sr0 + 16 * mt) * p.V, p.V, acc[mt], lane, 16);
      }
    }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
      for (int nt = 0; nt < NTV; ++nt) {
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[mt][nt][e] *= kg * lift;
      }
      const int a0 = sr0 + 16 * mt;
      if (!DELTA) {
        warp_gemm_scaled_a<T, NTV, 4, B_KN>(acc[mt], (BWD ? stage_q(s) : stage_k(s)) + a0, LDK, Gs + 64, stage_x(s), LDV, lane);
      } else if (!BWD) {
        warp_gemm<T, NTV, 4, A_COL, B_KN>(acc[mt], stage_k(s) + a0, LDK, A3, LDV, lane);
      } else {
        // Q^T (scale cin Gamma dO): needs nothing of the chain, ahead of the barrier the last product waits for
        warp_gemm_scaled_a<T, NTV, 4, B_KN>(acc[mt], stage_q(s) + a0, LDK, Gs + 64, stage_x(s), LDV, lane);
      }
#pragma unroll
      for (int nt = 0; nt < (kLift ? NTV : 0); ++nt) {
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[mt][nt][e] *= unlift;
      }
    }
    if (DELTA && BWD) {
      __syncthreads();  // A1 = -(cin Gamma) dW complete
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        warp_gemm<T, NTV, 4, A_COL, B_KN>(acc[mt], stage_k(s) + sr0 + 16 * mt, LDK, A1, LDV, lane);
      }
    }
#pragma unroll
    for (int mt = 0; mt < MT && DELTA; ++mt) store_acc<T, NTV>(Sb, LDV, sr0 + 16 * mt, 0, acc[mt], lane);
  }

  if (p.last) {
    float* f = p.last + ((long)row * p.H + h) * K * p.V + v0;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
      for (int nt = 0; nt < NTV; ++nt) {
        float* at = f + (long)(sr0 + 16 * mt + g) * p.V + nt * 8 + 2 * t;
        *reinterpret_cast<float2*>(at) = make_float2(acc[mt][nt][0], acc[mt][nt][1]);
        *reinterpret_cast<float2*>(at + 8 * p.V) = make_float2(acc[mt][nt][2], acc[mt][nt][3]);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------
// everything that is not serial: per chunk and head (row r, column c of the score tile are tokens of the chunk)
//   kOut: y = o = scale [(cin Gamma_r)(q_r h) + sum_{c <= r} (q_r . k_c) D_rc x_c],   x = Vn (v without the delta rule)
//   kZ  : y = Z = sum_{c >= r} scale (k_r . q_c) D_cr x_c in fp32,                    x = dO
enum { kOut = 0, kZ = 1 };

struct TokenParams {
  const ChunkMeta* meta;
  const float* gates;
  const unsigned char* runs;
  const void *a, *b;  // rows and columns of the scores: q, k (kOut) or k, q (kZ), [tokens, Hk, K]
  const void* x;      // [tokens, H, V], or [chunk slot, H, 64, V] where x_slots
  const void* h;      // [chunk slot, H, K, V]
  void* y;            // [tokens, H, V] in the tensors' dtype; kZ: [chunk slot, H, 64, V] f32
  int H, Hk, x_slots;
  float scale;
};

template <typename T, int K, int V, int MODE, int NH>
struct TokenSmem {
  static constexpr int LDK = K + 8, LDV = V + 8;
  static constexpr int kStageElems = 64 * LDV + (MODE == kZ ? 0 : K * LDV);
  static constexpr int kOutElems = MODE == kZ ? 0 : 64 * LDV;
  static constexpr int kBytes = (2 * 64 * LDK + kStageElems + kOutElems) * 2 + 2 * 256 + 64;
  static_assert(NH == 1 || kStageElems <= 2 * 64 * LDK, "the second stage lies over the key tiles");
};

// Four warps, 16 rows each. NH > 1: the CTA walks NH adjacent value heads of one key head, for which the raw scores are the
// same products: they stay in registers (as do a warp's rows of the state product's left operand), and the next head's
// tiles are on their way while one is worked on.
template <typename T, int K, int V, int MODE, int NH>
__global__ void __launch_bounds__(NT, NH > 1 ? 3 : 1) token_kernel(TokenParams p) {
  using L = TokenSmem<T, K, V, MODE, NH>;
  constexpr int LDK = L::LDK, LDV = L::LDV, NTV = V / 8;
  const int hgs = p.H / NH;
  const int c = blockIdx.x / hgs, hg = blockIdx.x - c * hgs;
  const ChunkMeta m = p.meta[c];
  if (m.len == 0) return;
  const int hk = (hg * NH) / (p.H / p.Hk);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  // the triangle gives the warps 1 to 4 k-steps of the second product: rotated over the CTAs, so that every scheduler
  // gets each share
  const int rb = (warp + blockIdx.x) & 3, r0 = 16 * rb;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* aS = reinterpret_cast<T*>(smem_raw);
  T* bS = aS + 64 * LDK;
  // NH > 1: once the scores and this warp's rows of the state product's left operand are in registers the two key tiles
  // are dead, and the second stage takes their place (three CTAs fit an SM)
  auto stage_x = [&](int s) { return s ? aS : bS + 64 * LDK; };
  auto stage_h = [&](int s) { return stage_x(s) + 64 * LDV; };
  T* yS = stage_x(0) + L::kStageElems;
  auto stage_g = [&](int s) { return reinterpret_cast<float*>(yS + L::kOutElems) + s * 64; };
  unsigned char* runs = reinterpret_cast<unsigned char*>(stage_g(2));

  auto issue_head = [&](int hi, int s) {
    const int h = hg * NH + hi;
    const long slot = (long)c * p.H + h;
    if (p.x_slots) {
      load_tile_async<T, 64, V>(stage_x(s), LDV, static_cast<const T*>(p.x) + slot * 64 * V, V, 64, tid, NT);
    } else {
      load_tile_async<T, 64, V>(stage_x(s), LDV, static_cast<const T*>(p.x) + ((long)m.tok0 * p.H + h) * V, (long)p.H * V,
                                m.len, tid, NT);
    }
    if (MODE != kZ) load_tile_async<T, K, V>(stage_h(s), LDV, static_cast<const T*>(p.h) + slot * K * V, V, K, tid, NT);
    if (tid < 16) cp_async16(stage_g(s) + tid * 4, p.gates + slot * 128 + tid * 4);
    cp_async_commit();
  };
  {
    const long key = ((long)m.tok0 * p.Hk + hk) * K;
    load_tile_async<T, 64, K>(aS, LDK, static_cast<const T*>(p.a) + key, (long)p.Hk * K, m.len, tid, NT);
    load_tile_async<T, 64, K>(bS, LDK, static_cast<const T*>(p.b) + key, (long)p.Hk * K, m.len, tid, NT);
    if (tid < 4) cp_async16(runs + tid * 16, p.runs + (long)c * 64 + tid * 16);
    cp_async_commit();
  }
  issue_head(0, 0);

  float scores[8][4];
  uint32_t rows_a[K / 16][4];  // this warp's 16 rows of a, as A fragments
  cp_async_wait<0>();
  __syncthreads();
#pragma unroll
  for (int ks = 0; ks < K / 16; ++ks) load_a<T, A_ROW>(rows_a[ks], aS + r0 * LDK, LDK, ks * 16, lane);
  zero_acc(scores);
  warp_gemm_ra<T, 8, K / 16, B_NK>(scores, rows_a, bS, LDK, lane);
  if (NH > 1) __syncthreads();  // the key tiles are free
#pragma unroll 1
  for (int hi = 0; hi < NH; ++hi) {
    const int h = hg * NH + hi, s = hi & 1;
    if (NH > 1 && hi + 1 < NH) {
      issue_head(hi + 1, s ^ 1);
      if (hi > 0) cp_async_wait<1>();
    } else if (NH > 1) {
      cp_async_wait<0>();
    }
    if (NH > 1) __syncthreads();
    const float* Gs = stage_g(s);
    const RowScalars rs0 = row_scalars(Gs, runs, m.flags, r0 + g);
    const RowScalars rs1 = row_scalars(Gs, runs, m.flags, r0 + g + 8);
    float acc[NTV][4];
    zero_acc(acc);
    if (MODE != kZ) {
      warp_gemm_ra<T, NTV, K / 16, B_KN>(acc, rows_a, stage_h(s), LDV, lane);
#pragma unroll
      for (int nt = 0; nt < NTV; ++nt) {
        acc[nt][0] *= rs0.gam, acc[nt][1] *= rs0.gam, acc[nt][2] *= rs1.gam, acc[nt][3] *= rs1.gam;
      }
    }
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {  // 16 columns of the score tile at a time, from the diagonal on
      if (MODE == kOut ? ks > rb : ks < rb) continue;
      float d[2][4];
#pragma unroll
      for (int n2 = 0; n2 < 2; ++n2) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int r = r0 + g + ((e >> 1) << 3), j = ks * 16 + n2 * 8 + 2 * t + (e & 1);
          const RowScalars& rs = (e >> 1) ? rs1 : rs0;
          const bool seen = (MODE == kOut ? j <= r : j >= r) && runs[j] == rs.run;
          const float x = MODE == kOut ? rs.G - Gs[j] : Gs[j] - rs.G;
          const float w = seen ? __expf(x) : 0.f;
          d[n2][e] = scores[2 * ks + n2][e] * (MODE == kOut ? w : p.scale * w);
        }
      }
      uint32_t frag[1][4];
      acc_to_afrag<T, 1>(frag, d);
      warp_gemm_ra<T, NTV, 1, B_KN>(acc, frag, stage_x(s) + ks * 16 * LDV, LDV, lane);
    }
    if (MODE == kZ) {
      float* z = static_cast<float*>(p.y) + ((long)c * p.H + h) * 64 * V + (long)(r0 + g) * V + 2 * t;
#pragma unroll
      for (int nt = 0; nt < NTV; ++nt) {
        *reinterpret_cast<float2*>(z + nt * 8) = make_float2(acc[nt][0], acc[nt][1]);
        *reinterpret_cast<float2*>(z + 8 * V + nt * 8) = make_float2(acc[nt][2], acc[nt][3]);
      }
    } else {  // through this warp's rows of the staging tile, in 16-byte stores
      store_acc<T, NTV>(yS, LDV, r0, 0, acc, lane, p.scale, p.scale);
      __syncwarp();
      const int rows = min(16, m.len - r0);
      if (rows > 0) {
        store_tile<T, V>(static_cast<T*>(p.y) + ((long)(m.tok0 + r0) * p.H + h) * V, (long)p.H * V, yS + r0 * LDV, LDV,
                         rows, lane, 32);
      }
    }
    if (NH > 1) __syncthreads();  // the stage may be refilled (and this warp's staging rows rewritten)
  }
}

// ---------------------------------------------------------------------------------------------------------
template <typename T, int K, int VB, bool DELTA, bool BWD>
int run_state(const StateParams& sp, int chains, cudaStream_t s) {
  auto* kern = state_kernel<T, K, VB, DELTA, BWD>;
  constexpr int smem = StateSmem<T, K, VB, DELTA, BWD>::kBytes;
  JLA_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  ProfScope ps(BWD ? kProfSplitBwd : kProfSplitFwd, s);
  kern<<<chains * (sp.V / VB), NT, smem, s>>>(sp);
  JLA_LAUNCH_OK();
  return JLA_OK;
}

// Value columns per CTA: blocks of 32 shorten a chunk's products and double the CTAs, at the price of reading q, k and Ag
// once per block; taken while blocks of 64 leave most SMs with less than three CTAs to hide each other's barriers.
template <typename T, int K, bool DELTA, bool BWD>
int run_state(const StateParams& sp, int chains, cudaStream_t s) {
  return (long)chains * (sp.V / 64) <= 2 * 148 ? run_state<T, K, 32, DELTA, BWD>(sp, chains, s)
                                              : run_state<T, K, 64, DELTA, BWD>(sp, chains, s);
}

template <typename T, int K, int V, int MODE, int NH>
int run_tokens_nh(const TokenParams& tp, int nc, cudaStream_t s) {
  auto* kern = token_kernel<T, K, V, MODE, NH>;
  constexpr int smem = TokenSmem<T, K, V, MODE, NH>::kBytes;
  JLA_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  ProfScope ps(MODE == kZ ? kProfSplitZ : kProfSplitOut, s);
  kern<<<nc * (tp.H / NH), NT, smem, s>>>(tp);
  JLA_LAUNCH_OK();
  return JLA_OK;
}

template <typename T, int K, int V, int MODE>
int run_tokens(const TokenParams& tp, int nc, cudaStream_t s) {
  // walks of 8 heads where key groups allow it and enough CTAs are left to fill the SMs
  if constexpr (V == 64) {
    if (tp.H / tp.Hk % 8 == 0 && (long)nc * tp.H / 8 >= 2 * 148) return run_tokens_nh<T, K, V, MODE, 8>(tp, nc, s);
  }
  return run_tokens_nh<T, K, V, MODE, 1>(tp, nc, s);
}

template <typename T, int K, int V>
int run_tokens(const TokenParams& tp, int mode, int nc, cudaStream_t s) {
  if (mode == kOut) return run_tokens<T, K, V, kOut>(tp, nc, s);
  return run_tokens<T, K, V, kZ>(tp, nc, s);
}

template <typename T>
int run_tokens(const TokenParams& tp, const jla_problem& p, int mode, int nc, cudaStream_t s) {
  if (p.K == 128) return p.V == 128 ? run_tokens<T, 128, 128>(tp, mode, nc, s) : run_tokens<T, 128, 64>(tp, mode, nc, s);
  return p.V == 128 ? run_tokens<T, 64, 128>(tp, mode, nc, s) : run_tokens<T, 64, 64>(tp, mode, nc, s);
}

template <typename T, bool BWD>
int run_states(const StateParams& sp, const jla_problem& p, bool delta, int chains, cudaStream_t s) {
  if (p.K == 128) {
    return delta ? run_state<T, 128, true, BWD>(sp, chains, s) : run_state<T, 128, false, BWD>(sp, chains, s);
  }
  return delta ? run_state<T, 64, true, BWD>(sp, chains, s) : run_state<T, 64, false, BWD>(sp, chains, s);
}

StateParams state_params(const ChunkedCtx& c) {
  const Plan& pl = c.plan;
  StateParams sp{};
  sp.meta = reinterpret_cast<const ChunkMeta*>(c.res + pl.meta);
  sp.row_chunks = reinterpret_cast<const int2*>(c.res + pl.row_chunks);
  sp.gates = reinterpret_cast<const float*>(c.res + pl.gates);
  sp.runs = reinterpret_cast<const unsigned char*>(c.res + pl.runs);
  sp.q = c.q_eff, sp.k = c.k_eff;
  sp.ag = c.res + pl.ag;
  sp.H = c.p.H, sp.Hk = c.p.Hk, sp.V = c.p.V, sp.scale = c.p.scale;
  return sp;
}

TokenParams token_params(const ChunkedCtx& c, int mode) {
  const Plan& pl = c.plan;
  TokenParams tp{};
  tp.meta = reinterpret_cast<const ChunkMeta*>(c.res + pl.meta);
  tp.gates = reinterpret_cast<const float*>(c.res + pl.gates);
  tp.runs = reinterpret_cast<const unsigned char*>(c.res + pl.runs);
  tp.a = mode == kOut ? c.q_eff : c.k_eff, tp.b = mode == kOut ? c.k_eff : c.q_eff;
  tp.H = c.p.H, tp.Hk = c.p.Hk, tp.scale = c.p.scale;
  return tp;
}

}  // namespace

int launch_split_fwd(const ChunkedCtx& c, const jla_fwd_io& io, cudaStream_t s) {
  const jla_problem& p = c.p;
  const Plan& pl = c.plan;
  if (pl.rows == 0) return JLA_OK;
  const bool bf = p.dtype == JLA_DTYPE_BF16;
  StateParams sp = state_params(c);
  sp.x = p.v;
  sp.first = p.h0, sp.last = io.final_state;
  sp.h = c.res + pl.h, sp.vn = c.res + pl.vn;
  const int chains = pl.rows * p.H;
  const int rc = bf ? run_states<__nv_bfloat16, false>(sp, p, pl.delta, chains, s)
                    : run_states<__half, false>(sp, p, pl.delta, chains, s);
  if (rc != JLA_OK) return rc;
  TokenParams tp = token_params(c, kOut);
  tp.x = pl.delta ? static_cast<const void*>(c.res + pl.vn) : p.v;
  tp.x_slots = pl.delta;
  tp.h = c.res + pl.h;
  tp.y = io.o;
  return bf ? run_tokens<__nv_bfloat16>(tp, p, kOut, pl.nc, s) : run_tokens<__half>(tp, p, kOut, pl.nc, s);
}

int launch_split_bwd_state(const ChunkedCtx& c, const jla_bwd_io& io, char* scratch, cudaStream_t s) {
  const jla_problem& p = c.p;
  const Plan& pl = c.plan;
  if (pl.rows == 0) return JLA_OK;
  const bool bf = p.dtype == JLA_DTYPE_BF16;
  if (pl.delta) {
    TokenParams tp = token_params(c, kZ);
    tp.x = io.d_o;
    tp.y = scratch + pl.z;
    const int rc = bf ? run_tokens<__nv_bfloat16>(tp, p, kZ, pl.nc, s) : run_tokens<__half>(tp, p, kZ, pl.nc, s);
    if (rc != JLA_OK) return rc;
  }
  StateParams sp = state_params(c);
  sp.x = io.d_o;
  sp.z = reinterpret_cast<const float*>(scratch + pl.z);
  sp.first = io.d_final, sp.last = io.dh0;
  sp.h = scratch + pl.dh, sp.vn = scratch + pl.dvn, sp.dv = io.dv;
  const int chains = pl.rows * p.H;
  return bf ? run_states<__nv_bfloat16, true>(sp, p, pl.delta, chains, s)
            : run_states<__half, true>(sp, p, pl.delta, chains, s);
}

}  // namespace jla
