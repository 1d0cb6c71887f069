// Backward of the scalar-gate family, chunk-64: a reverse serial pass that emits dv, dVn and the per-chunk dS+
// (chunked_split.cu, chunked_bwd_state_tc.cu), then a chunk-parallel kernel for dq, dk, dbeta, dg.
//
//   dVn = scale P^T dO + (tail Gamma_r)(K dS+)       dW = Ag^T dVn = dV
//   dS  = keep gamma dS+ + scale ((cin Gamma) Q)^T dO - ((cin Gamma) K)^T dW
//   dP  = scale (dO Vn^T) D      dQ = scale (cin Gamma)(dO S^T) + dP K
//   dAg = tril(dVn W^T)   dT0 = dAg D beta_j   dA0 = -strict(T0^T dT0 T0^T) same
//   dK  = (tail Gamma_r)(Vn dS+^T) - (cin Gamma)(dW S^T) + dP^T Q + (dA0 beta_i) K + (dA0 beta_i)^T K
// and the gate / beta gradients as row and column sums of the same tiles (the reference's split backward:
// src/jla/ops/mosaic_gpu/gated_delta_rule_bwd.py:303-853; here column sums are shuffle reductions instead of
// second, transposed products).
#include <stdlib.h>

#include <type_traits>

#include "chunked.cuh"
#include "profile.cuh"
#include "mma.cuh"

namespace jla {
namespace {

struct BwdParams {
  const ChunkMeta* meta;
  const float* gates;
  const unsigned char* runs;
  const void *q, *k, *v, *t0, *d_o, *h, *vn;
  const void *dh, *dvn, *dv;
  void* dv_out;            // dv where the gradient kernel itself writes it (without the delta rule)
  void *dq, *dk;          // tensor dtype, written directly when dq_acc == nullptr
  float *dq_acc, *dk_acc;  // [tokens, H, K] f32 otherwise
  float *dg, *dbeta;
  const float* qk_tab;  // Q K^T per (chunk, key head) in fragment order (qk_table_kernel), for walks over heads
  int H, Hk;
  float scale;
};

// ---------------------------------------------------------------------------------------------------------
// chunk-parallel gradients

// Reductions avoid shared-memory float atomics (a compare-and-swap loop): every warp adds into slots that only it
// writes (row sums: one slot array per column half; column sums: one per row quadrant), always from the same lane,
// and the slots are summed once at the end.
// vec[row] += sign * sum over this thread's columns, reduced over the 4 lanes of a quad.
template <int NT>
__device__ __forceinline__ void row_sums_add(const float (&x)[NT][4], float* vec, int r0, int lane, float sign) {
  float a = 0.f, b = 0.f;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    a += x[nt][0] + x[nt][1];
    b += x[nt][2] + x[nt][3];
  }
  a += __shfl_xor_sync(0xffffffffu, a, 1);
  a += __shfl_xor_sync(0xffffffffu, a, 2);
  b += __shfl_xor_sync(0xffffffffu, b, 1);
  b += __shfl_xor_sync(0xffffffffu, b, 2);
  if ((lane & 3) == 0) {
    vec[r0 + (lane >> 2)] += sign * a;
    vec[r0 + (lane >> 2) + 8] += sign * b;
  }
}

// vec[c0 + col] += sign * sum over the warp's 16 rows.
template <int NT>
__device__ __forceinline__ void col_sums_add(const float (&x)[NT][4], float* vec, int c0, int lane, float sign) {
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    float a = x[nt][0] + x[nt][2], b = x[nt][1] + x[nt][3];
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, off);
      b += __shfl_xor_sync(0xffffffffu, b, off);
    }
    if (lane < 4) {
      vec[c0 + nt * 8 + 2 * lane] += sign * a;
      vec[c0 + nt * 8 + 2 * lane + 1] += sign * b;
    }
  }
}

// sum_k x[i][k] * tile[i][k] for the warp's rows (tile in smem, 16-bit), reduced over the quad.
template <typename T, int NT>
__device__ __forceinline__ void row_dots(const float (&x)[NT][4], const T* tile, int ld, int r0, int c0, int lane,
                                         float& d0, float& d1) {
  const int g = lane >> 2, t = lane & 3;
  d0 = 0.f;
  d1 = 0.f;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const float2 a = unpack2<T>(*reinterpret_cast<const uint32_t*>(tile + (r0 + g) * ld + c0 + nt * 8 + 2 * t));
    const float2 b = unpack2<T>(*reinterpret_cast<const uint32_t*>(tile + (r0 + g + 8) * ld + c0 + nt * 8 + 2 * t));
    d0 += x[nt][0] * a.x + x[nt][1] * a.y;
    d1 += x[nt][2] * b.x + x[nt][3] * b.y;
  }
  d0 += __shfl_xor_sync(0xffffffffu, d0, 1);
  d0 += __shfl_xor_sync(0xffffffffu, d0, 2);
  d1 += __shfl_xor_sync(0xffffffffu, d1, 1);
  d1 += __shfl_xor_sync(0xffffffffu, d1, 2);
}

template <typename T, int K, int V>
struct GradSmem {
  static constexpr int LDK = K + 8, LDV = V + 8, LDC = 72;
  // k | q | do (q and do contiguous: later reused for dS+) | v (W, then dW) | Vn | S | T0, Xa, Xb, Xc | vectors
  static constexpr int kElems = 2 * 64 * LDK + 2 * 64 * LDV + 64 * LDV + K * LDV + 4 * 64 * LDC;
  static constexpr int kBytes = kElems * 2 + (128 + 13 * 64 + 16) * 4 + 64;
  static_assert(K * LDV <= 64 * LDK + 64 * LDV, "dS+ must fit in the q | do region");
};

template <typename T, int K, int V>
__global__ void __launch_bounds__(256, 1) sg_chunk_grads_kernel(BwdParams p) {
  using L = GradSmem<T, K, V>;
  constexpr int LDK = L::LDK, LDV = L::LDV, LDC = L::LDC;
  constexpr int ONT = V / 16, KNT = K / 16;
  const int c = blockIdx.x / p.H, h = blockIdx.x - c * p.H;
  const ChunkMeta m = p.meta[c];
  if (m.len == 0) return;
  const int hk = h / (p.H / p.Hk);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int r0 = 16 * (warp & 3), ch = warp >> 2;
  const int c0 = (V / 2) * ch, kc0 = (K / 2) * ch, cc0 = 32 * ch;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* kS = reinterpret_cast<T*>(smem_raw);
  T* qS = kS + 64 * LDK;
  T* doS = qS + 64 * LDK;             // dO, later dVn
  T* vS = doS + 64 * LDV;             // V -> W in place, later dW
  T* vnS = vS + 64 * LDV;
  T* SS = vnS + 64 * LDV;
  T* t0S = SS + K * LDV;
  T* Xa = t0S + 64 * LDC;
  T* Xb = Xa + 64 * LDC;
  T* Xc = Xb + 64 * LDC;
  float* Gs = reinterpret_cast<float*>(smem_raw + L::kElems * 2);
  float* betas = Gs + 64;
  float* dGrow = betas + 64;   // [2][64] row-wise dG terms per column half
  float* dGcol = dGrow + 128;  // [4][64] column-wise dG terms per row quadrant
  float* dbrow = dGcol + 256;  // [2][64]
  float* dbcol = dbrow + 128;  // [4][64]
  float* dGv = dbcol + 256;    // [64] folded dG
  float* tot = dGv + 64;       // [8] per warp
  float* sdot = tot + 8;       // [8] per warp
  unsigned char* runs = reinterpret_cast<unsigned char*>(sdot + 8);
  const int quad = warp & 3;
  T* dSS = qS;  // dS+ overlays q | do once both are dead
  float accK[KNT][4];  // dk, 16 rows x K/2 columns per warp
  float accQ[KNT][4];  // dq likewise
  zero_acc(accK);
  zero_acc(accQ);

  float tot_part = 0.f;
  const long ch_off = (long)c * p.H + h;
  // group 0: k, S, v, T0, gates, runs
  load_tile_async<T, 64, K>(kS, LDK, static_cast<const T*>(p.k) + ((long)m.tok0 * p.Hk + hk) * K, (long)p.Hk * K, m.len,
                            tid, 256);
  load_tile_async<T, K, V>(SS, LDV, static_cast<const T*>(p.h) + ch_off * K * V, V, K, tid, 256);
  load_tile_async<T, 64, V>(vS, LDV, static_cast<const T*>(p.v) + ((long)m.tok0 * p.H + h) * V, (long)p.H * V, m.len,
                            tid, 256);
  load_tile_async<T, 64, 64>(t0S, LDC, static_cast<const T*>(p.t0) + ch_off * 4096, 64, 64, tid, 256);
  if (tid < 32) cp_async16(Gs + tid * 4, p.gates + ch_off * 128 + tid * 4);
  if (tid >= 32 && tid < 36) cp_async16(runs + (tid - 32) * 16, p.runs + (long)c * 64 + (tid - 32) * 16);
  cp_async_commit();
  // group 1: dO, Vn, q
  load_tile_async<T, 64, V>(doS, LDV, static_cast<const T*>(p.d_o) + ((long)m.tok0 * p.H + h) * V, (long)p.H * V,
                            m.len, tid, 256);
  load_tile_async<T, 64, V>(vnS, LDV, static_cast<const T*>(p.vn) + ch_off * 64 * V, V, 64, tid, 256);
  load_tile_async<T, 64, K>(qS, LDK, static_cast<const T*>(p.q) + ((long)m.tok0 * p.Hk + hk) * K, (long)p.Hk * K, m.len,
                            tid, 256);
  cp_async_commit();
  for (int idx = tid; idx < 12 * 64; idx += 256) dGrow[idx] = 0.f;
  cp_async_wait<1>();
  __syncthreads();

  const RowScalars rs0 = row_scalars(Gs, runs, m.flags, r0 + g);
  const RowScalars rs1 = row_scalars(Gs, runs, m.flags, r0 + g + 8);

  {  // 1. W = V - (cin Gamma)(K S), in place over V
    float acc[ONT][4];
    zero_acc(acc);
    warp_gemm<T, ONT, K / 16, A_ROW, B_KN>(acc, kS + r0 * LDK, LDK, SS + c0, LDV, lane);
#pragma unroll
    for (int nt = 0; nt < ONT; ++nt) {
      const int col = c0 + nt * 8 + 2 * t;
      uint32_t* w0 = reinterpret_cast<uint32_t*>(vS + (r0 + g) * LDV + col);
      uint32_t* w1 = reinterpret_cast<uint32_t*>(vS + (r0 + g + 8) * LDV + col);
      const float2 v0 = unpack2<T>(*w0), v1 = unpack2<T>(*w1);
      *w0 = pack2<T>(v0.x - rs0.gam * acc[nt][0], v0.y - rs0.gam * acc[nt][1]);
      *w1 = pack2<T>(v1.x - rs1.gam * acc[nt][2], v1.y - rs1.gam * acc[nt][3]);
    }
  }
  cp_async_wait<0>();
  __syncthreads();  // S1

  {  // 2. dP = scale (dO Vn^T) D ; E = dP (Q K^T)
    float accP[4][4], accE[4][4];
    zero_acc(accP);
    zero_acc(accE);
    warp_gemm<T, 4, V / 16, A_ROW, B_NK>(accP, doS + r0 * LDV, LDV, vnS + cc0 * LDV, LDV, lane);
    warp_gemm<T, 4, K / 16, A_ROW, B_NK>(accE, qS + r0 * LDK, LDK, kS + cc0 * LDK, LDK, lane);
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const int j = cc0 + nt * 8 + 2 * t;
      accP[nt][0] *= p.scale * decay_ij(Gs, runs, r0 + g, j, rs0.G, rs0.run);
      accP[nt][1] *= p.scale * decay_ij(Gs, runs, r0 + g, j + 1, rs0.G, rs0.run);
      accP[nt][2] *= p.scale * decay_ij(Gs, runs, r0 + g + 8, j, rs1.G, rs1.run);
      accP[nt][3] *= p.scale * decay_ij(Gs, runs, r0 + g + 8, j + 1, rs1.G, rs1.run);
#pragma unroll
      for (int e = 0; e < 4; ++e) accE[nt][e] *= accP[nt][e];
    }
    row_sums_add<4>(accE, dGrow + ch * 64, r0, lane, 1.f);
    col_sums_add<4>(accE, dGcol + quad * 64, cc0, lane, -1.f);
    store_acc<T, 4>(Xa, LDC, r0, cc0, accP, lane);
  }
  {  // 3. dq = scale (cin Gamma)(dO S^T) + dP K
    const float s0 = p.scale * rs0.gam, s1 = p.scale * rs1.gam;
    float d0, d1;
    warp_gemm<T, KNT, V / 16, A_ROW, B_NK>(accQ, doS + r0 * LDV, LDV, SS + kc0 * LDV, LDV, lane);
#pragma unroll
    for (int nt = 0; nt < KNT; ++nt) {
      accQ[nt][0] *= s0;
      accQ[nt][1] *= s0;
      accQ[nt][2] *= s1;
      accQ[nt][3] *= s1;
    }
    row_dots<T, KNT>(accQ, qS, LDK, r0, kc0, lane, d0, d1);
    if (t == 0) {
      dGrow[ch * 64 + r0 + g] += d0;
      dGrow[ch * 64 + r0 + g + 8] += d1;
    }
  }
  __syncthreads();  // S2: Xa = dP complete
  warp_gemm<T, KNT, 4, A_ROW, B_KN>(accQ, Xa + r0 * LDC, LDC, kS + kc0, LDK, lane);
  {
    const long tok0 = (long)m.tok0 + r0 + g;
#pragma unroll
    for (int nt = 0; nt < KNT; ++nt) {
      const int col = kc0 + nt * 8 + 2 * t;
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        if (r0 + g + 8 * hh >= m.len) continue;
        const long tok = tok0 + 8 * hh;
        if (p.dq_acc) {
          *reinterpret_cast<float2*>(p.dq_acc + (tok * p.H + h) * K + col) = make_float2(accQ[nt][2 * hh], accQ[nt][2 * hh + 1]);
        } else {
          *reinterpret_cast<uint32_t*>(static_cast<T*>(p.dq) + (tok * p.Hk + hk) * K + col) =
              pack2<T>(accQ[nt][2 * hh], accQ[nt][2 * hh + 1]);
        }
      }
    }
  }
  // 4. dk += dP^T Q
  warp_gemm<T, KNT, 4, A_COL, B_KN>(accK, Xa + r0, LDC, qS + kc0, LDK, lane);
  __syncthreads();  // S3: q, dO dead

  {
    load_tile_async<T, 64, V>(doS, LDV, static_cast<const T*>(p.dvn) + ch_off * 64 * V, V, 64, tid, 256);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();  // S4: dVn landed (in the dO buffer)
    {  // 5. dAg = tril(dVn W^T); F = dAg Ag; dT0 = dAg D beta_j
      float accA[4][4], accF[4][4], accB[4][4];
      zero_acc(accA);
      warp_gemm<T, 4, V / 16, A_ROW, B_NK>(accA, doS + r0 * LDV, LDV, vS + cc0 * LDV, LDV, lane);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = r0 + g + ((e >> 1) << 3), j = cc0 + nt * 8 + 2 * t + (e & 1);
          const RowScalars& rs = (e >> 1) ? rs1 : rs0;
          const float d = decay_ij(Gs, runs, i, j, rs.G, rs.run);
          const float t0v = to_f32(t0S[i * LDC + j]);
          const float dag = accA[nt][e];
          accB[nt][e] = dag * t0v * d;          // -> dbeta_j (column sums)
          accF[nt][e] = accB[nt][e] * betas[j]; // dAg * Ag
          accA[nt][e] = dag * d * betas[j];     // dT0
        }
      }
      row_sums_add<4>(accF, dGrow + ch * 64, r0, lane, 1.f);
      col_sums_add<4>(accF, dGcol + quad * 64, cc0, lane, -1.f);
      col_sums_add<4>(accB, dbcol + quad * 64, cc0, lane, 1.f);
      store_acc<T, 4>(Xb, LDC, r0, cc0, accA, lane);
    }
    __syncthreads();  // S5: Xb = dT0 complete; W and dVn dead
    // prefetch dW (into the W buffer) and dS+ (over q | do)
    load_tile_async<T, 64, V>(vS, LDV, static_cast<const T*>(p.dv) + ((long)m.tok0 * p.H + h) * V, (long)p.H * V, m.len,
                              tid, 256);
    load_tile_async<T, K, V>(dSS, LDV, static_cast<const T*>(p.dh) + ch_off * K * V, V, K, tid, 256);
    cp_async_commit();
    {  // M1 = dT0 T0^T
      float accM[4][4];
      zero_acc(accM);
      warp_gemm<T, 4, 4, A_ROW, B_NK>(accM, Xb + r0 * LDC, LDC, t0S + cc0 * LDC, LDC, lane);
      store_acc<T, 4>(Xc, LDC, r0, cc0, accM, lane);
    }
    __syncthreads();  // S6: Xc = M1 complete, Xb free
    {  // dA0 = -strict(T0^T M1) same ; dbeta_i += sum_j dA0_ij (k_i . k_j)
      float accA0[4][4], accKK[4][4];
      zero_acc(accA0);
      zero_acc(accKK);
      warp_gemm<T, 4, 4, A_COL, B_KN>(accA0, t0S + r0, LDC, Xc + cc0, LDC, lane);
      warp_gemm<T, 4, K / 16, A_ROW, B_NK>(accKK, kS + r0 * LDK, LDK, kS + cc0 * LDK, LDK, lane);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = r0 + g + ((e >> 1) << 3), j = cc0 + nt * 8 + 2 * t + (e & 1);
          const float a = (j < i && runs[j] == runs[i]) ? -accA0[nt][e] : 0.f;
          accKK[nt][e] *= a;
          accA0[nt][e] = a * betas[i];
        }
      }
      row_sums_add<4>(accKK, dbrow + ch * 64, r0, lane, 1.f);
      store_acc<T, 4>(Xb, LDC, r0, cc0, accA0, lane);
    }
    __syncthreads();  // S7: Xb = dA0 beta_i complete
    warp_gemm<T, KNT, 4, A_ROW, B_KN>(accK, Xb + r0 * LDC, LDC, kS + kc0, LDK, lane);
    warp_gemm<T, KNT, 4, A_COL, B_KN>(accK, Xb + r0, LDC, kS + kc0, LDK, lane);
  }
  cp_async_wait<0>();
  __syncthreads();  // S8: dW, dS+ landed

  {  // 6. state terms of dk and dG
    float accT[KNT][4];
    float d0, d1;
    {  // - (cin Gamma)(dW S^T)
      zero_acc(accT);
      warp_gemm<T, KNT, V / 16, A_ROW, B_NK>(accT, vS + r0 * LDV, LDV, SS + kc0 * LDV, LDV, lane);
#pragma unroll
      for (int nt = 0; nt < KNT; ++nt) {
        accT[nt][0] *= rs0.gam;
        accT[nt][1] *= rs0.gam;
        accT[nt][2] *= rs1.gam;
        accT[nt][3] *= rs1.gam;
#pragma unroll
        for (int e = 0; e < 4; ++e) accK[nt][e] -= accT[nt][e];
      }
      row_dots<T, KNT>(accT, kS, LDK, r0, kc0, lane, d0, d1);
      if (t == 0) {
        dGrow[ch * 64 + r0 + g] -= d0;
        dGrow[ch * 64 + r0 + g + 8] -= d1;
      }
    }
    zero_acc(accT);  // (tail Gamma_r)(Vn dS+^T)
    warp_gemm<T, KNT, V / 16, A_ROW, B_NK>(accT, vnS + r0 * LDV, LDV, dSS + kc0 * LDV, LDV, lane);
#pragma unroll
    for (int nt = 0; nt < KNT; ++nt) {
      accT[nt][0] *= rs0.gamr;
      accT[nt][1] *= rs0.gamr;
      accT[nt][2] *= rs1.gamr;
      accT[nt][3] *= rs1.gamr;
#pragma unroll
      for (int e = 0; e < 4; ++e) accK[nt][e] += accT[nt][e];
    }
    row_dots<T, KNT>(accT, kS, LDK, r0, kc0, lane, d0, d1);
    if (t == 0) {
      dGrow[ch * 64 + r0 + g] -= d0;
      dGrow[ch * 64 + r0 + g + 8] -= d1;
      tot_part += d0 + d1;
    }
    // keep gamma <S, dS+>
    float part = 0.f;
    for (int idx = tid; idx < K * (V / 2); idx += 256) {
      const int r = idx / (V / 2), cidx = (idx - r * (V / 2)) * 2;
      const float2 a = unpack2<T>(*reinterpret_cast<const uint32_t*>(SS + r * LDV + cidx));
      const float2 b = unpack2<T>(*reinterpret_cast<const uint32_t*>(dSS + r * LDV + cidx));
      part += a.x * b.x + a.y * b.y;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
    if (lane == 0) sdot[warp] = part;
    // dk out
    const long tok0 = (long)m.tok0 + r0 + g;
#pragma unroll
    for (int nt = 0; nt < KNT; ++nt) {
      const int col = kc0 + nt * 8 + 2 * t;
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        if (r0 + g + 8 * hh >= m.len) continue;
        const long tok = tok0 + 8 * hh;
        if (p.dk_acc) {
          *reinterpret_cast<float2*>(p.dk_acc + (tok * p.H + h) * K + col) = make_float2(accK[nt][2 * hh], accK[nt][2 * hh + 1]);
        } else {
          *reinterpret_cast<uint32_t*>(static_cast<T*>(p.dk) + (tok * p.Hk + hk) * K + col) =
              pack2<T>(accK[nt][2 * hh], accK[nt][2 * hh + 1]);
        }
      }
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) tot_part += __shfl_xor_sync(0xffffffffu, tot_part, off);
  if (lane == 0) tot[warp] = tot_part;
  __syncthreads();  // S9
  if (tid < 64) {
    float dG = dGrow[tid] + dGrow[64 + tid] + dGcol[tid] + dGcol[64 + tid] + dGcol[128 + tid] + dGcol[192 + tid];
    if (tid == 63) {
#pragma unroll
      for (int w = 0; w < 8; ++w) dG += tot[w];
    }
    dGv[tid] = dG;
  }
  __syncthreads();
  if (tid < 64) {  // 7. dg = reverse cumulative sum of dG over the chunk
    float acc = 0.f;
    for (int j = 63; j >= tid; --j) acc += dGv[j];
    // the keep gamma <S, dS+> term belongs to the chunk's last position, so it is part of every suffix sum
    float sd = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) sd += sdot[w];
    acc += keep_gamma(Gs, runs, m.flags) * sd;
    if (tid < m.len) {
      if (p.dg) p.dg[((long)m.tok0 + tid) * p.H + h] = acc;
      p.dbeta[((long)m.tok0 + tid) * p.H + h] =
          dbrow[tid] + dbrow[64 + tid] + dbcol[tid] + dbcol[64 + tid] + dbcol[128 + tid] + dbcol[192 + tid];
    }
  }
}

// ---------------------------------------------------------------------------------------------------------
// chunk-parallel gradients without the delta rule (Vn = V), dv among them:
//   dP = scale (dO V^T) D      dQ = scale (cin Gamma)(dO S^T) + dP K      dK = (tail Gamma_r)(V dS+^T) + dP^T Q
//   dV = (tail Gamma_r)(K dS+) + P^T dO,  P = scale (Q K^T) D
// One CTA walks NH adjacent value heads of one key head for the same chunk (the reference sums the group inside its
// kernel as well, src/jla/ops/mosaic_gpu/scalar_gate_grouped.py:65-237): the sums of dq and dk over the heads stay in the
// accumulators, Q K^T comes from a table, and since K and Q are the same for every head only the sum of the dP tiles is
// multiplied with them, once.
//
// Sixteen warps in two groups of eight: the query group forms P, dP and the dq terms, the key group the dk terms, <S, dS+>
// and dV (for which it takes P from the query group). Bound by the latency of its dependent instructions at four warps a
// scheduler (0.3 issued a cycle, tensor pipe 15 %). Measured at B8 T2048 H64 P64 N128: 588 us; with the score table read
// from L2 for every head and the document test in every element 674 us; with <S, dS+> in the query group as well 768 us; as
// one group of eight warps, two CTAs an SM, both accumulators in every warp (spilling) 709 us; the form with a product with
// K and one with Q per head, and dV in a kernel of its own, 613 + 149 us. The tiles of the next head are on their way for
// the whole time of one head: one block-wide barrier a head, and a hand-over of P between the groups.
template <typename T, int K, int V>
struct DecayGradSmem {
  static constexpr int LDK = K + 8, LDV = V + 8, LDC = 72;
  static constexpr int kStageElems = 2 * K * LDV + 2 * 64 * LDV;
  static constexpr int kStageBytes = kStageElems * 2 + 256;  // + G[64]
  // per-head dG terms: rows [2][64] query group, [2][64] key group, columns [4][64], sums [16], two heads' worth
  static constexpr int kVecFloats = 128 + 128 + 256 + 16;
  static constexpr int kTabBytes = 64 * 64 * 4;  // the raw scores, in fragment order (walks over heads)
  static constexpr int kBytes = (2 * 64 * LDK + 2 * 64 * LDC) * 2 + 2 * kStageBytes + 2 * kVecFloats * 4 + 64 + kTabBytes;
  // (K = V = 128, which only an A/B switch sends here, has room for one head's tiles at a time)
  static constexpr bool kTwoStages = kBytes <= 227 * 1024;
  static constexpr int kAllocBytes = kTwoStages ? kBytes : kBytes - kStageBytes;
};

template <typename T, int K, int V, int NH>
__global__ void __launch_bounds__(512, 1) decay_grads_kernel(BwdParams p) {
  using L = DecayGradSmem<T, K, V>;
  constexpr int LDK = L::LDK, LDV = L::LDV, LDC = L::LDC, NT = 512;
  constexpr int ONT = V / 16, KNT = K / 16, HN = KNT / 2;
  static_assert(NH == 1 || L::kTwoStages, "a walk over heads has the next head's tiles in flight");
  const int hgs = p.H / NH;  // head groups of NH per chunk
  const int c = blockIdx.x / hgs, hg = blockIdx.x - c * hgs;
  const ChunkMeta m = p.meta[c];
  if (m.len == 0) return;
  const int hk = (hg * NH) / (p.H / p.Hk);  // NH divides the group size: every head of the walk shares the key head
  const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const bool keys = tid >= 256;  // the key group
  const int warp = (tid >> 5) & 7, quad = warp & 3, r0 = 16 * quad, ch = warp >> 2;
  const int c0 = (V / 2) * ch, kc0 = (K / 2) * ch, cc0 = 32 * ch;
  const bool lower = cc0 <= r0 + 15;  // this warp's 16 x 32 tile of the scores reaches the diagonal

  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* qS = reinterpret_cast<T*>(smem_raw);
  T* kS = qS + 64 * LDK;
  T* P0 = kS + 64 * LDK;  // P of this head and of the next; at the end P0 holds the sum of the dP tiles
  unsigned char* vec_base = reinterpret_cast<unsigned char*>(P0 + 2 * 64 * LDC);
  auto vecs = [&](int s) { return reinterpret_cast<float*>(vec_base) + s * L::kVecFloats; };
  unsigned char* runs = vec_base + 2 * L::kVecFloats * 4;
  float* tab = reinterpret_cast<float*>(runs + 64);
  unsigned char* stage_base = runs + 64 + L::kTabBytes;
  auto stage_s = [&](int s) { return reinterpret_cast<T*>(stage_base + s * L::kStageBytes); };
  auto stage_ds = [&](int s) { return stage_s(s) + K * LDV; };
  auto stage_v = [&](int s) { return stage_ds(s) + K * LDV; };
  auto stage_do = [&](int s) { return stage_v(s) + 64 * LDV; };
  auto stage_g = [&](int s) { return reinterpret_cast<float*>(stage_s(s) + L::kStageElems); };

  const long key = ((long)m.tok0 * p.Hk + hk) * K;
  load_tile_async<T, 64, K>(qS, LDK, static_cast<const T*>(p.q) + key, (long)p.Hk * K, m.len, tid, NT);
  load_tile_async<T, 64, K>(kS, LDK, static_cast<const T*>(p.k) + key, (long)p.Hk * K, m.len, tid, NT);
  if (tid < 4) cp_async16(runs + tid * 16, p.runs + (long)c * 64 + tid * 16);
  if (NH > 1) {
    const float* src = p.qk_tab + ((long)c * p.Hk + hk) * kQkTabFloats;
    for (int i = tid * 4; i < 64 * 64; i += NT * 4) cp_async16(tab + i, src + i);
  }
  auto load_head = [&](int hi) {
    const int h = hg * NH + hi, s = hi & 1;
    const long slot = (long)c * p.H + h, val = ((long)m.tok0 * p.H + h) * V;
    load_tile_async<T, 64, V>(stage_do(s), LDV, static_cast<const T*>(p.d_o) + val, (long)p.H * V, m.len, tid, NT);
    load_tile_async<T, 64, V>(stage_v(s), LDV, static_cast<const T*>(p.v) + val, (long)p.H * V, m.len, tid, NT);
    load_tile_async<T, K, V>(stage_s(s), LDV, static_cast<const T*>(p.h) + slot * K * V, V, K, tid, NT);
    load_tile_async<T, K, V>(stage_ds(s), LDV, static_cast<const T*>(p.dh) + slot * K * V, V, K, tid, NT);
    if (tid < 16) cp_async16(stage_g(s) + tid * 4, p.gates + slot * 128 + tid * 4);
    cp_async_commit();
  };
  // dg of a head from its dG terms (one warp): reverse cumulative sum over the chunk, two tokens a lane
  auto write_dg = [&](int hi) {
    const float* x = vecs(hi & 1);
    const int t0 = 2 * lane, t1 = t0 + 1;
    auto terms = [&](int i) {
      return (x[i] + x[64 + i]) + (x[128 + i] + x[192 + i]) + ((x[256 + i] + x[320 + i]) + (x[384 + i] + x[448 + i]));
    };
    const float a = terms(t0), b = terms(t1);
    float last = 0.f;  // the terms of S+ belong to the chunk's last position, so they are part of every suffix sum
#pragma unroll
    for (int w = 0; w < 16; ++w) last += x[512 + w];
    float incl = a + b;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const float y = __shfl_down_sync(0xffffffffu, incl, off);
      if (lane + off < 32) incl += y;
    }
    float* dg = p.dg + (long)m.tok0 * p.H + hg * NH + hi;
    if (t0 < m.len) dg[(long)t0 * p.H] = incl + last;
    if (t1 < m.len) dg[(long)t1 * p.H] = incl - a + last;
  };

  float acc[KNT][4];   // dq (query group) or dk (key group), 16 rows x K/2 columns, summed over the heads
  float sumP[4][4];    // query group: the sum of the dP tiles, 16 rows x 32 columns
  zero_acc(acc);
  zero_acc(sumP);
  load_head(0);

#pragma unroll 1
  for (int hi = 0; hi < NH; ++hi) {
    const int h = hg * NH + hi, s = hi & 1;
    T* Ps = P0 + s * 64 * LDC;
    float* out = vecs(s);
    cp_async_wait<0>();
    __syncthreads();  // the head's tiles have landed; the head before is done with its own
    if (hi + 1 < NH) load_head(hi + 1);
    if (hi > 0 && p.dg && keys && warp == 0) write_dg(hi - 1);  // (the key group has the shorter way)
    const float* Gs = stage_g(s);
    const bool one_run = runs[63] == 0;  // one document in the chunk
    const RowScalars rs0 = row_scalars(Gs, runs, m.flags, r0 + g);
    const RowScalars rs1 = row_scalars(Gs, runs, m.flags, r0 + g + 8);
    float row0 = 0.f, row1 = 0.f;  // this warp's share of dG for its rows r0 + g and r0 + g + 8
    if (!keys) {
      {  // P and dP, the sums of dP (Q K^T) over rows and columns
        float accP[4][4], tile[4][4];
        zero_acc(accP);
        zero_acc(tile);
        if (NH > 1) {
          const float4* src = reinterpret_cast<const float4*>(tab) + (quad * 8 + 4 * ch) * 32 + lane;
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) {
            if (!lower) break;
            const float4 x = src[nt * 32];
            tile[nt][0] = x.x, tile[nt][1] = x.y, tile[nt][2] = x.z, tile[nt][3] = x.w;
          }
        } else if (lower) {
          warp_gemm<T, 4, K / 16, A_ROW, B_NK>(tile, qS + r0 * LDK, LDK, kS + cc0 * LDK, LDK, lane);
        }
        if (lower) warp_gemm<T, 4, V / 16, A_ROW, B_NK>(accP, stage_do(s) + r0 * LDV, LDV, stage_v(s) + cc0 * LDV, LDV, lane);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = r0 + g + ((e >> 1) << 3), j = cc0 + nt * 8 + 2 * t + (e & 1);
            const RowScalars& rs = (e >> 1) ? rs1 : rs0;
            const bool seen = lower && j <= i && (one_run || runs[j] == rs.run);
            const float w = seen ? p.scale * __expf(rs.G - Gs[j]) : 0.f;
            const float dp = accP[nt][e] * w;
            sumP[nt][e] += dp;
            accP[nt][e] = dp * tile[nt][e];
            tile[nt][e] *= w;
          }
        }
        store_acc<T, 4>(Ps, LDC, r0, cc0, tile, lane);
        asm volatile("bar.arrive 1, 512;" ::: "memory");  // P of this head is complete (the key group waits for it)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          row0 += accP[nt][0] + accP[nt][1], row1 += accP[nt][2] + accP[nt][3];
          float a = accP[nt][0] + accP[nt][2], b = accP[nt][1] + accP[nt][3];
#pragma unroll
          for (int off = 4; off < 32; off <<= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, off);
            b += __shfl_xor_sync(0xffffffffu, b, off);
          }
          if (lane < 4) {
            *reinterpret_cast<float2*>(out + 256 + quad * 64 + cc0 + nt * 8 + 2 * lane) = make_float2(-a, -b);
          }
        }
        row0 += __shfl_xor_sync(0xffffffffu, row0, 1), row0 += __shfl_xor_sync(0xffffffffu, row0, 2);
        row1 += __shfl_xor_sync(0xffffffffu, row1, 1), row1 += __shfl_xor_sync(0xffffffffu, row1, 2);
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {  // scale (cin Gamma)(dO S^T); in halves, which bounds the registers
        const int col = kc0 + half * HN * 8;
        float x[HN][4], d0, d1;
        zero_acc(x);
        warp_gemm<T, HN, V / 16, A_ROW, B_NK>(x, stage_do(s) + r0 * LDV, LDV, stage_s(s) + col * LDV, LDV, lane);
        const float s0 = p.scale * rs0.gam, s1 = p.scale * rs1.gam;
#pragma unroll
        for (int nt = 0; nt < HN; ++nt) {
          x[nt][0] *= s0, x[nt][1] *= s0, x[nt][2] *= s1, x[nt][3] *= s1;
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[half * HN + nt][e] += x[nt][e];
        }
        row_dots<T, HN>(x, qS, LDK, r0, col, lane, d0, d1);
        row0 += d0, row1 += d1;
      }
    } else {
      float tail = 0.f;
#pragma unroll
      for (int half = 0; half < 2; ++half) {  // (tail Gamma_r)(V dS+^T)
        const int col = kc0 + half * HN * 8;
        float x[HN][4], d0, d1;
        zero_acc(x);
        warp_gemm<T, HN, V / 16, A_ROW, B_NK>(x, stage_v(s) + r0 * LDV, LDV, stage_ds(s) + col * LDV, LDV, lane);
#pragma unroll
        for (int nt = 0; nt < HN; ++nt) {
          x[nt][0] *= rs0.gamr, x[nt][1] *= rs0.gamr, x[nt][2] *= rs1.gamr, x[nt][3] *= rs1.gamr;
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[half * HN + nt][e] += x[nt][e];
        }
        row_dots<T, HN>(x, kS, LDK, r0, col, lane, d0, d1);
        row0 -= d0, row1 -= d1;
        tail += d0 + d1;
      }
      if (t != 0) tail = 0.f;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) tail += __shfl_xor_sync(0xffffffffu, tail, off);
      if (lane == 0) out[512 + 8 + warp] = tail;
      // dV
      float x[ONT][4];
      zero_acc(x);
      warp_gemm<T, ONT, K / 16, A_ROW, B_KN>(x, kS + r0 * LDK, LDK, stage_ds(s) + c0, LDV, lane);
#pragma unroll
      for (int nt = 0; nt < ONT; ++nt) {
        x[nt][0] *= rs0.gamr, x[nt][1] *= rs0.gamr, x[nt][2] *= rs1.gamr, x[nt][3] *= rs1.gamr;
      }
      // <S, dS+>, while the query group may still be busy with P
      float part = 0.f;
      const T* SS = stage_s(s);
      const T* dSS = stage_ds(s);
      for (int idx = tid - 256; idx < K * (V / 8); idx += 256) {
        const int r = idx / (V / 8), at = r * LDV + (idx - r * (V / 8)) * 8;
        const uint4 a = *reinterpret_cast<const uint4*>(SS + at), b = *reinterpret_cast<const uint4*>(dSS + at);
        const uint32_t as[4] = {a.x, a.y, a.z, a.w}, bs[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 u = unpack2<T>(as[i]), w = unpack2<T>(bs[i]);
          part += u.x * w.x + u.y * w.y;
        }
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
      if (lane == 0) out[512 + warp] = keep_gamma(Gs, runs, m.flags) * part;
      asm volatile("bar.sync 1, 512;" ::: "memory");
      warp_gemm<T, ONT, 4, A_COL, B_KN>(x, Ps + r0, LDC, stage_do(s) + c0, LDV, lane);
      store_acc_wide<T, ONT>(static_cast<T*>(p.dv_out) + ((long)(m.tok0 + r0) * p.H + h) * V + c0, (long)p.H * V, x, lane,
                             m.len - r0);
    }
    if (t == 0) {
      float* rows = out + (keys ? 128 : 0) + ch * 64 + r0 + g;
      rows[0] = row0, rows[8] = row1;
    }
  }

  // The sum of the heads' dP tiles may leave the range of f16 where each of them is inside: their mean is taken then.
  bool over = false;
  if (NH > 1 && std::is_same<T, __half>::value) {
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
      for (int e = 0; e < 4; ++e) over |= !(fabsf(sumP[nt][e]) <= 65504.f);
    }
  }
  over = __syncthreads_or(over);  // every head's terms are complete, P is free
  auto scale_acc = [&](float x) {
#pragma unroll
    for (int nt = 0; nt < KNT; ++nt) {
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[nt][e] *= x;
    }
  };
  constexpr float kMean = 1.f / NH;
  const float share = over ? kMean : 1.f;
  if (p.dg && tid < 32) write_dg(NH - 1);
  if (!keys) store_acc<T, 4>(P0, LDC, r0, cc0, sumP, lane, share, share);
  if (over) scale_acc(kMean);
  __syncthreads();
  if (!keys) warp_gemm<T, KNT, 4, A_ROW, B_KN>(acc, P0 + r0 * LDC, LDC, kS + kc0, LDK, lane);
  else warp_gemm<T, KNT, 4, A_COL, B_KN>(acc, P0 + r0, LDC, qS + kc0, LDK, lane);
  if (over) scale_acc(NH);
  float* sums = keys ? p.dk_acc : p.dq_acc;
  T* direct = static_cast<T*>(keys ? p.dk : p.dq);
#pragma unroll
  for (int nt = 0; nt < KNT; ++nt) {
    const int col = kc0 + nt * 8 + 2 * t;
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      if (r0 + g + 8 * hh >= m.len) continue;
      const long tok = (long)m.tok0 + r0 + g + 8 * hh;
      if (sums) {
        *reinterpret_cast<float2*>(sums + (tok * hgs + hg) * K + col) = make_float2(acc[nt][2 * hh], acc[nt][2 * hh + 1]);
      } else {
        *reinterpret_cast<uint32_t*>(direct + (tok * p.Hk + hk) * K + col) = pack2<T>(acc[nt][2 * hh], acc[nt][2 * hh + 1]);
      }
    }
  }
}

template <typename T, int K, int V>
int launch_delta(const BwdParams& bp, int blocks, cudaStream_t s) {
  constexpr int smem = GradSmem<T, K, V>::kBytes;
  auto* kern = sg_chunk_grads_kernel<T, K, V>;
  JLA_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  ProfScope ps(kProfSgChunkGrads, s);
  kern<<<blocks, 256, smem, s>>>(bp);
  JLA_LAUNCH_OK();
  return JLA_OK;
}

template <typename T, int K, int V, int NH>
int launch_decay_nh(const BwdParams& bp, int blocks, cudaStream_t s) {
  constexpr int smem = DecayGradSmem<T, K, V>::kAllocBytes;
  auto* kern = decay_grads_kernel<T, K, V, NH>;
  JLA_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  ProfScope ps(kProfSgChunkGrads, s);
  kern<<<blocks / NH, 512, smem, s>>>(bp);
  JLA_LAUNCH_OK();
  return JLA_OK;
}

template <typename T, int K, int V>
int launch_decay(const BwdParams& bp, int blocks, int walk, cudaStream_t s) {
  if constexpr (V == 64) {
    if (walk == 8) return launch_decay_nh<T, K, V, 8>(bp, blocks, s);
    if (walk == 4) return launch_decay_nh<T, K, V, 4>(bp, blocks, s);
    if (walk == 2) return launch_decay_nh<T, K, V, 2>(bp, blocks, s);
  }
  return launch_decay_nh<T, K, V, 1>(bp, blocks, s);
}

template <typename T, int K, int V>
int launch_one(const BwdParams& bp, bool delta, int blocks, int walk, cudaStream_t s) {
  return delta ? launch_delta<T, K, V>(bp, blocks, s) : launch_decay<T, K, V>(bp, blocks, walk, s);
}

template <typename T>
int launch_kv(const BwdParams& bp, const jla_problem& p, bool delta, int blocks, int walk, cudaStream_t s) {
  if (p.K == 128) {
    return p.V == 128 ? launch_one<T, 128, 128>(bp, delta, blocks, walk, s) : launch_one<T, 128, 64>(bp, delta, blocks, walk, s);
  }
  return p.V == 128 ? launch_one<T, 64, 128>(bp, delta, blocks, walk, s) : launch_one<T, 64, 64>(bp, delta, blocks, walk, s);
}

}  // namespace

int launch_sg_bwd(const ChunkedCtx& c, const jla_bwd_io& io, char* scratch, cudaStream_t s) {
  const jla_problem& p = c.p;
  const Plan& pl = c.plan;
  const long tokens = (long)p.B * p.T;
  if (pl.rows == 0) return JLA_OK;
  const bool kda = p.kind == JLA_KIND_KDA;
  const bool direct = p.H == p.Hk && !pl.l2norm;
  BwdParams bp{};
  bp.meta = reinterpret_cast<const ChunkMeta*>(c.res + pl.meta);
  bp.gates = reinterpret_cast<const float*>(c.res + pl.gates);
  bp.runs = reinterpret_cast<const unsigned char*>(c.res + pl.runs);
  bp.q = c.q_eff;
  bp.k = c.k_eff;
  bp.v = p.v;
  bp.t0 = c.res + pl.t0;
  bp.d_o = io.d_o;
  bp.h = c.res + pl.h;
  bp.vn = c.res + pl.vn;
  bp.dh = scratch + pl.dh;
  bp.dvn = scratch + pl.dvn;
  bp.dv = bp.dv_out = io.dv;
  bp.dq = io.dq;
  bp.dk = io.dk;
  bp.dq_acc = direct ? nullptr : reinterpret_cast<float*>(scratch + pl.dq_acc);
  bp.dk_acc = direct ? nullptr : reinterpret_cast<float*>(scratch + pl.dk_acc);
  bp.dg = io.dg;
  bp.qk_tab = shares_scores(p) ? reinterpret_cast<const float*>(c.res + pl.qk_tab) : nullptr;
  bp.dbeta = io.dbeta;
  bp.H = p.H;
  bp.Hk = p.Hk;
  bp.scale = p.scale;
  const int cb = pl.nc * p.H;
  const bool legacy = !use_tc_kernels(p);  // mma.sync chunk gradients (row-major residuals)
  // heads per CTA walk of the gradient kernel without the delta rule (sums dq, dk over them in registers): grouped key
  // heads with 64 value channels only
  const int group = p.H / p.Hk;
  const int walk = (legacy && !direct && !pl.delta && p.V == 64) ? (group % 8 == 0 ? 8 : group % 4 == 0 ? 4 : group % 2 == 0 ? 2 : 1) : 1;
  int rc = legacy ? launch_split_bwd_state(c, io, scratch, s) : launch_sg_bwd_state_tc(c, io, scratch, s);
  if (rc == JLA_OK && legacy) {
    rc = p.dtype == JLA_DTYPE_BF16 ? launch_kv<__nv_bfloat16>(bp, p, pl.delta, cb, walk, s)
                                   : launch_kv<__half>(bp, p, pl.delta, cb, walk, s);
  }
  if (rc == JLA_OK && !legacy && (p.flags & JLA_FLAG_STATE_GRADS_ONLY)) return rc;
  if (rc == JLA_OK && !legacy) rc = kda ? launch_kda_grads(c, io, scratch, s) : launch_chunk_grads_tc(c, io, scratch, direct, s);
  if (rc != JLA_OK || direct) return rc;
  rc = finalize_key_grad(bp.dq_acc, p.q, io.dq, p.dtype, tokens, p.H / walk, p.Hk, p.K, pl.l2norm, s);
  if (rc != JLA_OK) return rc;
  return finalize_key_grad(bp.dk_acc, p.k, io.dk, p.dtype, tokens, p.H / walk, p.Hk, p.K, pl.l2norm, s);
}

}  // namespace jla
