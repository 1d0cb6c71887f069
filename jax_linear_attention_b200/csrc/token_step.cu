// One decoding step: every row of the call is a single token with a state coming in and a state going out.
//
//   S' = exp(g) S (per head, or per key channel);  u = beta (v - k_read S')  (delta rule; v without it)
//   S+ = S' + k u^T;   o = scale q S+ = scale (q S' + (q . k) u)
//
// Bound by HBM: the fp32 state is read once and written once (2 * K * V * 4 bytes per head; the tokens themselves are
// a few hundred bytes), so the kernel is one pass with the state in registers. A CTA of 256 threads owns VB (128 or 64)
// value columns of one head: thread = (key slice, four adjacent columns), all of its 16-byte state loads are issued
// before anything else happens, and the norms and dot products of the key vectors are formed by the first warp while
// they are in flight. Both key reductions (k S' and q S') go through shared memory together, one barrier each way.
// The chunk kernels ran these calls as chunks of one valid token out of 64: 109 us of kernels for B64 H16 K = V = 128,
// where the state traffic (134 MB) takes 21 us at the measured copy rate.
//
// JLA_FLAG_SAVE_RESIDUALS calls keep the chunk kernels, whose backward needs their residuals. All arithmetic is fp32.
//
// The SSD form (jla_ssd_step) takes Mamba-2's layer inputs instead of v and g: v = round(x * dt), g = dt * A, and
// y = round(round(o) + D * x), the roundings of the glue kernels of ssd_glue.cu around the op.
#include "common.cuh"
#include "profile.cuh"

namespace jla {
namespace {

constexpr int NT = 256;

struct StepParams {
  int H, Hk, V;
  int l2norm;
  float scale;
  const void *q, *k, *k_read, *v;
  const float *g, *beta, *h0;
  void* o;
  float* final_state;
  int wide_in, wide_out;    // the states are 16-byte aligned (else four-byte accesses)
  const float *dt, *a, *d;  // SSD form (dt != nullptr): v is x, g is unused, d may be nullptr
};

enum { kNoGate = 0, kHeadGate = 1, kChannelGate = 2 };

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
  return x;
}

template <typename T, int K, int VB, int GATE, bool DELTA>
__global__ void __launch_bounds__(NT) token_step_kernel(StepParams p) {
  constexpr int CT = VB / 4;    // threads across the columns
  constexpr int NG = NT / CT;   // key slices
  constexpr int RPT = K / NG;   // state rows of a thread
  constexpr int KPL = K / 32;   // key channels of a lane of the first warp
  static_assert(K % NG == 0 && K % 32 == 0, "key slices");
  __shared__ float qs[K], ks[K], ws[DELTA ? K : 1], eg[GATE == kChannelGate ? K : 1];  // ws: the read key
  __shared__ float4 red[2][NG][CT];
  __shared__ float qk_s;
  const int tid = threadIdx.x, lane = tid & 31, cg = tid % CT, ng = tid / CT;
  const int vblocks = p.V / VB, per_row = p.H * vblocks;
  const int b = blockIdx.x / per_row, hc = blockIdx.x - b * per_row;  // batch row; its head and block of columns
  const int h = hc / vblocks, v0 = (hc - h * vblocks) * VB + 4 * cg;
  const long row = (long)b * p.H + h;  // (batch row, value head)
  const int hk = h / (p.H / p.Hk);

  float4 S[RPT];
  const float* sin = p.h0 ? p.h0 + row * K * p.V + (long)(ng * RPT) * p.V + v0 : nullptr;
  if (!sin || p.wide_in) {
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      S[i] = sin ? *reinterpret_cast<const float4*>(sin + (long)i * p.V) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  } else {
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const float* x = sin + (long)i * p.V;
      S[i] = make_float4(x[0], x[1], x[2], x[3]);
    }
  }

  if (tid < 32) {
    const long key = ((long)b * p.Hk + hk) * K;
    float q[KPL], k[KPL];
    float sq = 0.f, sk = 0.f;
#pragma unroll
    for (int i = 0; i < KPL; ++i) {
      q[i] = to_f32(static_cast<const T*>(p.q)[key + lane + 32 * i]);
      k[i] = to_f32(static_cast<const T*>(p.k)[key + lane + 32 * i]);
      sq += q[i] * q[i];
      sk += k[i] * k[i];
    }
    if (p.l2norm) {  // normalised in fp32 and rounded to the tensors' dtype (reference.py:65-69)
      const float iq = rsqrtf(warp_sum(sq) + 1e-6f), ik = rsqrtf(warp_sum(sk) + 1e-6f);
#pragma unroll
      for (int i = 0; i < KPL; ++i) {
        q[i] = to_f32(from_f32<T>(q[i] * iq));
        k[i] = to_f32(from_f32<T>(k[i] * ik));
      }
    }
    float qk = 0.f;
#pragma unroll
    for (int i = 0; i < KPL; ++i) {
      qk += q[i] * k[i];
      qs[lane + 32 * i] = q[i];
      ks[lane + 32 * i] = k[i];
      if (DELTA) ws[lane + 32 * i] = p.k_read ? to_f32(static_cast<const T*>(p.k_read)[row * K + lane + 32 * i]) : k[i];
    }
    qk = warp_sum(qk);
    if (lane == 0) qk_s = qk;
  } else if (GATE == kChannelGate) {
    for (int c = tid - 32; c < K; c += NT - 32) eg[c] = expf(p.g[row * K + c]);
  }
  float gamma = 1.f;
  if (GATE == kHeadGate) gamma = expf(p.dt ? p.dt[row] * p.a[h] : p.g[row]);
  const float beta = DELTA ? p.beta[row] : 1.f;
  float xv[4], u[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) xv[c] = to_f32(static_cast<const T*>(p.v)[row * p.V + v0 + c]);
#pragma unroll
  for (int c = 0; c < 4; ++c) u[c] = p.dt ? to_f32(from_f32<T>(xv[c] * p.dt[row])) : xv[c];
  __syncthreads();

  float4 rk = make_float4(0.f, 0.f, 0.f, 0.f), ro = rk;
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int kr = ng * RPT + i;
    const float e = GATE == kChannelGate ? eg[kr] : gamma;
    if (GATE != kNoGate) S[i].x *= e, S[i].y *= e, S[i].z *= e, S[i].w *= e;
    const float qi = qs[kr];
    ro.x += qi * S[i].x, ro.y += qi * S[i].y, ro.z += qi * S[i].z, ro.w += qi * S[i].w;
    if (DELTA) {
      const float wi = ws[kr];
      rk.x += wi * S[i].x, rk.y += wi * S[i].y, rk.z += wi * S[i].z, rk.w += wi * S[i].w;
    }
  }
  red[0][ng][cg] = ro;
  if (DELTA) red[1][ng][cg] = rk;
  __syncthreads();
  if (DELTA) {
    float4 r = red[1][0][cg];
#pragma unroll
    for (int n = 1; n < NG; ++n) {
      const float4 x = red[1][n][cg];
      r.x += x.x, r.y += x.y, r.z += x.z, r.w += x.w;
    }
    u[0] = beta * (u[0] - r.x), u[1] = beta * (u[1] - r.y), u[2] = beta * (u[2] - r.z), u[3] = beta * (u[3] - r.w);
  }
  if (p.final_state) {
    float* sout = p.final_state + row * K * p.V + (long)(ng * RPT) * p.V + v0;
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const float ki = ks[ng * RPT + i];
      const float4 x = make_float4(S[i].x + ki * u[0], S[i].y + ki * u[1], S[i].z + ki * u[2], S[i].w + ki * u[3]);
      float* y = sout + (long)i * p.V;
      if (p.wide_out) *reinterpret_cast<float4*>(y) = x;
      else y[0] = x.x, y[1] = x.y, y[2] = x.z, y[3] = x.w;
    }
  }
  if (ng == 0 && p.o) {
    float4 r = red[0][0][cg];
#pragma unroll
    for (int n = 1; n < NG; ++n) {
      const float4 x = red[0][n][cg];
      r.x += x.x, r.y += x.y, r.z += x.z, r.w += x.w;
    }
    const float qk = qk_s;
    T* o = static_cast<T*>(p.o) + row * p.V + v0;
    const float y[4] = {r.x + qk * u[0], r.y + qk * u[1], r.z + qk * u[2], r.w + qk * u[3]};
    const float skip = p.d ? p.d[h] : 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const T oc = from_f32<T>(p.scale * y[c]);
      o[c] = p.d ? from_f32<T>(to_f32(oc) + skip * xv[c]) : oc;
    }
  }
}

template <typename T, int K, int VB>
int launch_gate(const StepParams& sp, int kind, dim3 grid, cudaStream_t s) {
  ProfScope ps(kProfTokenStep, s);
  switch (kind) {
    case JLA_KIND_SIMPLE_GLA: token_step_kernel<T, K, VB, kHeadGate, false><<<grid, NT, 0, s>>>(sp); break;
    case JLA_KIND_DELTANET: token_step_kernel<T, K, VB, kNoGate, true><<<grid, NT, 0, s>>>(sp); break;
    case JLA_KIND_GATED_DELTANET: token_step_kernel<T, K, VB, kHeadGate, true><<<grid, NT, 0, s>>>(sp); break;
    default: token_step_kernel<T, K, VB, kChannelGate, true><<<grid, NT, 0, s>>>(sp); break;
  }
  JLA_LAUNCH_OK();
  return JLA_OK;
}

template <typename T>
int launch_dims(const StepParams& sp, const jla_problem& p, cudaStream_t s) {
  const int vb = p.V % 128 == 0 ? 128 : 64;
  const dim3 grid((unsigned)((long)p.B * p.H * (p.V / vb)));  // (below 2^31: token_step_applies)
  switch (p.K) {
    case 64: return vb == 128 ? launch_gate<T, 64, 128>(sp, p.kind, grid, s) : launch_gate<T, 64, 64>(sp, p.kind, grid, s);
    case 128: return vb == 128 ? launch_gate<T, 128, 128>(sp, p.kind, grid, s) : launch_gate<T, 128, 64>(sp, p.kind, grid, s);
    default: return vb == 128 ? launch_gate<T, 256, 128>(sp, p.kind, grid, s) : launch_gate<T, 256, 64>(sp, p.kind, grid, s);
  }
}

bool aligned16(const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15) == 0; }

StepParams base_params(const jla_problem& p, void* o, float* final_state) {
  StepParams sp{};
  sp.H = p.H, sp.Hk = p.Hk, sp.V = p.V;
  sp.l2norm = (p.flags & JLA_FLAG_QK_L2NORM) != 0;
  sp.scale = p.scale;
  sp.q = p.q, sp.k = p.k, sp.k_read = p.k_read, sp.v = p.v, sp.g = p.g, sp.beta = p.beta, sp.h0 = p.h0;
  sp.o = o, sp.final_state = final_state;
  sp.wide_in = aligned16(p.h0), sp.wide_out = aligned16(final_state);
  return sp;
}

int launch_dtype(const StepParams& sp, const jla_problem& p, cudaStream_t s) {
  switch (p.dtype) {
    case JLA_DTYPE_BF16: return launch_dims<__nv_bfloat16>(sp, p, s);
    case JLA_DTYPE_F16: return launch_dims<__half>(sp, p, s);
    default: return launch_dims<float>(sp, p, s);
  }
}

}  // namespace

// Whether a forward is a decoding step that this file runs: one token per dense row (a single token never restarts its
// row's state, so segment_ids do not matter), nothing to keep for a backward, states in whole 16-byte groups. The
// explicitly requested chunk kernels (JLA_PATH_CHUNKED) are left alone.
bool token_step_applies(const jla_problem& p) {
  return p.T == 1 && p.B > 0 && p.num_seqs == 0 && p.path != JLA_PATH_CHUNKED &&
         !(p.flags & (JLA_FLAG_SAVE_RESIDUALS | JLA_FLAG_PREP_DONE)) && (p.K == 64 || p.K == 128 || p.K == 256) &&
         p.V % 64 == 0 && (long)p.B * p.H * (p.V / 64) < (1L << 31);
}

int token_step_fwd(const jla_problem& p, const jla_fwd_io& io, cudaStream_t s) {
  return launch_dtype(base_params(p, io.o, io.final_state), p, s);
}

}  // namespace jla

using namespace jla;

extern "C" int jla_ssd_step(const jla_problem* p, const float* dt, const float* a, const float* d, void* y,
                            float* final_state, jla_stream_t stream) {
  if (!p || !dt || !a || !y || !p->q || !p->k || !p->v) {
    set_error("ssd step: null argument");
    return JLA_ERR_BAD_ARGUMENT;
  }
  if (p->kind != JLA_KIND_SIMPLE_GLA || p->dtype == JLA_DTYPE_F32 || p->k_read || p->Hk <= 0 || p->H <= 0 ||
      p->H % p->Hk || !token_step_applies(*p)) {
    set_error("ssd step: one 16-bit token per row, N in (64, 128, 256), P a multiple of 64");
    return JLA_ERR_UNSUPPORTED;
  }
  StepParams sp = base_params(*p, y, final_state);
  sp.dt = dt, sp.a = a, sp.d = d;
  return launch_dtype(sp, *p, static_cast<cudaStream_t>(stream));
}
