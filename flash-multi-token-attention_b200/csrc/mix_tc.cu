// Driver of the tensor-core head-mix path (mix_tc.cuh): workspace layout, chunking over (batch, group) units, launches.
#include "mix_tc.cuh"

namespace fmta {

namespace {

inline size_t up(size_t x) { return (x + 1023) / 1024 * 1024; }

// P (and dC) of one (batch, group) unit takes 2 (4) bytes per entry of the N x N score matrices of its G heads, so a launch
// handles as many units as fit kMixChunkBytes: enough CTAs for the GPU, and a workspace that does not grow with the batch.
// A unit above kMixUnitMax is left to the kernels that need no such buffers.
constexpr size_t kMixChunkBytes = (size_t)4500 << 20, kMixUnitMax = (size_t)16 << 30;

struct MixPlan {
  int nRT, N8, RP, U, nU, nKC, kch;
  size_t unit;            // bytes of one operand tensor (P or dC) of a unit
  size_t kt, cband, dkt, theta_part, dw_part, stat, x8;      // bytes of the workspace's parts (0: absent)
  size_t rows;
  int theta_band_slots, theta_post_slots, dw_slots;
};

MixPlan plan(int B, int H, int N, int d, int cq, int ck, int G, bool conv, bool causal, bool bwd) {
  MixPlan m = {};
  m.nRT = (N + 127) / 128; m.N8 = m.nRT * 128; m.RP = m.N8 + 16;
  m.U = B * (H / G);
  m.unit = (size_t)G * (m.N8 / 8) * m.RP * 16;
  const size_t per = m.unit * (bwd ? 2 : 1);
  m.nU = (int)(kMixChunkBytes / per);
  m.nU = m.nU < 1 ? 1 : (m.nU > m.U ? m.U : m.nU);
  // keys per CTA: long chunks keep the row tile's operands and amortise the fixed cost of a CTA; about three CTAs per SM
  // (dead ones above the diagonal not counted) even out the load
  m.kch = 1024;
  auto live = [&]() { return (long)m.nRT * ((m.N8 + m.kch - 1) / m.kch) * m.nU / (causal ? 2 : 1); };
  while (m.kch > 128 && live() < 3 * 148) m.kch /= 2;
  // a GPU that is not full: half as long CTAs (a block is at most 64 keys there; with a filter a CTA's fixed cost is larger)
  if (live() < (conv ? 74 : 148) && G >= (conv ? 4 : 8)) m.kch = 64;
  m.nKC = (m.N8 + m.kch - 1) / m.kch;
  m.rows = (size_t)B * H * N;
  const int band = (cq - 1) + (ck - 1) / 2;
  if (conv) {
    m.kt = up(m.rows * cq * 2 * d * 2);
    if (causal) m.cband = up(m.rows * (band > 0 ? band : 1) * 4);
    if (bwd) {
      m.dkt = up(m.rows * cq * 2 * d * 2);
      m.theta_band_slots = causal ? bwd_band_theta_slots(B, N, cq, ck) : 0;
      m.theta_post_slots = bwd_tc_theta_slots(B, N, d);
      m.theta_part = up((size_t)(m.theta_band_slots + m.theta_post_slots) * H * cq * ck * 4);
    }
  }
  if (bwd) {
    m.dw_slots = B * m.nRT * m.nKC;
    m.dw_part = up((size_t)m.dw_slots * H * G * 4);
  } else {
    m.stat = up((size_t)m.nU * G * 2 * m.nKC * 3 * m.RP * 4);
  }
  m.x8 = up((size_t)m.nU * m.unit);
  return m;
}

}  // namespace

bool mix_tc_supported(const TrainParams& p) {
  if (!p.Wmix || !tensor_maps_available()) return false;
  if (p.G != 2 && p.G != 4 && p.G != 8 && p.G != 16) return false;
  if ((p.d != 64 && p.d != 128) || (p.theta && p.cq > 7)) return false;
  const size_t n8 = (size_t)(p.N + 127) / 128 * 128;
  return (size_t)p.G * (n8 / 8) * (n8 + 16) * 32 <= kMixUnitMax;
}

// Neither the causal flag nor the presence of a filter is an argument of fmta_workspace_bytes: the most of all.
size_t mix_tc_workspace_bytes(int B, int H, int N, int d, int cq, int ck, int G, bool bwd) {
  if (G < 2 || H % G != 0) return 0;
  size_t most = 0;
  for (int causal = 0; causal < 2; ++causal) {
    const MixPlan m = plan(B, H, N, d, cq, ck, G, true, causal, bwd);
    size_t n = 2048 + m.kt + m.cband * (bwd ? 2 : 1) + m.dkt + m.theta_part + m.dw_part + m.stat + m.x8 * (bwd ? 2 : 1);
    if (bwd) n += up(m.rows * 4) + up(m.rows * d * 2) + (causal ? 2 * up(m.rows * d * 4) : 0);
    if (n > most) most = n;
  }
  return most;
}

static void fill(MixParams& q, const TrainParams& p, const MixPlan& m, int* status) {
  q = MixParams{};
  q.W = p.Wmix; q.LSE = p.LSE; q.Dvec = p.Dvec; q.status = status;
  q.B = p.B; q.H = p.H; q.N = p.N; q.G = p.G; q.cq = p.cq; q.ck = p.ck; q.causal = p.causal;
  q.nRT = m.nRT; q.nKC = m.nKC; q.kch = m.kch; q.RP = m.RP; q.N8 = m.N8;
  q.c2 = p.theta ? 1.f : p.scale * kLog2e;
  q.cw = p.theta ? kLn2 : p.scale;
}

#define FMTA_TRY(x) do { const cudaError_t e_ = (x); if (e_ != cudaSuccess) return e_; } while (0)

cudaError_t launch_mix_fwd(const TrainParams& p_, void* workspace, cudaStream_t stream) {
  TrainParams p = p_;
  const MixPlan m = plan(p.B, p.H, p.N, p.d, p.cq, p.ck, p.G, p.theta != nullptr, p.causal, false);
  unsigned char* w = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(workspace) + 1023) & ~uintptr_t(1023));
  int* status = nullptr;
  FMTA_TRY(status_word_of(reinterpret_cast<int*>(w), stream, &status)); w += 1024;
  __nv_bfloat16* Kt = reinterpret_cast<__nv_bfloat16*>(w); w += m.kt;
  MixParams q;
  fill(q, p, m, status);
  if (p.theta) {
    FMTA_TRY(launch_ktilde(p, Kt, stream, true));
    if (p.causal) { p.Cband = reinterpret_cast<float*>(w); q.Cband = p.Cband; w += m.cband; FMTA_TRY(launch_band_scores(p, stream)); }
  }
  q.stat = reinterpret_cast<float*>(w); w += m.stat;
  q.P8 = reinterpret_cast<bf16*>(w);
  for (q.u0 = 0; q.u0 < m.U; q.u0 += m.nU) {
    q.nU = m.U - q.u0 < m.nU ? m.U - q.u0 : m.nU;
    FMTA_TRY(launch_mix_score(p, q, Kt, false, stream));
    FMTA_TRY(launch_mix_pv(p, q, stream));
  }
  return cudaSuccess;
}

// dO / O in do_f32 / o_bf16; want: 1 = dQ (and dTheta, dW), 2 = dK, dV, 3 = all
cudaError_t launch_mix_bwd(const TrainParams& p_, const void* dO, bool do_f32, const void* O, bool o_bf16, float* dTheta, float* dW, int want,
                           void* workspace, cudaStream_t stream) {
  TrainParams p = p_;
  const bool conv = p.theta != nullptr;
  const MixPlan m = plan(p.B, p.H, p.N, p.d, p.cq, p.ck, p.G, conv, p.causal, true);
  unsigned char* w = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(workspace) + 1023) & ~uintptr_t(1023));
  auto take = [&](size_t n) { unsigned char* r = w; w += n; return r; };
  int* status = nullptr;
  FMTA_TRY(status_word_of(reinterpret_cast<int*>(take(1024)), stream, &status));
  __nv_bfloat16* Kt = reinterpret_cast<__nv_bfloat16*>(take(m.kt));
  if (conv && p.causal) { p.Cband = reinterpret_cast<float*>(take(m.cband)); p.dCband = reinterpret_cast<float*>(take(m.cband)); }
  __nv_bfloat16* dKt = reinterpret_cast<__nv_bfloat16*>(take(m.dkt));
  float* theta_part = reinterpret_cast<float*>(take(m.theta_part));
  float* dw_part = reinterpret_cast<float*>(take(m.dw_part));
  float* D = reinterpret_cast<float*>(take(up(m.rows * 4)));
  bf16* dOb = reinterpret_cast<bf16*>(take(up(m.rows * p.d * 2)));
  if (conv && p.causal) { p.dQ = reinterpret_cast<float*>(take(up(m.rows * p.d * 4))); p.dK = reinterpret_cast<float*>(take(up(m.rows * p.d * 4))); }
  p.dV = nullptr;
  FMTA_TRY(launch_rowdot(dO, O, o_bf16, do_f32 ? dOb : nullptr, D, m.rows, p.d, stream));
  p.dO = do_f32 ? dOb : reinterpret_cast<const __nv_bfloat16*>(dO);
  p.Dvec = D;
  MixParams q;
  fill(q, p, m, status);
  q.Cband = p.Cband; q.dCband = p.dCband; q.dW_part = dw_part;
  q.P8 = reinterpret_cast<bf16*>(take(m.x8)); q.C8 = reinterpret_cast<bf16*>(take(m.x8));
  if (conv) {
    FMTA_TRY(launch_ktilde(p, Kt, stream, true));
    if (p.causal) FMTA_TRY(launch_band_scores(p, stream));
  }
  p.dTheta_part = theta_part;
  for (q.u0 = 0; q.u0 < m.U; q.u0 += m.nU) {
    q.nU = m.U - q.u0 < m.nU ? m.U - q.u0 : m.nU;
    FMTA_TRY(launch_mix_score(p, q, Kt, true, stream));
    if (conv && p.causal) FMTA_TRY(launch_bwd_band_given(p, q.u0 * p.G, q.nU * p.G, stream));
    if (want & 1) FMTA_TRY(launch_mix_dq(p, q, Kt, stream));
    if ((want & 2) || conv) FMTA_TRY(launch_mix_dkdv(p, q, dKt, want & 1, stream));      // dTheta comes out of dKt
  }
  if (conv) {
    FMTA_TRY(launch_dk_post(p, dKt, true, theta_part + (size_t)m.theta_band_slots * p.H * p.cq * p.ck, status, stream));
    if (want & 1) FMTA_TRY(launch_reduce_partials(theta_part, dTheta, m.theta_band_slots + m.theta_post_slots, p.H * p.cq * p.ck, stream));
  }
  if (want & 1) FMTA_TRY(launch_reduce_partials(dw_part, dW, m.dw_slots, p.H * p.G, stream));
  return cudaSuccess;
}

}  // namespace fmta
