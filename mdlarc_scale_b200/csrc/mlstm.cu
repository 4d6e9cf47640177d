// Token-by-token form of the matrix-memory recurrence: the decode step, and prefill where the chunkwise
// kernel does not apply.
//
// One CTA owns one (sequence, head) and keeps the whole fp32 state in registers: thread (rg, c4) holds rows of four
// neighbouring value columns.  A decode step reads and writes the state once, 16 bytes a lane and contiguous across the
// warp, with all of a thread's loads in flight together; nothing else of the step is large, so the launch is bound by
// that traffic.  The head's RMS norm, gain and output gate are applied before the row leaves.
#include <atomic>

#include "launch.cuh"
#include "mlstm.cuh"

namespace {

template <int DMAX, int VP>
struct MlstmCfg {
  static constexpr int NT = (DMAX * VP / 64 > 256) ? DMAX * VP / 64 : 256;
  static constexpr int C4 = VP / 4;          // threads across the value columns
  static constexpr int RG = NT / C4;         // row groups
  static constexpr int RPT = DMAX / RG;      // rows per thread
  static constexpr int STEP_CTAS = RPT <= 4 ? 4 : RPT <= 8 ? 3 : NT <= 256 ? 2 : 1;   // of a decode step, on an SM
};

template <int DMAX, int VP>
__global__ void __launch_bounds__(MlstmCfg<DMAX, VP>::NT, (MlstmCfg<DMAX, VP>::STEP_CTAS))
mlstm_step_kernel(MlstmArgs a) {
  using C = MlstmCfg<DMAX, VP>;
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float s_q[DMAX], s_k[DMAX];
  __shared__ __align__(16) float s_red[C::RG][VP];
  __shared__ float s_nq[C::NT / 32], s_ss[C::NT / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int h = blockIdx.x, sg = blockIdx.y;
  const int row = sg, seq = sg, pos0 = a.pos[sg];
  bool held = pos0 < 0;
  if (seq >= a.n_seqs) {
    if (tid == 0) arcb_set_error(a.err, ARCB_DEV_BAD_INDEX);
    held = true;
  }
  if (held) {
    // a held row still feeds the next product: give it zeros
    if (tid < VP) st_act(a.out, ((size_t)row * a.H + h) * VP + tid, 0.f, a.fmt);
    return;
  }
  const int c4 = tid % C::C4, rg = tid / C::C4;
  float* Sg = a.S + ((size_t)seq * a.H + h) * a.dim * VP;
  float* ng = a.n + ((size_t)seq * a.H + h) * a.dimp;
  float* mg = a.m + (size_t)seq * a.H + h;

  float4 S[C::RPT];
  float n = 0.f, m = 0.f;
  const bool fresh = pos0 == 0;
#pragma unroll
  for (int j = 0; j < C::RPT; ++j) {
    const int r = rg + j * C::RG;
    S[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!fresh && r < a.dim) S[j] = *reinterpret_cast<const float4*>(Sg + (size_t)r * VP + c4 * 4);
  }
  if (!fresh) {
    if (tid < a.dim) n = ng[tid];
    m = *mg;
  }
  const float inv_v = 1.f / (float)a.vdim;
  const size_t base = (size_t)row * a.pitch;
  if (tid < DMAX) {
    s_q[tid] = tid < a.dim ? ld_act(a.proj, base + a.off_q + (size_t)h * a.dimp + tid, a.fmt) : 0.f;
    s_k[tid] = tid < a.dim ? ld_act(a.proj, base + a.off_k + (size_t)h * a.dimp + tid, a.fmt) : 0.f;
  }
  const float4 v = ld_act4(a.proj, base + a.off_v + (size_t)h * VP + c4 * 4, a.fmt);
  const float gi = gate_log(a.gates[(size_t)row * 2 * a.H + h], a.gate_cap, false);
  const float gf = gate_log(a.gates[(size_t)row * 2 * a.H + a.H + h], a.gate_cap, true);
  const float m_new = fmaxf(gf + m, gi);
  const float keep = expf(gf + m - m_new), add = expf(gi - m_new);
  m = m_new;
  __syncthreads();
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int j = 0; j < C::RPT; ++j) {
    const int r = rg + j * C::RG;
    const float kk = add * s_k[r], qq = s_q[r];
    S[j].x = fmaf(kk, v.x, keep * S[j].x);
    S[j].y = fmaf(kk, v.y, keep * S[j].y);
    S[j].z = fmaf(kk, v.z, keep * S[j].z);
    S[j].w = fmaf(kk, v.w, keep * S[j].w);
    acc.x = fmaf(S[j].x, qq, acc.x);
    acc.y = fmaf(S[j].y, qq, acc.y);
    acc.z = fmaf(S[j].z, qq, acc.z);
    acc.w = fmaf(S[j].w, qq, acc.w);
  }
  *reinterpret_cast<float4*>(&s_red[rg][c4 * 4]) = acc;
  float nq = 0.f;
  if (tid < DMAX) {
    n = fmaf(add, s_k[tid], keep * n);
    nq = n * s_q[tid];
  }
  if (tid < ((DMAX + 31) & ~31)) {
    nq = warp_sum(nq);
    if (lane == 0) s_nq[warp] = nq;
  }
  __syncthreads();
  float o = 0.f;
  if (tid < VP) {
#pragma unroll
    for (int j = 0; j < C::RG; ++j) o += s_red[j][tid];
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < (DMAX + 31) / 32; ++j) dot += s_nq[j];
    o /= fmaxf(fabsf(dot), expf(-m)) + 1e-6f;
    const float ss = warp_sum(o * o);     // padding columns are exactly zero
    if (lane == 0) s_ss[warp] = ss;
  }
  __syncthreads();
  if (tid < VP) {
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < VP / 32; ++j) ss += s_ss[j];
    o *= 1.f / sqrtf(ss * inv_v + a.eps);
    o *= a.norm_w[(size_t)h * VP + tid] * ld_act(a.proj, base + a.off_g + (size_t)h * VP + tid, a.fmt);
    st_act(a.out, ((size_t)row * a.H + h) * VP + tid, o, a.fmt);
  }
#pragma unroll
  for (int j = 0; j < C::RPT; ++j) {
    const int r = rg + j * C::RG;
    if (r < a.dim) *reinterpret_cast<float4*>(Sg + (size_t)r * VP + c4 * 4) = S[j];
  }
  if (tid < a.dim) ng[tid] = n;
  if (tid == 0) *mg = m;
}

// Segments of any length.  A walk is a chain of tokens, so what a token costs is latency: gates, decays and the head norm
// are taken for TC tokens at a time, beside the state's updates instead of between them, and the chunk's operands are
// fetched one chunk ahead.  Three barriers a chunk.  B200, 20 heads of 64 x 64, two segments of up to 999
// tokens in fp32: 1427 us token by token, 356 here.  REST: only the rows that mlstm_chunked_rows leaves.
template <int DMAX, int VP>
struct WalkCfg {
  using C = MlstmCfg<DMAX, VP>;
  static constexpr int TC = 2048 / C::NT;                 // tokens a chunk: 32 KB of partial rows
  static constexpr int ROW = 2 * DMAX + 2 * VP;           // operands of a token: q, k, v, output gate
  static constexpr int NL = TC * ROW / C::NT;             // of them a thread fetches
  static constexpr int SMEM = (2 * TC * ROW + TC * C::RG * VP + TC * DMAX) * 4;
};

template <int DMAX, int VP, bool REST = false>
__global__ void __launch_bounds__(MlstmCfg<DMAX, VP>::NT, 1)
mlstm_walk_kernel(MlstmArgs a) {
  using C = MlstmCfg<DMAX, VP>;
  using Wk = WalkCfg<DMAX, VP>;
  constexpr int TC = Wk::TC, ROW = Wk::ROW, NL = Wk::NL, WARPS = C::NT / 32, CPL = VP / 32;
  static_assert(C::RPT % 4 == 0 && TC <= 32 && TC * ROW % C::NT == 0, "sizes");
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  float* s_in = sm;                                       // [2][TC][ROW]
  float* s_red = sm + 2 * TC * ROW;                       // [TC][RG][VP]
  float* s_nq = s_red + TC * C::RG * VP;                  // [TC][DMAX]
  __shared__ float s_gl[2][TC], s_keep[TC], s_add[TC], s_floor[TC];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int h = blockIdx.x, sg = blockIdx.y;
  const int done = REST ? mlstm_chunked_rows(a.seg_rows[sg]) : 0;
  const int row0 = a.seg_row0[sg] + done, rows = a.seg_rows[sg] - done, seq = a.seg_seq[sg], pos0 = a.seg_pos0[sg] + done;
  if (seq < 0 || seq >= a.n_seqs) {
    if (tid == 0) arcb_set_error(a.err, ARCB_DEV_BAD_INDEX);
    return;
  }
  if (rows <= 0) return;
  const int c4 = tid % C::C4, rg = tid / C::C4;
  float* Sg = a.S + ((size_t)seq * a.H + h) * a.dim * VP;
  float* ng = a.n + ((size_t)seq * a.H + h) * a.dimp;
  float* mg = a.m + (size_t)seq * a.H + h;
  float4 S[C::RPT];
  float n = 0.f, m = 0.f;
  const bool fresh = pos0 == 0;
#pragma unroll
  for (int j = 0; j < C::RPT; ++j) {
    const int r = rg * C::RPT + j;
    S[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!fresh && r < a.dim) S[j] = *reinterpret_cast<const float4*>(Sg + (size_t)r * VP + c4 * 4);
  }
  if (!fresh) {
    if (tid < a.dim) n = ng[tid];
    m = *mg;
  }
  const float inv_v = 1.f / (float)a.vdim;
  float in[NL], gl = 0.f;
  auto fetch = [&](int t0) {
#pragma unroll
    for (int i = 0; i < NL; ++i) {
      const int e = tid + i * C::NT, t = t0 + e / ROW, c = e % ROW;
      in[i] = 0.f;
      if (t < rows) {
        const size_t at = (size_t)(row0 + t) * a.pitch;
        if (c < DMAX) { if (c < a.dim) in[i] = ld_act(a.proj, at + a.off_q + (size_t)h * a.dimp + c, a.fmt); }
        else if (c < 2 * DMAX) { if (c - DMAX < a.dim) in[i] = ld_act(a.proj, at + a.off_k + (size_t)h * a.dimp + c - DMAX, a.fmt); }
        else if (c < 2 * DMAX + VP) in[i] = ld_act(a.proj, at + a.off_v + (size_t)h * VP + c - 2 * DMAX, a.fmt);
        else in[i] = ld_act(a.proj, at + a.off_g + (size_t)h * VP + c - 2 * DMAX - VP, a.fmt);
      }
    }
    if (tid < 2 * TC && t0 + tid % TC < rows) gl = a.gates[(size_t)(row0 + t0 + tid % TC) * 2 * a.H + (tid < TC ? 0 : a.H) + h];
  };
  fetch(0);
  for (int t0 = 0, buf = 0; t0 < rows; t0 += TC, buf ^= 1) {
    float* cur = s_in + buf * TC * ROW;
#pragma unroll
    for (int i = 0; i < NL; ++i) cur[tid + i * C::NT] = in[i];
    if (tid < 2 * TC) s_gl[tid / TC][tid % TC] = gate_log(gl, a.gate_cap, tid >= TC);
    if (t0 + TC < rows) fetch(t0 + TC);
    const int nt = min(TC, rows - t0);
    __syncthreads();
    {
      // the stabiliser is a chain of two operations a token; its exponentials are one a lane
      float before = m, at = m;
      for (int t = 0; t < nt; ++t) {
        const float next = fmaxf(s_gl[1][t] + at, s_gl[0][t]);
        if (t == lane) { before = at; m = next; }
        at = next;
      }
      if (warp == 0 && lane < nt) {
        s_keep[lane] = expf(s_gl[1][lane] + before - m);
        s_add[lane] = expf(s_gl[0][lane] - m);
        s_floor[lane] = expf(-m);
      }
      m = at;
    }
    __syncthreads();
    for (int t = 0; t < nt; ++t) {
      const float* q = cur + t * ROW;
      const float* k = q + DMAX;
      const float4 v = *reinterpret_cast<const float4*>(k + DMAX + c4 * 4);
      const float keep = s_keep[t], add = s_add[t];
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int j = 0; j < C::RPT; j += 4) {
        const float4 k4 = *reinterpret_cast<const float4*>(k + rg * C::RPT + j), q4 = *reinterpret_cast<const float4*>(q + rg * C::RPT + j);
        const float kk[4] = {add * k4.x, add * k4.y, add * k4.z, add * k4.w}, qq[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float4& s = S[j + i];
          s.x = fmaf(kk[i], v.x, keep * s.x);
          s.y = fmaf(kk[i], v.y, keep * s.y);
          s.z = fmaf(kk[i], v.z, keep * s.z);
          s.w = fmaf(kk[i], v.w, keep * s.w);
          acc.x = fmaf(s.x, qq[i], acc.x);
          acc.y = fmaf(s.y, qq[i], acc.y);
          acc.z = fmaf(s.z, qq[i], acc.z);
          acc.w = fmaf(s.w, qq[i], acc.w);
        }
      }
      *reinterpret_cast<float4*>(s_red + (t * C::RG + rg) * VP + c4 * 4) = acc;
      if (tid < DMAX) {
        n = fmaf(add, k[tid], keep * n);
        s_nq[t * DMAX + tid] = n * q[tid];
      }
    }
    __syncthreads();
    for (int t = warp; t < nt; t += WARPS) {              // a warp finishes a token's row
      float dot = 0.f, o[CPL], ss = 0.f;
#pragma unroll
      for (int j = 0; j < DMAX / 32; ++j) dot += s_nq[t * DMAX + j * 32 + lane];
      dot = warp_sum(dot);
      const float den = fmaxf(fabsf(dot), s_floor[t]) + 1e-6f;
#pragma unroll
      for (int c = 0; c < CPL; ++c) {
        o[c] = 0.f;
#pragma unroll
        for (int j = 0; j < C::RG; ++j) o[c] += s_red[(t * C::RG + j) * VP + c * 32 + lane];
        o[c] /= den;
        ss += o[c] * o[c];                                // padding columns are exactly zero
      }
      const float norm = 1.f / sqrtf(warp_sum(ss) * inv_v + a.eps);
      const float* gate = cur + t * ROW + 2 * DMAX + VP;
#pragma unroll
      for (int c = 0; c < CPL; ++c) {
        const int u = c * 32 + lane;
        st_act(a.out, ((size_t)(row0 + t0 + t) * a.H + h) * VP + u, o[c] * norm * (a.norm_w[(size_t)h * VP + u] * gate[u]), a.fmt);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < C::RPT; ++j) {
    const int r = rg * C::RPT + j;
    if (r < a.dim) *reinterpret_cast<float4*>(Sg + (size_t)r * VP + c4 * 4) = S[j];
  }
  if (tid < a.dim) ng[tid] = n;
  if (tid == 0) *mg = m;
}

template <int DMAX, int VP>
cudaError_t launch_step(const MlstmArgs& a, cudaStream_t stream) {
  const dim3 grid(a.H, a.n_segs), block(MlstmCfg<DMAX, VP>::NT);
  if (!a.seg_seq) return arcb_launch(mlstm_step_kernel<DMAX, VP>, grid, block, 0, stream, a);
  return arcb_launch(mlstm_walk_kernel<DMAX, VP>, grid, block, WalkCfg<DMAX, VP>::SMEM, stream, a);
}

template <int DMAX, int VP>
cudaError_t init_walk() {
  return cudaFuncSetAttribute(mlstm_walk_kernel<DMAX, VP>, cudaFuncAttributeMaxDynamicSharedMemorySize, WalkCfg<DMAX, VP>::SMEM);
}

}  // namespace

// shared-memory opt-in of the walk (once per device, outside any capture)
int arcb_mlstm_walk_init() {
  cudaError_t e;
  if ((e = init_walk<64, 64>()) != cudaSuccess || (e = init_walk<64, 128>()) != cudaSuccess || (e = init_walk<64, 256>()) != cudaSuccess ||
      (e = init_walk<128, 64>()) != cudaSuccess || (e = init_walk<128, 128>()) != cudaSuccess || (e = init_walk<128, 256>()) != cudaSuccess ||
      (e = init_walk<256, 64>()) != cudaSuccess || (e = init_walk<256, 128>()) != cudaSuccess || (e = init_walk<256, 256>()) != cudaSuccess)
    return (int)e;
  return 0;
}

int arcb_launch_mlstm_rest64(const MlstmArgs& a, cudaStream_t stream) {
  static std::atomic<unsigned long long> opted{0};
  cudaError_t e = arcb_opt_in_smem(mlstm_walk_kernel<64, 64, true>, WalkCfg<64, 64>::SMEM, opted);
  if (e == cudaSuccess) e = arcb_launch(mlstm_walk_kernel<64, 64, true>, dim3(a.H, a.n_segs), dim3(MlstmCfg<64, 64>::NT), WalkCfg<64, 64>::SMEM, stream, a);
  arcb_count_launch(1);
  return (int)e;
}

int arcb_launch_mlstm_step(const MlstmArgs& a, cudaStream_t stream) {
  if (a.n_segs <= 0) return 0;
  if (a.n_segs > 65535) return -1;
  cudaError_t e = cudaErrorInvalidValue;
  switch (a.dimp * 1000 + a.vdimp) {
    case 64064: e = launch_step<64, 64>(a, stream); break;
    case 64128: e = launch_step<64, 128>(a, stream); break;
    case 64256: e = launch_step<64, 256>(a, stream); break;
    case 128064: e = launch_step<128, 64>(a, stream); break;
    case 128128: e = launch_step<128, 128>(a, stream); break;
    case 128256: e = launch_step<128, 256>(a, stream); break;
    case 256064: e = launch_step<256, 64>(a, stream); break;
    case 256128: e = launch_step<256, 128>(a, stream); break;
    case 256256: e = launch_step<256, 256>(a, stream); break;
  }
  arcb_count_launch(1);
  return (int)e;
}
