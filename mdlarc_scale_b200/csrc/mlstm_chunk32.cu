// Chunkwise prefill of the matrix-memory recurrence in 32 bits, heads of up to 64 x 64.
//
// The same unrolling as the 16-bit kernel's (mlstm_chunk.cu): chunks of 64 tokens, with F_t the running sum of the log forget gates,
// c_s = i_s - F_s and M_t = max(m, max_{s <= t} c_s),
//   num_t = exp(m - M_t) S^T q_t + sum_{s <= t} exp(c_s - M_t) (q_t . k_s) v_s,   S' = exp(m - M_L) S + sum_s exp(c_s - M_L) k_s v_s^T
// (n alike with k alone).  Running sums and exponents are taken in 64 bits: F may be large where only its differences count.
// Token by token the chain of a token's loads, updates and barriers costs 0.4 us; here a chunk is four 64 x 64 x 64 products of two-wide
// multiply-adds, a 4 x 4 tile a thread, operands in shared memory in the layout each product reads by quads, the next chunk's in
// registers.  What bounds it: a chunk is 14 us of products behind one another on one CTA an SM, 11 us of an SM's time on two.
//
// A chunk costs nearly the same whatever it holds, so few tokens are left to the walk (mlstm.cu): segments of up to C32_ALONE, and up to
// C32_TAIL behind the last whole chunk (mlstm_chunked_rows).  The rule looks at a segment's length alone and its chunks start at its
// first row, so its results depend on nothing else in the call.  B200, 20 heads, us of both launches / of the walk alone / of chunks
// alone; one segment: 36 rows 17.5 / 17.6 / 18.5, 40 16.1 / 18.7 / 17.5, 65 21.6 / 29.7 / 32.0, 80 26.3 / 34.5 / 32.0, 900 205 / 360 / 224;
// 64 segments: 8 rows 31 / 27 / 150, 30 85 / 82 / 163, 40 112 / 105 / 167, 48 121 / 124 / 173, 65 160 / 169 / 306, 80 189 / 199 / 309,
// 100 236 / 248 / 326, 200 409 / 475 / 594 (chunks alone: one CTA an SM, and all products of a chunk whatever it holds).
#include <atomic>

#include "gemm.cuh"
#include "launch.cuh"
#include "mlstm.cuh"

namespace {

constexpr int CL = C32_CHUNK, CD = 64, CP = 68;         // tokens of a chunk, columns of a head, pitch of a tile
constexpr int CT_THREADS = 256;
constexpr int TILE = 64 * CP;
// q^T, k^T, weighted k, v, scores^T, state
constexpr int C32_SMEM = 6 * TILE * 4;

// acc[i][j] += sum_k a[k][4 ty + i] * b[k][4 tx + j], k = 0 .. n - 1
__device__ __forceinline__ void tile_product(uint64_t (&acc)[4][2], const float* a, const float* b, int ty, int tx, int n = 64) {
#pragma unroll 8
  for (int k = 0; k < n; ++k) {
    const float4 x = *reinterpret_cast<const float4*>(a + k * CP + 4 * ty);
    const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(b + k * CP + 4 * tx);
    const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint64_t xx;
      asm("mov.b64 %0, {%1, %1};" : "=l"(xx) : "f"(xs[i]));
      asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][0]) : "l"(xx), "l"(y.x));
      asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][1]) : "l"(xx), "l"(y.y));
    }
  }
}
__device__ __forceinline__ float4 quad_of(const uint64_t (&v)[2]) {
  float4 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v[0]));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.z), "=f"(f.w) : "l"(v[1]));
  return f;
}
__device__ __forceinline__ void set_quad(uint64_t (&v)[2], float4 f) {
  asm("mov.b64 %0, {%1, %2};" : "=l"(v[0]) : "f"(f.x), "f"(f.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(v[1]) : "f"(f.z), "f"(f.w));
}
__device__ __forceinline__ float sum16(float v) {
#pragma unroll
  for (int o = 1; o < 16; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// CTAS an SM: one keeps the next chunk's loads and a product's operands in registers (212), where CTAs are more than SMs two are quicker
// with 128: 64 segments of 64 rows 147 us, one CTA an SM 179.  The arithmetic is the same.
template <int CTAS>
__global__ void __launch_bounds__(CT_THREADS, CTAS)
mlstm_chunk32_kernel(MlstmArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  float* qt = sm;                 // [d][t]
  float* kt = qt + TILE;          // [d][t]
  float* kw = kt + TILE;          // [t][d], times the token's weight in the state
  float* vs = kw + TILE;          // [t][v]
  float* pt = vs + TILE;          // [s][t]
  float* S = pt + TILE;           // [d][v]
  __shared__ double s_c[CL], s_M[CL];
  __shared__ float s_row[CL], s_floor[CL], s_w[CL], s_n[CD], s_nq[4][CL], s_np[4][CD], s_end[2];
  const int tid = threadIdx.x, lane = tid & 31, tx = tid & 15, ty = tid >> 4, tok = tid & 63, part = tid >> 6;
  const int h = blockIdx.x, sg = blockIdx.y;
  const int row0 = a.seg_row0[sg], rows = mlstm_chunked_rows(a.seg_rows[sg]), seq = a.seg_seq[sg];
  const bool fresh = a.seg_pos0[sg] == 0;
  if (seq < 0 || seq >= a.n_seqs) {
    if (tid == 0) arcb_set_error(a.err, ARCB_DEV_BAD_INDEX);
    return;
  }
  if (rows <= 0) return;
  float* Sg = a.S + ((size_t)seq * a.H + h) * a.dim * CD;
  float* ng = a.n + ((size_t)seq * a.H + h) * a.dimp;
  float* mg = a.m + (size_t)seq * a.H + h;
  for (int i = tid; i < CD * CD / 4; i += CT_THREADS) {
    const int d = i >> 4, c = (i & 15) * 4;
    *reinterpret_cast<float4*>(S + d * CP + c) = !fresh && d < a.dim ? *reinterpret_cast<const float4*>(Sg + (size_t)d * CD + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (tid < CD) s_n[tid] = !fresh && tid < a.dim ? ng[tid] : 0.f;
  double m = fresh ? 0. : (double)*mg;           // of warp 0

  // a thread's share of a chunk: 16 columns of one token of q, k and v
  float4 q[4], k[4], v[4];
  float gi[2], gf[2];
  auto fetch = [&](int t0) {
    const int t = t0 + tok;
    const size_t at = (size_t)(row0 + t) * a.pitch;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = part * 16 + i * 4;
      q[i] = k[i] = v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t < rows) {
        q[i] = ld_act4(a.proj, at + a.off_q + (size_t)h * a.dimp + c, a.fmt);
        k[i] = ld_act4(a.proj, at + a.off_k + (size_t)h * a.dimp + c, a.fmt);
        v[i] = ld_act4(a.proj, at + a.off_v + (size_t)h * CD + c, a.fmt);
        if (c + 3 >= a.dim) {
          float* const qf = reinterpret_cast<float*>(&q[i]);
          float* const kf = reinterpret_cast<float*>(&k[i]);
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (c + e >= a.dim) qf[e] = kf[e] = 0.f;
        }
      }
    }
    if (tid < 32)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int s = t0 + 2 * lane + u;
        gi[u] = s < rows ? a.gates[(size_t)(row0 + s) * 2 * a.H + h] : 0.f;
        gf[u] = s < rows ? a.gates[(size_t)(row0 + s) * 2 * a.H + a.H + h] : 0.f;
      }
  };
  fetch(0);
  const float inv_v = 1.f / (float)a.vdim;
  for (int t0 = 0; t0 < rows; t0 += CL) {
    const int nt = min(CL, rows - t0);
    if (tid < 32) {
      // lane: tokens 2 lane and 2 lane + 1; those behind the end add nothing
      const double lf0 = 2 * lane < nt ? (double)gate_log(gf[0], a.gate_cap, true) : 0., lf1 = 2 * lane + 1 < nt ? (double)gate_log(gf[1], a.gate_cap, true) : 0.;
      double sum = lf0 + lf1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += u;
      }
      double ahead = __shfl_up_sync(0xffffffffu, sum, 1);
      if (lane == 0) ahead = 0.;
      const double F1 = sum, F0 = ahead + lf0;   // not sum - lf1: nothing of a token reaches the one ahead of it
      const double none = -1e300;
      const double c0 = 2 * lane < nt ? (double)gate_log(gi[0], a.gate_cap, false) - F0 : none, c1 = 2 * lane + 1 < nt ? (double)gate_log(gi[1], a.gate_cap, false) - F1 : none;
      double top = fmax(c0, c1);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, top, o);
        if (lane >= o) top = fmax(top, u);
      }
      double before = __shfl_up_sync(0xffffffffu, top, 1);
      if (lane == 0) before = none;
      const double M0 = fmax(m, fmax(before, c0)), M1 = fmax(m, top);
      const double ML = __shfl_sync(0xffffffffu, M1, 31), FL = __shfl_sync(0xffffffffu, F1, 31);
      s_c[2 * lane] = c0; s_c[2 * lane + 1] = c1;
      s_M[2 * lane] = M0; s_M[2 * lane + 1] = M1;
      s_row[2 * lane] = expf((float)(m - M0)); s_row[2 * lane + 1] = expf((float)(m - M1));
      s_floor[2 * lane] = expf(-(float)(F0 + M0)); s_floor[2 * lane + 1] = expf(-(float)(F1 + M1));
      s_w[2 * lane] = expf((float)(c0 - ML)); s_w[2 * lane + 1] = expf((float)(c1 - ML));
      if (lane == 0) s_end[0] = expf((float)(m - ML));
      m = (double)(float)(FL + ML);              // as it is kept between calls
    }
    __syncthreads();
    {
      const float w = s_w[tok];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = part * 16 + i * 4;
        const float qf[4] = {q[i].x, q[i].y, q[i].z, q[i].w}, kf[4] = {k[i].x, k[i].y, k[i].z, k[i].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          qt[(c + e) * CP + tok] = qf[e];
          kt[(c + e) * CP + tok] = kf[e];
        }
        *reinterpret_cast<float4*>(kw + tok * CP + c) = make_float4(w * kf[0], w * kf[1], w * kf[2], w * kf[3]);
        *reinterpret_cast<float4*>(vs + tok * CP + c) = v[i];
      }
    }
    if (t0 + CL < rows) fetch(t0 + CL);
    __syncthreads();
    {
      float nq = 0.f;
#pragma unroll
      for (int d = 0; d < 16; ++d) nq = fmaf(s_n[part * 16 + d], qt[(part * 16 + d) * CP + tok], nq);
      s_nq[part][tok] = nq;
    }
    const bool live = (ty & ~1) * 4 < nt;        // the warp has rows
    // scores, weighted
    uint64_t acc[4][2] = {};
    float psum[4];
    if (live) {
      tile_product(acc, qt, kt, ty, tx);
      float p[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 f = quad_of(acc[i]);
        const float x[4] = {f.x, f.y, f.z, f.w};
        const double M = s_M[4 * ty + i];
        psum[i] = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          p[i][j] = 4 * tx + j <= 4 * ty + i ? x[j] * expf((float)(s_c[4 * tx + j] - M)) : 0.f;
          psum[i] += p[i][j];
        }
        psum[i] = sum16(psum[i]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(pt + (4 * tx + j) * CP + 4 * ty) = make_float4(p[0][j], p[1][j], p[2][j], p[3][j]);
    }
    __syncthreads();
    if (live) {
      // numerators: the carried state's part, then the chunk's
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0ull;
      tile_product(acc, qt, S, ty, tx);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float r = s_row[4 * ty + i];
        const float4 f = quad_of(acc[i]);
        set_quad(acc[i], make_float4(r * f.x, r * f.y, r * f.z, r * f.w));
      }
      // tokens ahead of the thread's four rows, then the rows' own, each up to itself: a later token's value may be anything, and zero
      // times that is not always zero
      tile_product(acc, pt, vs, ty, tx, 4 * ty);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 x = *reinterpret_cast<const float4*>(pt + (4 * ty + j) * CP + 4 * ty);
        const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(vs + (4 * ty + j) * CP + 4 * tx);
        const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int i = j; i < 4; ++i) {
          uint64_t xx;
          asm("mov.b64 %0, {%1, %1};" : "=l"(xx) : "f"(xs[i]));
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][0]) : "l"(xx), "l"(y.x));
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][1]) : "l"(xx), "l"(y.y));
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = 4 * ty + i;
        const float dot = fmaf(s_row[t], (s_nq[0][t] + s_nq[1][t]) + (s_nq[2][t] + s_nq[3][t]), psum[i]);
        const float den = fmaxf(fabsf(dot), s_floor[t]) + 1e-6f;
        float4 o = quad_of(acc[i]);
        o.x /= den; o.y /= den; o.z /= den; o.w /= den;
        const float ss = sum16((o.x * o.x + o.y * o.y) + (o.z * o.z + o.w * o.w));      // padding columns are exactly zero
        const float norm = 1.f / sqrtf(ss * inv_v + a.eps);
        if (t < nt) {
          const size_t row = row0 + t0 + t;
          const float4 g = ld_act4(a.proj, row * a.pitch + a.off_g + (size_t)h * CD + 4 * tx, a.fmt);
          const float4 w = __ldg(reinterpret_cast<const float4*>(a.norm_w + (size_t)h * CD + 4 * tx));
          st_act4(a.out, (row * a.H + h) * CD + 4 * tx, make_float4(o.x * norm * (w.x * g.x), o.y * norm * (w.y * g.y), o.z * norm * (w.z * g.z), o.w * norm * (w.w * g.w)), a.fmt);
        }
      }
    }
    // state: rows d = 4 ty + i
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0ull;
    tile_product(acc, kw, vs, ty, tx, (nt + 7) & ~7);      // the others are zeros
    {
      float n = 0.f;
#pragma unroll
      for (int s = 0; s < 16; ++s) n += kw[(part * 16 + s) * CP + tok];
      s_np[part][tok] = n;
    }
    const float keep = s_end[0];
    __syncthreads();                             // the old state and n are read
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float4* at = reinterpret_cast<float4*>(S + (4 * ty + i) * CP + 4 * tx);
      const float4 f = quad_of(acc[i]), old = *at;
      *at = make_float4(fmaf(keep, old.x, f.x), fmaf(keep, old.y, f.y), fmaf(keep, old.z, f.z), fmaf(keep, old.w, f.w));
    }
    if (tid < CD) s_n[tid] = fmaf(keep, s_n[tid], (s_np[0][tid] + s_np[1][tid]) + (s_np[2][tid] + s_np[3][tid]));
    __syncthreads();                             // also before the next chunk's gates and tiles
  }
  for (int i = tid; i < CD * CD / 4; i += CT_THREADS) {
    const int d = i >> 4, c = (i & 15) * 4;
    if (d < a.dim) *reinterpret_cast<float4*>(Sg + (size_t)d * CD + c) = *reinterpret_cast<const float4*>(S + d * CP + c);
  }
  if (tid < a.dim) ng[tid] = s_n[tid];
  if (tid == 0) *mg = (float)m;
}

}  // namespace

bool arcb_mlstm_chunk32_supported(int dimp, int vdimp, int fmt) { return dimp == CD && vdimp == CD && fmt == 2; }

int arcb_launch_mlstm_chunk32(const MlstmArgs& a, cudaStream_t stream) {
  if (a.n_segs <= 0) return 0;
  if (a.n_segs > 65535) return -1;
  if (a.n_rows > C32_ALONE) {                    // else no segment is long enough
    static std::atomic<unsigned long long> opted[2];
    const bool two = (long long)a.H * a.n_segs > arcb_num_sms();
    auto kernel = two ? mlstm_chunk32_kernel<2> : mlstm_chunk32_kernel<1>;
    cudaError_t e = arcb_opt_in_smem(kernel, C32_SMEM, opted[two]);
    if (e == cudaSuccess) e = arcb_launch(kernel, dim3(a.H, a.n_segs), dim3(CT_THREADS), C32_SMEM, stream, a);
    arcb_count_launch(1);
    if (e != cudaSuccess) return (int)e;
  }
  return arcb_launch_mlstm_rest64(a, stream);
}
