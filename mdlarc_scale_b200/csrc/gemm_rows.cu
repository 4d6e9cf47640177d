// y = A[M,K] * W[N,K]^T for few rows (decode steps of small batches), with the epilogues of epilogue.cuh.
//
// What bounds such a product is not arithmetic: its weights (0.1 to 20 MB) cross once, and the rest is fixed cost.  The
// tcgen05 kernels pay tensor-memory allocation, descriptor fetches, a TMA round trip per stage of one CTA's tile and an
// accumulator drain in a row, with 8 to 50 CTAs on 148 SMs: 10 to 12 us at 16 rows of 1024 to 1280 columns, whatever
// the size.  Here every CTA owns 16 or 32 output columns over the whole of K, so 64 to 350 CTAs pull weights at once:
//   * a warp takes every eighth block of 32 K values: a lane loads 16 consecutive bytes of a weight row and of an
//     activation row straight into registers, in the order that mma.m16n8k16 wants its fragments once K is permuted
//     the same way in both operands (weights are the 16-row operand, activations the 8-column one);
//   * the first blocks' weights are requested before the wait for the previous kernel (programmatic dependent launch):
//     they depend on nothing; what the epilogue needs besides the sums (old residual, biases, rotations) is requested
//     with the first activations, not behind the last sum;
//   * the eight warps' sums meet in shared memory, always in the same order, and leave through the epilogues' quads.
// B200, us a launch inside the captured step, tcgen05 tiles / here: 16 rows, QKV of width 1024 10.3 / 4.6, gate/up 10.6 / 5.4,
// out and down 10.7 / 3.9; 1 row of width 256 6.1 to 6.8 / 1.9 to 2.4; 1 row, mixer projection of width 1280 14.2 / 6.5.
// Steps of up to 32 rows, and of up to 64 in products with column groups (step_rules.cuh draws the line to gemm_mid.cu).
#include <atomic>

#include "common.cuh"
#include "gemm.cuh"
#include "gemm_rows.cuh"
#include "launch.cuh"
#include "ptx_sm100.cuh"
#include "step_rules.cuh"

namespace {

constexpr int GR_WARPS = 8;
constexpr int GR_THREADS = 32 * GR_WARPS;

template <int NT, int MT>
struct GrCfg {
  static constexpr int PITCH = 16 * NT + 4;          // floats: 8 x 4 consecutive accumulators fall on 32 banks
  static constexpr int ROWS = 8 * MT;
  // Blocks of K in flight a warp: weights in registers, activations in registers up to 16 rows and in shared memory beyond
  // (asynchronous copies; a lane reads back only its own bytes, so there is no barrier).  Two CTAs fit an SM in every form,
  // which makes products of up to 2 x 148 column tiles one wave.
  static constexpr bool RING = MT >= 4;
  static constexpr int WD = NT == 1 ? (MT <= 2 ? 6 : 3) : MT <= 4 ? 3 : 2;
  static constexpr int XD = RING ? (MT == 4 ? 4 : 3) : WD;
  static constexpr int RING_BYTES = RING ? GR_WARPS * XD * MT * 512 : 0;
  static constexpr int SUM_BYTES = GR_WARPS * ROWS * PITCH * 4;     // the sums take the ring's place
  static constexpr int SMEM = RING_BYTES > SUM_BYTES ? RING_BYTES : SUM_BYTES;
};

template <bool F16>
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (F16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// gate columns and the matching up columns, 64 further, are tiles of one CTA
template <int MODE>
__host__ __device__ constexpr bool gr_paired() { return MODE == EPI_SWIGLU || MODE == EPI_GLU; }

// first weight row of tile nt of column block `blk`
template <int NT, int MODE>
__device__ __forceinline__ int gr_col(int blk, int nt) {
  if constexpr (gr_paired<MODE>()) {
    constexpr int PER = 64 / (8 * NT);               // CTAs of one group of 64 gate columns
    return (blk / PER) * 128 + (blk % PER) * 8 * NT + (nt >> 1) * 16 + (nt & 1) * 64;
  }
  return (blk * NT + nt) * 16;
}

// A head's 64 or 128 columns lie in 4 or 8 CTAs of one cluster, which exchange their rows' sums of squares through shared
// memory; every thread of the cluster takes part.
template <int ROWS>
__device__ __forceinline__ float cluster_head_sum(float ss, int row, int q, bool wanted, int width, int in_head) {
  __shared__ float part[ROWS];
  ss += __shfl_xor_sync(0xffffffffu, ss, 1);
  ss += __shfl_xor_sync(0xffffffffu, ss, 2);
  if (q == 0 && row < ROWS) part[row] = ss;
  sm100::cluster_sync_all();
  float sum = 0.f;
  if (wanted) {
    const uint32_t first = sm100::cluster_ctarank() - (uint32_t)(in_head >> 4);
    for (int c = 0; c < width >> 4; ++c) sum += sm100::ld_shared_cluster_f32(sm100::smem_u32(part + row), first + c);
  }
  sm100::cluster_sync_all();                     // nobody leaves while its sums are read
  return sum;
}

template <int NT, int MT, int MODE, bool F16>
__device__ __forceinline__ void rows_product(const uint16_t* A, const uint16_t* W, const GemmEpilogue& ep, int K, float* red) {
  using Cfg = GrCfg<NT, MT>;
  constexpr int WD = Cfg::WD, XD = Cfg::XD, PITCH = Cfg::PITCH;
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = gr_col<NT, MODE>(blockIdx.x, 0), m0 = blockIdx.y * Cfg::ROWS;
  const int blocks = (K / 32 - warp + GR_WARPS - 1) / GR_WARPS;      // this warp's blocks of K
  const int step = GR_WARPS * 32;

  const uint16_t* wp[NT];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) wp[nt] = W + (size_t)(gr_col<NT, MODE>(blockIdx.x, nt) + g) * K + warp * 32 + t * 8;
  uint4 w[WD][NT][2];
  auto load_w = [&](int slot, int i) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      w[slot][nt][0] = ldg_stream16(wp[nt] + (size_t)i * step);
      w[slot][nt][1] = ldg_stream16(wp[nt] + (size_t)8 * K + (size_t)i * step);
    }
  };
#pragma unroll
  for (int p = 0; p < WD; ++p)
    if (p < blocks) load_w(p, p);
  pdl_wait();

  const size_t lda = ep.grp.lda ? ep.grp.lda : K;
  const uint16_t* xp = A + (size_t)(m0 + g) * lda + (ep.grp.n_group ? n0 / ep.grp.n_group * ep.grp.a_group : 0) + warp * 32 + t * 8;
  uint4 x[Cfg::RING ? 1 : XD][Cfg::RING ? 1 : MT];
  const uint32_t ring = sm100::smem_u32(red) + warp * XD * MT * 512 + lane * 16;
  auto load_x = [&](int slot, int i) {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const bool in = m0 + mt * 8 + g < ep.M;
      const uint16_t* src = xp + (size_t)(in ? mt * 8 : 0) * lda + (size_t)i * step;
      if constexpr (Cfg::RING)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ring + (slot * MT + mt) * 512), "l"(in ? src : A), "r"(in ? 16 : 0)
                     : "memory");
      else
        x[Cfg::RING ? 0 : slot][Cfg::RING ? 0 : mt] = in ? __ldcg(reinterpret_cast<const uint4*>(src)) : make_uint4(0u, 0u, 0u, 0u);
    }
  };
#pragma unroll
  for (int p = 0; p < XD; ++p) {
    if (p < blocks) load_x(p, p);
    if constexpr (Cfg::RING) asm volatile("cp.async.commit_group;" ::: "memory");
  }
  constexpr int QUADS = gr_paired<MODE>() ? 2 * NT : 4 * NT;         // output quads of a row
  QuadAhead ahead;
  if constexpr (MODE != EPI_HEADS && MT <= 4) {
    const int row = threadIdx.x / QUADS;
    if (row < Cfg::ROWS && m0 + row < ep.M) ahead.load<MODE>(ep, m0 + row, n0 + (threadIdx.x - row * QUADS) * 4);
  }

  float acc[NT][MT][4];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[nt][mt][j] = 0.f;

  int slot = 0;
  for (int i = 0; i < blocks; i += WD) {
#pragma unroll
    for (int p = 0; p < WD; ++p) {
      if (i + p >= blocks) break;
      if constexpr (Cfg::RING) {
        asm volatile("cp.async.wait_group %0;" ::"n"(XD - 1) : "memory");
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {        // one fragment at a time: registers are for sums and weights
          uint4 v;
          asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                       : "r"(ring + (slot * MT + mt) * 512)
                       : "memory");
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            const uint4 lo = w[p][nt][0], hi = w[p][nt][1];
            mma16816<F16>(acc[nt][mt], lo.x, hi.x, lo.y, hi.y, v.x, v.y);
            mma16816<F16>(acc[nt][mt], lo.z, hi.z, lo.w, hi.w, v.z, v.w);
          }
        }
      } else {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          const uint4 lo = w[p][nt][0], hi = w[p][nt][1];
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) mma16816<F16>(acc[nt][mt], lo.x, hi.x, lo.y, hi.y, x[p][mt].x, x[p][mt].y);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) mma16816<F16>(acc[nt][mt], lo.z, hi.z, lo.w, hi.w, x[p][mt].z, x[p][mt].w);
        }
      }
      if (i + p + WD < blocks) load_w(p, i + p + WD);
      if (i + p + XD < blocks) load_x(Cfg::RING ? slot : p, i + p + XD);
      if constexpr (Cfg::RING) {
        asm volatile("cp.async.commit_group;" ::: "memory");
        slot = slot + 1 == XD ? 0 : slot + 1;
      }
    }
  }
  if constexpr (Cfg::RING) __syncthreads();      // every warp is done with its part of the ring

  float* mine = red + warp * Cfg::ROWS * PITCH;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      float* r = mine + (mt * 8 + 2 * t) * PITCH + nt * 16 + g;
      r[0] = acc[nt][mt][0];
      r[PITCH] = acc[nt][mt][1];
      r[8] = acc[nt][mt][2];
      r[PITCH + 8] = acc[nt][mt][3];
    }
  __syncthreads();
  auto total = [&](int row, int c) {
    float4 v = *reinterpret_cast<const float4*>(red + row * PITCH + c);
#pragma unroll
    for (int k = 1; k < GR_WARPS; ++k) {
      const float4 o = *reinterpret_cast<const float4*>(red + (k * Cfg::ROWS + row) * PITCH + c);
      v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
    }
    return v;
  };
  if constexpr (MODE == EPI_HEADS) {
    static_assert(Cfg::ROWS * QUADS <= GR_THREADS, "one quad a thread");
    const int row = threadIdx.x / QUADS, q = threadIdx.x % QUADS;    // norms need NT = 1: quads of a row in neighbouring lanes of four
    const bool in = row < Cfg::ROWS && m0 + row < ep.M;
    epi_heads_quad(ep, in ? m0 + row : -1, n0 + q * 4, in ? total(row, q * 4) : make_float4(0.f, 0.f, 0.f, 0.f),
                   [&](float ss, bool wanted, int width, int in_head) { return cluster_head_sum<Cfg::ROWS>(ss, row, q, wanted, width, in_head); });
    return;
  }
  for (int u = threadIdx.x; u < Cfg::ROWS * QUADS; u += GR_THREADS) {
    const int row = u / QUADS, q = u - row * QUADS, m = m0 + row, n = n0 + q * 4;
    if (m >= ep.M) break;
    if (MT > 4 || u != threadIdx.x) ahead.load<MODE>(ep, m, n);
    if constexpr (gr_paired<MODE>()) {
      const int c = (q >> 2) * 32 + (q & 3) * 4;                     // gate tile 2 (q / 4), its up tile 16 columns on
      const float4 gate = total(row, c), up = total(row, c + 16);
      if constexpr (MODE == EPI_SWIGLU) epi_swiglu_quad(ep, m, n, gate, up, ahead.a, ahead.b);
      else epi_glu_quad(ep, m, n, gate, up);
    } else {
      const float4 v = total(row, q * 4);
      if constexpr (MODE == EPI_QKV_ROPE)
        epi_qkv_quad(ep, ahead.rr, m, n, v, make_float2(ahead.a.x, ahead.a.y), make_float2(ahead.a.z, ahead.a.w));
      else if constexpr (MODE == EPI_RESID) epi_resid_quad(ep, m, n, v, ahead.a, ahead.b);
      else if constexpr (MODE == EPI_RELU2) epi_relu2_quad(ep, m, n, v);
      else if constexpr (MODE == EPI_ACT) epi_act_quad(ep, m, n, v);
      else epi_store_quad(ep, m, n, v);
    }
  }
}

template <int NT, int MT, int MODE, bool F16>
__global__ void __launch_bounds__(GR_THREADS, 2)
gemm_rows_kernel(const uint16_t* A, const uint16_t* W, GemmEpilogue ep, int K) {
  extern __shared__ __align__(16) float red[];     // float4 and 16-byte asynchronous copies
  rows_product<NT, MT, MODE, F16>(A, W, ep, K, red);
}

// clusters of the CTAs that share 128 columns
template <int MT, bool F16>
__global__ void __cluster_dims__(8, 1, 1) __launch_bounds__(GR_THREADS, 2)
gemm_rows_heads_kernel(const uint16_t* A, const uint16_t* W, GemmEpilogue ep, int K) {
  extern __shared__ __align__(16) float red[];     // float4 and 16-byte asynchronous copies
  rows_product<1, MT, EPI_HEADS, F16>(A, W, ep, K, red);
}

template <int NT, int MT, int MODE>
cudaError_t launch(const void* a, const void* w, const GemmEpilogue& ep, int K, int act_f16, cudaStream_t stream) {
  using Cfg = GrCfg<NT, MT>;
  const dim3 grid(ep.N / (16 * NT), (ep.M + Cfg::ROWS - 1) / Cfg::ROWS);
  auto kernel = act_f16 ? gemm_rows_kernel<NT, MT, MODE, true> : gemm_rows_kernel<NT, MT, MODE, false>;
  static std::atomic<unsigned long long> opted[2];
  const cudaError_t e = arcb_opt_in_smem(kernel, Cfg::SMEM, opted[act_f16 ? 1 : 0]);
  if (e != cudaSuccess) return e;
  return arcb_launch(kernel, grid, dim3(GR_THREADS), Cfg::SMEM, stream, reinterpret_cast<const uint16_t*>(a),
                     reinterpret_cast<const uint16_t*>(w), ep, K);
}

bool wide_columns(const GemmEpilogue& ep) { return rows_wide_columns(ep.M, ep.N, arcb_num_sms()); }

template <int MT>
cudaError_t launch_heads(const void* a, const void* w, const GemmEpilogue& ep, int K, int act_f16, cudaStream_t stream) {
  using Cfg = GrCfg<1, MT>;
  auto kernel = act_f16 ? gemm_rows_heads_kernel<MT, true> : gemm_rows_heads_kernel<MT, false>;
  static std::atomic<unsigned long long> opted[2];
  const cudaError_t e = arcb_opt_in_smem(kernel, Cfg::SMEM, opted[act_f16 ? 1 : 0]);
  if (e != cudaSuccess) return e;
  return arcb_launch(kernel, dim3(ep.N / 16, (ep.M + Cfg::ROWS - 1) / Cfg::ROWS), dim3(GR_THREADS), Cfg::SMEM, stream,
                     reinterpret_cast<const uint16_t*>(a), reinterpret_cast<const uint16_t*>(w), ep, K);
}

template <int MODE>
cudaError_t launch_mode(const void* a, const void* w, const GemmEpilogue& ep, int K, int act_f16, cudaStream_t stream) {
  constexpr int N1 = gr_paired<MODE>() ? 2 : 1;
  if (N1 == 1 && wide_columns(ep)) return ep.M <= 8 ? launch<2, 1, MODE>(a, w, ep, K, act_f16, stream) : launch<2, 2, MODE>(a, w, ep, K, act_f16, stream);
  if (ep.M <= 8) return launch<N1, 1, MODE>(a, w, ep, K, act_f16, stream);
  if (ep.M <= 16) return launch<N1, 2, MODE>(a, w, ep, K, act_f16, stream);
  if constexpr (MODE == EPI_ACT)
    if (ep.M > 32) return launch<2, 8, MODE>(a, w, ep, K, act_f16, stream);
  return launch<2, 4, MODE>(a, w, ep, K, act_f16, stream);
}

}  // namespace

// Steps only: K is added in other parts than in the tcgen05 tiles of more rows, and a prompt row's result does not depend on what else
// its call holds (48 rows of width 1280, gated units: 10.5 us here, 12.7 there).
// With column groups, which the transposed tiles do not take, up to 64 rows: the weights' 16-row fragments meet eight 8-row
// activation fragments, and the activations of a CTA (64 rows x K) are re-read from L2 by every CTA.  One row tile more would read
// the weights twice.
bool arcb_gemm_rows_applies(const void* a, const void* w, const GemmEpilogue& ep, int K, int act_f16) {
  if (!ep.step || ep.M > (ep.grp.n_group ? 64 : 32) || act_f16 == 2 || K % 64 || ep.N % 128) return false;   // other K: the CUDA-core kernels, as beyond 64 rows
  const GroupArgs& g = ep.grp;
  if (g.tile_src || g.tile_group || g.n_tiles || g.panels || (g.n_group && g.n_group % 32) || g.lda % 8 || g.a_group % 8) return false;
  // 16-byte accesses; what is not aligned meets the tensor maps' refusal
  const uintptr_t all = (uintptr_t)a | (uintptr_t)w | (uintptr_t)ep.x | (uintptr_t)ep.y | (uintptr_t)ep.out16 | (uintptr_t)ep.bias | (uintptr_t)ep.pj.out;
  if (all & 15) return false;
  // normed heads span CTAs of one cluster of 128 columns
  return ep.mode != EPI_HEADS || !(ep.pj.q_norm || ep.pj.k_norm) || ep.pj.dimp <= 128;
}

int arcb_launch_gemm_rows(const void* a, const void* w, const GemmEpilogue& ep, int K, int act_f16, cudaStream_t stream) {
  cudaError_t e = cudaErrorInvalidValue;
  switch (ep.mode) {
    case EPI_STORE_F32: e = launch_mode<EPI_STORE_F32>(a, w, ep, K, act_f16, stream); break;
    case EPI_QKV_ROPE: e = launch_mode<EPI_QKV_ROPE>(a, w, ep, K, act_f16, stream); break;
    case EPI_RESID: e = launch_mode<EPI_RESID>(a, w, ep, K, act_f16, stream); break;
    case EPI_SWIGLU: e = launch_mode<EPI_SWIGLU>(a, w, ep, K, act_f16, stream); break;
    case EPI_RELU2: e = launch_mode<EPI_RELU2>(a, w, ep, K, act_f16, stream); break;
    case EPI_ACT: e = launch_mode<EPI_ACT>(a, w, ep, K, act_f16, stream); break;
    case EPI_GLU: e = launch_mode<EPI_GLU>(a, w, ep, K, act_f16, stream); break;
    case EPI_HEADS:
      if (!ep.pj.q_norm && !ep.pj.k_norm && wide_columns(ep)) {
        e = ep.M <= 8 ? launch<2, 1, EPI_HEADS>(a, w, ep, K, act_f16, stream) : launch<2, 2, EPI_HEADS>(a, w, ep, K, act_f16, stream);
        break;
      }
      e = ep.M <= 8    ? launch_heads<1>(a, w, ep, K, act_f16, stream)
          : ep.M <= 16 ? launch_heads<2>(a, w, ep, K, act_f16, stream)
                       : launch_heads<4>(a, w, ep, K, act_f16, stream);
      break;
  }
  arcb_count_launch(1);
  return (int)e;
}
