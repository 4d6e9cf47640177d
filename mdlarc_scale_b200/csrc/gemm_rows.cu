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
//     they depend on nothing;
//   * the eight warps' sums meet in shared memory, always in the same order, and leave through the epilogues' quads.
#include "common.cuh"
#include "gemm.cuh"
#include "gemm_rows.cuh"
#include "launch.cuh"

namespace {

constexpr int GR_WARPS = 8;
constexpr int GR_THREADS = 32 * GR_WARPS;

template <int NT, int MT>
struct GrCfg {
  static constexpr int PITCH = 16 * NT + 4;          // floats: 8 x 4 consecutive accumulators fall on 32 banks
  static constexpr int ROWS = 8 * MT;
  static constexpr int SMEM = GR_WARPS * ROWS * PITCH * 4;
  static constexpr int WD = NT == 1 ? 6 : NT == 2 ? 4 : 2;   // weight blocks in flight a warp
  static constexpr int XD = MT <= 2 ? WD : MT == 4 ? 2 : 1;  // activation blocks in flight; divides WD
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

template <int NT, int MT, int MODE, bool F16>
__global__ void __launch_bounds__(GR_THREADS)
gemm_rows_kernel(const uint16_t* A, const uint16_t* W, GemmEpilogue ep, int K) {
  using Cfg = GrCfg<NT, MT>;
  constexpr int WD = Cfg::WD, XD = Cfg::XD, PITCH = Cfg::PITCH;
  pdl_launch_dependents();
  extern __shared__ float red[];
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
  uint4 x[XD][MT];
  auto load_x = [&](int slot, int i) {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
      x[slot][mt] = m0 + mt * 8 + g < ep.M ? __ldcg(reinterpret_cast<const uint4*>(xp + (size_t)mt * 8 * lda + (size_t)i * step))
                                           : make_uint4(0u, 0u, 0u, 0u);
  };
#pragma unroll
  for (int p = 0; p < XD; ++p)
    if (p < blocks) load_x(p, p);

  float acc[NT][MT][4];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[nt][mt][j] = 0.f;

  for (int i = 0; i < blocks; i += WD) {
#pragma unroll
    for (int p = 0; p < WD; ++p) {
      if (i + p >= blocks) break;
      const int s = p % XD;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const uint4 lo = w[p][nt][0], hi = w[p][nt][1];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) mma16816<F16>(acc[nt][mt], lo.x, hi.x, lo.y, hi.y, x[s][mt].x, x[s][mt].y);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) mma16816<F16>(acc[nt][mt], lo.z, hi.z, lo.w, hi.w, x[s][mt].z, x[s][mt].w);
      }
      if (i + p + WD < blocks) load_w(p, i + p + WD);
      if (i + p + XD < blocks) load_x(s, i + p + XD);
    }
  }

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
  constexpr int QUADS = gr_paired<MODE>() ? 2 * NT : 4 * NT;         // output quads of a row
  for (int u = threadIdx.x; u < Cfg::ROWS * QUADS; u += GR_THREADS) {
    const int row = u / QUADS, q = u - row * QUADS, m = m0 + row;
    if (m >= ep.M) break;
    if constexpr (gr_paired<MODE>()) {
      const int c = (q >> 2) * 32 + (q & 3) * 4;                     // gate tile 2 (q / 4), its up tile 16 columns on
      const float4 gate = total(row, c), up = total(row, c + 16);
      const int n = n0 + q * 4;
      if constexpr (MODE == EPI_SWIGLU) epi_swiglu_quad(ep, m, n, gate, up);
      else epi_glu_quad(ep, m, n, gate, up);
    } else {
      const float4 v = total(row, q * 4);
      const int n = n0 + q * 4;
      if constexpr (MODE == EPI_QKV_ROPE) epi_qkv_quad(ep, rope_row_ctx(ep, m), m, n, v);
      else if constexpr (MODE == EPI_RESID) epi_resid_quad(ep, m, n, v);
      else if constexpr (MODE == EPI_RELU2) epi_relu2_quad(ep, m, n, v);
      else if constexpr (MODE == EPI_ACT) epi_act_quad(ep, m, n, v);
      else epi_store_quad(ep, m, n, v);
    }
  }
}

template <int NT, int MT, int MODE>
cudaError_t launch(const void* a, const void* w, const GemmEpilogue& ep, int K, int act_f16, cudaStream_t stream) {
  using Cfg = GrCfg<NT, MT>;
  const dim3 grid(ep.N / (16 * NT), (ep.M + Cfg::ROWS - 1) / Cfg::ROWS);
  auto kernel = act_f16 ? gemm_rows_kernel<NT, MT, MODE, true> : gemm_rows_kernel<NT, MT, MODE, false>;
  return arcb_launch(kernel, grid, dim3(GR_THREADS), Cfg::SMEM, stream, reinterpret_cast<const uint16_t*>(a),
                     reinterpret_cast<const uint16_t*>(w), ep, K);
}

template <int MODE>
cudaError_t launch_mode(const void* a, const void* w, const GemmEpilogue& ep, int K, int act_f16, cudaStream_t stream) {
  constexpr int N1 = gr_paired<MODE>() ? 2 : 1;
  if (ep.M <= 8) return launch<N1, 1, MODE>(a, w, ep, K, act_f16, stream);
  if (ep.M <= 16) return launch<N1, 2, MODE>(a, w, ep, K, act_f16, stream);
  if (ep.M <= 32) return launch<2, 4, MODE>(a, w, ep, K, act_f16, stream);
  return launch<2, 8, MODE>(a, w, ep, K, act_f16, stream);
}

// the widest form's partial sums need more than the default 48 KB of shared memory
template <int MODE>
cudaError_t init_mode() {
  const int bytes = GrCfg<2, 8>::SMEM;
  const cudaError_t e = cudaFuncSetAttribute(gemm_rows_kernel<2, 8, MODE, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(gemm_rows_kernel<2, 8, MODE, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

}  // namespace

int arcb_gemm_rows_init() {
  cudaError_t e;
  if ((e = init_mode<EPI_STORE_F32>()) != cudaSuccess) return (int)e;
  if ((e = init_mode<EPI_QKV_ROPE>()) != cudaSuccess) return (int)e;
  if ((e = init_mode<EPI_RESID>()) != cudaSuccess) return (int)e;
  if ((e = init_mode<EPI_SWIGLU>()) != cudaSuccess) return (int)e;
  if ((e = init_mode<EPI_RELU2>()) != cudaSuccess) return (int)e;
  if ((e = init_mode<EPI_ACT>()) != cudaSuccess) return (int)e;
  return (int)init_mode<EPI_GLU>();
}

// Up to 64 rows: the weights' 16-row fragments meet eight 8-row activation fragments, and the activations of a CTA
// (64 rows x K) are re-read from L2 by every CTA; the step of the latent-attention model with 48 rows takes 3 % less
// with it.  One row tile more would read the weights twice.
bool arcb_gemm_rows_applies(const GemmEpilogue& ep, int K, int act_f16) {
  if (ep.M > 64 || act_f16 == 2 || K % 32 || ep.N % 128) return false;
  const GroupArgs& g = ep.grp;
  if (g.tile_src || g.tile_group || g.n_tiles || g.panels || (g.n_group && g.n_group % 32)) return false;
  return ep.mode != EPI_HEADS;
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
  }
  arcb_count_launch(1);
  return (int)e;
}
