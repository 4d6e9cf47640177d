// Row-wise kernels (float4 accesses; one warp per row, bound by HBM, or in steps of few rows one CTA per row, bound by latency):
//   embed_norm    : token + example embedding -> residual stream, fused first RMSNorm
//   rmsnorm       : RMSNorm of the residual stream -> 16-bit GEMM operand
//   decode_begin  : grid-state position update + embedding + first RMSNorm of a decode step
//   head          : final RMSNorm -> 14 logits -> argmax (+ greedy-loop bookkeeping)
//   pack_rows     : fp32 -> bf16-rounded weights in kernel layout
#include "rowops.cuh"
#include "greedy_loop.cuh"
#include "launch.cuh"

namespace {

constexpr int ROWS_PER_CTA = 4;

// One CTA per row instead of one warp in steps: launches of at most this many rows leave most of the machine idle
// otherwise, and a row's time is then one warp's chain of loads and shuffles (1280 columns: 40 floats a lane).
// B200, us per launch inside the captured step, warp / CTA per row: norm of 6 rows of 1280 columns 4.8 / 1.8, of 128 rows
// of 1024 3.8 / 1.8; head of 16 rows of 1024 21.5 / 4.0, step begin 9.1 / 2.9.  2048 CTAs of 128 threads are one wave (the
// head's of 256 threads two); above that the warp form reads at the HBM rate.  The two add in different orders, so a prompt's
// rows, whose results do not depend on what else their call holds, always have a warp each.
constexpr int CTA_ROW_MAX = 2048;
constexpr int CTA_THREADS = 128;
constexpr int CTA_MAX_D = CTA_THREADS * 4 * 4;   // columns a CTA holds in registers

// sum of squares of a row held in global memory, warp-cooperative
__device__ __forceinline__ float row_sumsq(const float* __restrict__ x, int d, int lane) {
  float ss = 0.f;
  for (int i = lane * 4; i < d; i += 128) {
    const float4 v = *reinterpret_cast<const float4*>(x + i);
    ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
  }
  return warp_sum(ss);
}

// out16 = (x * rsqrt(mean(x^2) + eps)) * w    (src/transformer.py:45-48)
// Rows of up to 128 * NV floats are held in registers: every load of the row is in flight at once
// and the row is read from memory once.  The sum of squares is accumulated in the same order as
// row_sumsq, so both forms give the same bits.
template <int NV>
__device__ __forceinline__ void row_norm_store_regs(const float* __restrict__ x, const float* __restrict__ w,
                                                    uint16_t* __restrict__ out, int d, float eps, int act_f16,
                                                    int lane) {
  float4 v[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = lane * 4 + k * 128;
    v[k] = (i < d) ? *reinterpret_cast<const float4*>(x + i) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < NV; ++k)
    if (lane * 4 + k * 128 < d) ss += v[k].x * v[k].x + v[k].y * v[k].y + v[k].z * v[k].z + v[k].w * v[k].w;
  ss = warp_sum(ss);
  const float inv = rsqrtf(ss / (float)d + eps);
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = lane * 4 + k * 128;
    if (i < d) {
      const float4 g = __ldg(reinterpret_cast<const float4*>(w + i));
      uint2 pk;
      pk.x = pack2_act((v[k].x * inv) * g.x, (v[k].y * inv) * g.y, act_f16);
      pk.y = pack2_act((v[k].z * inv) * g.z, (v[k].w * inv) * g.w, act_f16);
      *reinterpret_cast<uint2*>(out + i) = pk;
    }
  }
}

__device__ __forceinline__ void row_norm_store(const float* __restrict__ x, const float* __restrict__ w,
                                               uint16_t* __restrict__ out, int d, float eps, int act_f16,
                                               int lane) {
  if (d <= 128 * 2) return row_norm_store_regs<2>(x, w, out, d, eps, act_f16, lane);
  if (d <= 128 * 6) return row_norm_store_regs<6>(x, w, out, d, eps, act_f16, lane);
  if (d <= 128 * 10) return row_norm_store_regs<10>(x, w, out, d, eps, act_f16, lane);
  if (d <= 128 * 16) return row_norm_store_regs<16>(x, w, out, d, eps, act_f16, lane);
  const float ss = row_sumsq(x, d, lane);
  const float inv = rsqrtf(ss / (float)d + eps);
  for (int i = lane * 4; i < d; i += 128) {
    const float4 v = *reinterpret_cast<const float4*>(x + i);
    const float4 g = __ldg(reinterpret_cast<const float4*>(w + i));
    uint2 pk;
    pk.x = pack2_act((v.x * inv) * g.x, (v.y * inv) * g.y, act_f16);
    pk.y = pack2_act((v.z * inv) * g.z, (v.w * inv) * g.w, act_f16);
    *reinterpret_cast<uint2*>(out + i) = pk;
  }
}

// Embedding row into registers (a CTA's share of it), and into the residual stream.
template <int NV>
__device__ __forceinline__ void cta_embed(float4 (&v)[NV], float* x, const float* tok_row, const float* ex_row, int d) {
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = (threadIdx.x + k * CTA_THREADS) * 4;
    v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < d) {
      v[k] = __ldg(reinterpret_cast<const float4*>(tok_row + i));
      if (ex_row) {
        const float4 e = __ldg(reinterpret_cast<const float4*>(ex_row + i));
        v[k].x += e.x; v[k].y += e.y; v[k].z += e.z; v[k].w += e.w;
      }
      *reinterpret_cast<float4*>(x + i) = v[k];
    }
  }
}

__device__ __forceinline__ void row_embed(float* __restrict__ x, const float* __restrict__ tok_row,
                                          const float* __restrict__ ex_row, int d, int lane) {
  for (int i = lane * 4; i < d; i += 128) {
    float4 v = __ldg(reinterpret_cast<const float4*>(tok_row + i));
    if (ex_row) {
      const float4 e = __ldg(reinterpret_cast<const float4*>(ex_row + i));
      v.x += e.x; v.y += e.y; v.z += e.z; v.w += e.w;
    }
    *reinterpret_cast<float4*>(x + i) = v;
  }
  __syncwarp();
}

// Sum over the CTA's four warps, in a fixed order; every thread gets it.
__device__ __forceinline__ float cta_sum4(float v, float* sm) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  return (sm[0] + sm[1]) + (sm[2] + sm[3]);
}

// The row's columns tid * 4 + k * 512 in v (zeros beyond d): norm, gain, 16-bit operand.
template <int NV>
__device__ __forceinline__ void cta_norm_store(const float4 (&v)[NV], const float* w, uint16_t* out, int d, float eps,
                                               int act_f16, float* sm) {
  float4 g[NV];
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = (threadIdx.x + k * CTA_THREADS) * 4;
    g[k] = i < d ? __ldg(reinterpret_cast<const float4*>(w + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
    ss += (v[k].x * v[k].x + v[k].y * v[k].y) + (v[k].z * v[k].z + v[k].w * v[k].w);
  }
  const float inv = rsqrtf(cta_sum4(ss, sm) / (float)d + eps);
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = (threadIdx.x + k * CTA_THREADS) * 4;
    if (i < d) {
      uint2 pk;
      pk.x = pack2_act((v[k].x * inv) * g[k].x, (v[k].y * inv) * g[k].y, act_f16);
      pk.y = pack2_act((v[k].z * inv) * g[k].z, (v[k].w * inv) * g[k].w, act_f16);
      *reinterpret_cast<uint2*>(out + i) = pk;
    }
  }
}

template <int NV>
__global__ void __launch_bounds__(CTA_THREADS)
rmsnorm_cta_kernel(const float* x, const float* w, uint16_t* out, int d, float eps, int act_f16) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float sm[4];
  const float* row = x + (size_t)blockIdx.x * d;
  float4 v[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = (threadIdx.x + k * CTA_THREADS) * 4;
    v[k] = i < d ? __ldcg(reinterpret_cast<const float4*>(row + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  cta_norm_store<NV>(v, w, out + (size_t)blockIdx.x * d, d, eps, act_f16, sm);
}

__global__ void __launch_bounds__(ROWS_PER_CTA * 32)
rmsnorm_kernel(const float* __restrict__ x, const float* __restrict__ w, uint16_t* __restrict__ out,
               int rows, int d, float eps, int act_f16) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x * ROWS_PER_CTA + (threadIdx.x >> 5);
  if (row >= rows) return;
  row_norm_store(x + (size_t)row * d, w, out + (size_t)row * d, d, eps, act_f16, threadIdx.x & 31);
}

__global__ void __launch_bounds__(ROWS_PER_CTA * 32)
embed_norm_kernel(EmbedArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x * ROWS_PER_CTA + (threadIdx.x >> 5);
  if (row >= a.rows) return;
  const int lane = threadIdx.x & 31;
  int tok = a.token_ids[row];
  tok = min(max(tok, 0), a.vocab - 1);
  const float* ex_row = nullptr;
  if (a.example_ids) {
    int ex = a.example_ids[a.seq ? a.seq[row] : row];
    ex = min(max(ex, 0), a.num_examples - 1);
    ex_row = a.example_embed + (size_t)ex * a.d;
  }
  float* x = a.x + (size_t)row * a.d;
  row_embed(x, a.token_embed + (size_t)tok * a.d, ex_row, a.d, lane);
  row_norm_store(x, a.ln_w, a.xn16 + (size_t)row * a.d, a.d, a.eps, a.act_f16, lane);
}

// Grid state, then the embedding of the fed token and the first RMSNorm of the step; one warp or one CTA per sequence.
__global__ void __launch_bounds__(ROWS_PER_CTA * 32)
decode_begin_kernel(DecodeState st, EmbedArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.x * ROWS_PER_CTA + (threadIdx.x >> 5);
  if (b >= st.n_seqs) return;
  const int lane = threadIdx.x & 31;
  const int tok = st.cur_tok[b];
  if (lane == 0) grid_step(st, b, tok);
  const int tk = min(max(tok, 0), a.vocab - 1);
  float* x = a.x + (size_t)b * a.d;
  row_embed(x, a.token_embed + (size_t)tk * a.d, example_row(a, b), a.d, lane);
  row_norm_store(x, a.ln_w, a.xn16 + (size_t)b * a.d, a.d, a.eps, a.act_f16, lane);
}

template <int NV>
__global__ void __launch_bounds__(CTA_THREADS)
decode_begin_cta_kernel(DecodeState st, EmbedArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float sm[4];
  const int b = blockIdx.x;
  const int tok = st.cur_tok[b];
  const int tk = min(max(tok, 0), a.vocab - 1);
  float4 v[NV];
  cta_embed<NV>(v, a.x + (size_t)b * a.d, a.token_embed + (size_t)tk * a.d, example_row(a, b), a.d);
  if (threadIdx.x == CTA_THREADS - 1) grid_step(st, b, tok);   // a thread with the fewest columns
  cta_norm_store<NV>(v, a.ln_w, a.xn16 + (size_t)b * a.d, a.d, a.eps, a.act_f16, sm);
}

__global__ void __launch_bounds__(ROWS_PER_CTA * 32)
head_kernel(HeadArgs a, DecodeState st) {
  pdl_launch_dependents();
  pdl_wait();
  const int i = blockIdx.x * ROWS_PER_CTA + (threadIdx.x >> 5);
  if (i >= a.rows) return;
  const int lane = threadIdx.x & 31;
  const int row = a.row_index ? a.row_index[i] : i;
  const float* x = a.x + (size_t)row * a.d;
  const float ss = row_sumsq(x, a.d, lane);
  const float inv = rsqrtf(ss / (float)a.d + a.eps);
  float acc[ARCB_VOCAB];
#pragma unroll
  for (int v = 0; v < ARCB_VOCAB; ++v) acc[v] = 0.f;
  for (int c = lane * 4; c < a.d; c += 128) {
    const float4 xv = *reinterpret_cast<const float4*>(x + c);
    const float4 g = __ldg(reinterpret_cast<const float4*>(a.lnf_w + c));
    const float n0 = (xv.x * inv) * g.x, n1 = (xv.y * inv) * g.y, n2 = (xv.z * inv) * g.z,
                n3 = (xv.w * inv) * g.w;
#pragma unroll
    for (int v = 0; v < ARCB_VOCAB; ++v) {
      const float4 w = __ldg(reinterpret_cast<const float4*>(a.lm_head + (size_t)v * a.d + c));
      acc[v] += n0 * w.x + n1 * w.y + n2 * w.z + n3 * w.w;
    }
  }
#pragma unroll
  for (int v = 0; v < ARCB_VOCAB; ++v) acc[v] = warp_sum(acc[v]);
  if (lane == 0) head_finish(a, st, i, acc);
}

// One CTA of eight warps per row: NV float4 of the row a thread, the 14 sums met in shared memory.
constexpr int HEAD_THREADS = 256;
template <int NV>
__global__ void __launch_bounds__(HEAD_THREADS)
head_cta_kernel(HeadArgs a, DecodeState st) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float sm[HEAD_THREADS / 32][16];
  const int i = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const float* x = a.x + (size_t)(a.row_index ? a.row_index[i] : i) * a.d;
  // the norm's factor is the same for all columns: it multiplies the finished sums
  float part[15];
#pragma unroll
  for (int v = 0; v < 15; ++v) part[v] = 0.f;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int c = (tid + k * HEAD_THREADS) * 4;
    if (c < a.d) {
      const float4 xv = __ldcg(reinterpret_cast<const float4*>(x + c));
      const float4 g = __ldg(reinterpret_cast<const float4*>(a.lnf_w + c));
      part[14] += (xv.x * xv.x + xv.y * xv.y) + (xv.z * xv.z + xv.w * xv.w);
      const float4 n = make_float4(xv.x * g.x, xv.y * g.y, xv.z * g.z, xv.w * g.w);
#pragma unroll
      for (int v = 0; v < ARCB_VOCAB; ++v) {
        const float4 w = __ldg(reinterpret_cast<const float4*>(a.lm_head + (size_t)v * a.d + c));
        part[v] += (n.x * w.x + n.y * w.y) + (n.z * w.z + n.w * w.w);
      }
    }
  }
#pragma unroll
  for (int v = 0; v < 15; ++v) {
    const float s = warp_sum(part[v]);
    if (lane == 0) sm[warp][v] = s;
  }
  __syncthreads();
  if (warp != 0) return;
  float s = 0.f;
  if (lane < 15) {
#pragma unroll
    for (int w = 0; w < HEAD_THREADS / 32; ++w) s += sm[w][lane];
  }
  const float inv = rsqrtf(__shfl_sync(0xffffffffu, s, 14) / (float)a.d + a.eps);
  s *= inv;
  float acc[ARCB_VOCAB];
#pragma unroll
  for (int v = 0; v < ARCB_VOCAB; ++v) acc[v] = __shfl_sync(0xffffffffu, s, v);
  if (lane == 0) head_finish(a, st, i, acc);
}

// dst row = (r / blk) * blk_stride + blk_off + r % blk.  Every value is first rounded to bf16 (the
// model's precision); container: 0 = fp32, 1 = bf16, 2 = IEEE half holding the bf16-rounded value
// (exact for |w| >= 2^-14, within 2^-25 absolute below; saturates at +-65504).
__global__ void pack_rows_kernel(const float* __restrict__ src, void* __restrict__ dst, long long rows,
                                 long long cols, int blk, int blk_stride, int blk_off, int to_bf16) {
  const long long n = rows * cols;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / cols, c = i - r * cols;
    const long long dr = (r / blk) * blk_stride + blk_off + (r % blk);
    const __nv_bfloat16 h = __float2bfloat16_rn(src[i]);
    if (to_bf16 == 1) {
      reinterpret_cast<__nv_bfloat16*>(dst)[dr * cols + c] = h;
    } else if (to_bf16 == 2) {
      const float f = fminf(fmaxf(__bfloat162float(h), -65504.f), 65504.f);
      reinterpret_cast<__half*>(dst)[dr * cols + c] = __float2half_rn(f);
    } else {
      reinterpret_cast<float*>(dst)[dr * cols + c] = __bfloat162float(h);
    }
  }
}

}  // namespace

static bool cta_per_row(bool step, int rows, int d) { return step && rows <= CTA_ROW_MAX && d <= CTA_MAX_D; }

int arcb_launch_rmsnorm(const float* x, const float* w, void* out16, int rows, int d, float eps,
                        int act_f16, bool step, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (d % 4) return -1;
  uint16_t* out = reinterpret_cast<uint16_t*>(out16);
  auto cta = [&](auto kernel) { return arcb_launch(kernel, dim3(rows), dim3(CTA_THREADS), 0, stream, x, w, out, d, eps, act_f16); };
  const cudaError_t e = !cta_per_row(step, rows, d) ? arcb_launch(rmsnorm_kernel, dim3((rows + ROWS_PER_CTA - 1) / ROWS_PER_CTA),
                                                            dim3(ROWS_PER_CTA * 32), 0, stream, x, w, out, rows, d, eps, act_f16)
                        : d <= CTA_THREADS * 4 ? cta(rmsnorm_cta_kernel<1>)
                        : d <= CTA_THREADS * 8 ? cta(rmsnorm_cta_kernel<2>)
                                               : cta(rmsnorm_cta_kernel<4>);
  arcb_count_launch(1);
  return (int)e;
}

int arcb_launch_embed_norm(const EmbedArgs& a, cudaStream_t stream) {
  if (a.rows <= 0) return 0;
  const cudaError_t e = arcb_launch(embed_norm_kernel, dim3((a.rows + ROWS_PER_CTA - 1) / ROWS_PER_CTA),
                                    dim3(ROWS_PER_CTA * 32), 0, stream, a);
  arcb_count_launch(1);
  return (int)e;
}

int arcb_launch_decode_begin(const DecodeState& st, const EmbedArgs& a, cudaStream_t stream) {
  auto cta = [&](auto kernel) { return arcb_launch(kernel, dim3(st.n_seqs), dim3(CTA_THREADS), 0, stream, st, a); };
  const cudaError_t e = !cta_per_row(true, st.n_seqs, a.d) ? arcb_launch(decode_begin_kernel, dim3((st.n_seqs + ROWS_PER_CTA - 1) / ROWS_PER_CTA),
                                                                   dim3(ROWS_PER_CTA * 32), 0, stream, st, a)
                        : a.d <= CTA_THREADS * 4 ? cta(decode_begin_cta_kernel<1>)
                        : a.d <= CTA_THREADS * 8 ? cta(decode_begin_cta_kernel<2>)
                                                 : cta(decode_begin_cta_kernel<4>);
  arcb_count_launch(1);
  return (int)e;
}

int arcb_launch_head(const HeadArgs& a, const DecodeState& st, cudaStream_t stream) {
  if (a.rows <= 0) return 0;
  auto cta = [&](auto kernel) { return arcb_launch(kernel, dim3(a.rows), dim3(HEAD_THREADS), 0, stream, a, st); };
  const cudaError_t e = !cta_per_row(a.step != 0, a.rows, a.d) ? arcb_launch(head_kernel, dim3((a.rows + ROWS_PER_CTA - 1) / ROWS_PER_CTA),
                                                                dim3(ROWS_PER_CTA * 32), 0, stream, a, st)
                        : a.d <= HEAD_THREADS * 4 ? cta(head_cta_kernel<1>)
                                                  : cta(head_cta_kernel<2>);
  arcb_count_launch(1);
  return (int)e;
}

int arcb_launch_pack_rows(const float* src, void* dst, long long rows, long long cols, int blk,
                          int blk_stride, int blk_off, int to_bf16, cudaStream_t stream) {
  const long long n = rows * cols;
  if (n <= 0) return 0;
  const int threads = 256;
  long long blocks = (n + threads - 1) / threads;
  if (blocks > 148 * 16) blocks = 148 * 16;
  pack_rows_kernel<<<(unsigned)blocks, threads, 0, stream>>>(src, dst, rows, cols, blk, blk_stride, blk_off,
                                                            to_bf16);
  arcb_count_launch(1);
  return (int)cudaGetLastError();
}
