// y = A[M,K] * W[N,K]^T for one tile of up to 256 rows (decode steps of mid-sized batches, wide heads), epilogues of epilogue.cuh.
//
// With 128 x 128 tiles of A rows and W rows, such a product is 8 to 65 CTAs that each pull (128 + 128) x K operands through
// one SM's 110 GB/s, one after the other.  Here the product is transposed: 128 rows of W are the matrix instruction's rows
// and all rows of A, rounded up to 16, its columns, so weights cross once whatever the row count and no second row tile is
// mostly padding.  The K blocks of a tile are divided among the CTAs of a cluster: each loads its share (most or all of it in
// flight at once), leaves its fp32 partial in its own shared memory, and sums a slice of the rows over the cluster's
// partials, always in the same order, into the epilogue.  What is left is a chain: first operands 1.3 us after the start,
// accumulators 0.6 us after the last, 0.4 us into shared memory, 2 to 3 us to meet, sum and store.
// B200, us a launch in a captured chain with weights from memory, 128 x 128 tiles (or their split in two) / here: 128 rows,
// 1024 x 1024 9.3 / 7.5, 1024 x 2752 16.3 / 8.8, 3072 x 1024 9.5 / 8.3, 5504 x 1024 10.2 / 9.7; 150 rows, 2048 x 2048 14.0 / 10.0,
// 2048 x 8192 38.7 / 14.6, 8320 x 2048 15.0 / 14.2, 32000 x 2048 53 / 34.
#include <cuda.h>

#include <atomic>
#include <mutex>

#include "common.cuh"
#include "gemm.cuh"
#include "gemm_mid.cuh"
#include "launch.cuh"
#include "ptx_sm100.cuh"
#include "step_rules.cuh"

using namespace sm100;

namespace {

constexpr int GM_THREADS = 256;
// SMAX: no more CTAs in a cluster (1, 4 or 8); what a thread sums is requested before the first addition.
template <int MODE, int SMAX>
__global__ void __launch_bounds__(GM_THREADS, SMAX == 1 ? 2 : 1)
gemm_mid_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a, GemmEpilogue ep, int num_k,
                uint32_t idesc, GmShape sh) {
  pdl_launch_dependents();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  const int stage_bytes = GM_W_BYTES + sh.rows * 128, ring = sh.stages * stage_bytes, part_bytes = sh.rows * 512;
  const uint32_t bars = base + (ring > part_bytes ? ring : part_bytes);      // full[stages], empty[stages], acc
  const uint32_t bar_acc = bars + 16 * sh.stages;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(base_ptr + (bar_acc + 8 - base));
  volatile uint32_t* abort_flag = tmem_slot + 1;
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // known to be the same in a warp
  const int rank = blockIdx.x % sh.splits, n0 = blockIdx.x / sh.splits * 128;
  const int kb0 = rank * num_k / sh.splits, kb1 = (rank + 1) * num_k / sh.splits;
  const uint32_t tmem_cols = sh.rows <= 128 ? 128 : 256;

  // warp 0 lane 0: barriers, then operands at once; nobody else is needed for either
  auto fetch = [&](int kb, int stage) {
    const uint32_t dst = base + stage * stage_bytes, full = bars + 8 * stage;
    mbar_expect_tx(full, stage_bytes);
    tma_load_2d(dst, &tmap_w, kb * 64, n0, full);
    tma_load_2d(dst + GM_W_BYTES, &tmap_a, kb * 64, 0, full);
  };
  const int first = min(sh.stages, kb1 - kb0);
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2 * sh.stages; ++s) mbar_init(bars + 8 * s, 1);
    mbar_init(bar_acc, 1);
    *abort_flag = 0;
    mbar_fence_init();
    pdl_wait();
    for (int i = 0; i < first; ++i) fetch(kb0 + i, i);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  pdl_wait();

  if (warp == 0 && lane == 0) {
    for (int i = first, s = 0, turn = 0; i < kb1 - kb0; ++i) {
      if (!mbar_wait_bounded(bars + 8 * (sh.stages + s), turn)) {
        arcb_set_error(ep.err, ARCB_DEV_WAIT_TIMEOUT_MMA);
        *abort_flag = 1;
        break;
      }
      if (*abort_flag) break;
      fetch(kb0 + i, s);
      if (++s == sh.stages) { s = 0; turn ^= 1; }
    }
  } else if (warp == 1) {
    // the whole warp, an elected lane issues: operands stay in uniform registers (48 rows x 1280 columns 7.3 -> 6.9 us a
    // launch, gated 9.6 -> 8.8)
    const uint32_t el = elect_one();
    bool ok = true;
    for (int i = 0, s = 0, turn = 0; i < kb1 - kb0; ++i) {
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(bars + 8 * s, turn))) {
        arcb_set_error(ep.err, ARCB_DEV_WAIT_TIMEOUT_TMA);
        *abort_flag = 1;
        ok = false;
        break;
      }
      tc_fence_after();
      const uint64_t dw = umma_desc_k_sw128(base + s * stage_bytes), da = umma_desc_k_sw128(base + s * stage_bytes + GM_W_BYTES);
#pragma unroll
      for (int k4 = 0; k4 < 4; ++k4) umma_f16_if(el, tmem, dw + 2 * k4, da + 2 * k4, idesc, (i | k4) ? 1u : 0u);
      umma_commit_if(el, bars + 8 * (sh.stages + s));
      if (++s == sh.stages) { s = 0; turn ^= 1; }
    }
    if (ok) umma_commit_if(el, bar_acc);
  }
  __syncwarp();

  // this CTA's slice of the rows, and what its first rows need besides the sums
  constexpr bool PAIRED = MODE == EPI_SWIGLU || MODE == EPI_GLU;
  constexpr int U = SMAX == 8 || PAIRED ? 2 : 4, STEP = PAIRED ? 16 : 8;   // rows in flight a thread, rows a pass of the CTA
  const int per = (sh.rows + sh.splits - 1) / sh.splits;
  const int r_end = min(min((rank + 1) * per, sh.rows), ep.M);
  const int r_first = rank * per + (PAIRED ? warp * 2 + (lane >> 4) : warp);
  const int c = (PAIRED ? lane & 15 : lane) * 4, n = n0 + c;
  QuadAhead ahead[U];
  auto load_ahead = [&](int r0) {
    if constexpr (MODE == EPI_RESID || MODE == EPI_SWIGLU || MODE == EPI_QKV_ROPE)
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (r0 + u * STEP < r_end) ahead[u].template load<MODE>(ep, r0 + u * STEP, n);
  };
  load_ahead(r_first);

  const bool ok = __syncthreads_and(mbar_wait_bounded(bar_acc, 0)) != 0;
  if (!ok && threadIdx.x == 0) arcb_set_error(ep.err, ARCB_DEV_WAIT_TIMEOUT_ACC);
  tc_fence_after();
  float* part = reinterpret_cast<float*>(base_ptr);                  // [rows][128], in the ring's place
  if (ok) {
    const int quarter = warp & 3;
    const uint32_t t_row = tmem + ((uint32_t)(quarter * 32) << 16);
    for (int r0 = (warp >> 2) * 32; r0 < sh.rows; r0 += 64) {
      uint32_t v[32];
      tmem_ld_32x32(t_row + r0, v);
      tmem_wait_ld();
      float* dst = part + r0 * 128 + quarter * 32 + lane;
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (r0 + i < sh.rows) dst[i * 128] = __uint_as_float(v[i]);
    }
  }
  tc_fence_before();
  if constexpr (SMAX > 1) cluster_sync_all();
  else __syncthreads();

  // the same for a whole warp: epilogues shuffle
  const int r_warp = r_first - (PAIRED ? lane >> 4 : 0), passes = ok && r_warp < r_end ? (r_end - r_warp + U * STEP - 1) / (U * STEP) : 0;
  if constexpr (SMAX > 1)
    if (passes == 0) cluster_arrive();
  const uint32_t at = base + c * 4;
  constexpr int H = PAIRED ? 2 : 1;              // gate and up quads
  for (int pass = 0; pass < passes; ++pass) {
    const int r0 = r_first + pass * U * STEP;
    if (pass > 0) load_ahead(r0);
    float4 o[SMAX][U][H];
#pragma unroll
    for (int k = 0; k < SMAX; ++k)
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int h = 0; h < H; ++h) {
          o[k][u][h] = make_float4(0.f, 0.f, 0.f, 0.f);
          const int r = r0 + u * STEP;
          if (k < sh.splits && r < r_end) {
            if constexpr (SMAX > 1) o[k][u][h] = ld_shared_cluster_v4(at + r * 512 + h * 256, k);
            else o[k][u][h] = *reinterpret_cast<const float4*>(part + r * 128 + c + h * 64);
          }
        }
    float4 v[U], up[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int h = 0; h < H; ++h) {
        float4 sum = o[0][u][h];
#pragma unroll
        for (int k = 1; k < SMAX; ++k)
          if (k < sh.splits) { sum.x += o[k][u][h].x; sum.y += o[k][u][h].y; sum.z += o[k][u][h].z; sum.w += o[k][u][h].w; }
        if (h == 0) v[u] = sum;
        else up[u] = sum;
      }
    if constexpr (SMAX > 1) {
      __syncwarp();
      if (pass + 1 == passes) cluster_arrive();                      // all that this warp reads of its peers is read
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int m = r0 + u * STEP;
      if constexpr (MODE == EPI_HEADS) {
        // a warp holds a row's 128 columns: one head of 128 or two of 64
        epi_heads_quad(ep, m < r_end ? m : -1, n, v[u], [&](float ss, bool, int width, int) {
#pragma unroll
          for (int o = 1; o < 16; o <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
          const float other = __shfl_xor_sync(0xffffffffu, ss, 16);
          return width > 64 ? ss + other : ss;
        });
        continue;
      }
      if (m >= r_end) continue;
      if constexpr (MODE == EPI_QKV_ROPE)
        epi_qkv_quad(ep, ahead[u].rr, m, n, v[u], make_float2(ahead[u].a.x, ahead[u].a.y), make_float2(ahead[u].a.z, ahead[u].a.w));
      else if constexpr (MODE == EPI_RESID) epi_resid_quad(ep, m, n, v[u], ahead[u].a, ahead[u].b);
      else if constexpr (MODE == EPI_SWIGLU) epi_swiglu_quad(ep, m, n, v[u], up[u], ahead[u].a, ahead[u].b);
      else if constexpr (MODE == EPI_GLU) epi_glu_quad(ep, m, n, v[u], up[u]);
      else if constexpr (MODE == EPI_RELU2) epi_relu2_quad(ep, m, n, v[u]);
      else if constexpr (MODE == EPI_ACT) epi_act_quad(ep, m, n, v[u]);
      else if constexpr (MODE == EPI_STORE_F32) epi_store_quad(ep, m, n, v[u]);
    }
  }
  if constexpr (SMAX > 1) cluster_wait();        // nobody leaves while its partial is read
  else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, tmem_cols);
  }
}

constexpr int GM_DEVICES = 64;

int current_device() {
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < GM_DEVICES ? dev : 0;
}

// clusters of `splits` CTAs, one CTA an SM, that run at once on this device
int clusters_at_once(int splits) {
  static std::mutex mu;
  static int known[GM_DEVICES][GM_SPLIT_MAX + 1];
  static std::atomic<unsigned long long> opted{0};
  std::lock_guard<std::mutex> lock(mu);
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = splits;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(splits * arcb_num_sms());
  cfg.blockDim = dim3(GM_THREADS);
  cfg.dynamicSmemBytes = GM_SMEM_MAX;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return asked_once(known[current_device()][splits], [&](int& n) {
    const bool ok = arcb_opt_in_smem(gemm_mid_kernel<EPI_RESID, 8>, GM_SMEM_MAX, opted) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&n, gemm_mid_kernel<EPI_RESID, 8>, &cfg) == cudaSuccess;
    if (!ok) cudaGetLastError();
    return ok;
  });
}

template <int MODE>
int launch(const void* a, const void* w, const GemmEpilogue& ep, int K, int act_f16, cudaStream_t stream) {
  const GmShape sh = gm_shape(ep.M, ep.N, K, arcb_num_sms(), clusters_at_once);
  CUtensorMap tw, ta;
  int r = arcb_make_tmap_2d_16b(&tw, w, (uint64_t)ep.N, (uint64_t)K, 128, 64, act_f16);
  if (!r) r = arcb_make_tmap_2d_16b(&ta, a, (uint64_t)ep.M, (uint64_t)(ep.grp.lda ? ep.grp.lda : K), sh.rows, 64, act_f16);
  if (r) return 1000 + r;
  const uint32_t idesc = umma_idesc_f16(128, sh.rows, act_f16 ? 0 : 1, act_f16 ? 0 : 1);
  static std::atomic<unsigned long long> opted[3];
  auto run = [&](auto kernel, std::atomic<unsigned long long>& done) {
    const cudaError_t e = arcb_opt_in_smem(kernel, GM_SMEM_MAX, done);
    return e != cudaSuccess ? e : arcb_launch_cluster(kernel, sh.splits, dim3(ep.N / 128 * sh.splits), dim3(GM_THREADS), sh.smem(), stream, tw, ta, ep,
                                                      K / 64, idesc, sh);
  };
  const cudaError_t e = sh.splits == 1   ? run(gemm_mid_kernel<MODE, 1>, opted[0])
                        : sh.splits <= 4 ? run(gemm_mid_kernel<MODE, 4>, opted[1])
                                         : run(gemm_mid_kernel<MODE, 8>, opted[2]);
  arcb_count_launch(1);
  return (int)e;
}

}  // namespace

// Decode steps only: how a sum is divided depends on the number of rows, and a prompt row's result does not depend on what
// else its call holds.
bool arcb_gemm_mid_applies(const void* a, const void* w, const GemmEpilogue& ep, int K, int act_f16) {
  if (!ep.step || !mid_transposes(ep.M, ep.N, K, arcb_num_sms()) || act_f16 == 2 || K % 64 || ep.N % 128) return false;
  const GroupArgs& g = ep.grp;
  if (g.tile_src || g.tile_group || g.n_tiles || g.panels || g.n_group || g.lda % 8) return false;
  // 16-byte accesses of the epilogues' quads; what is not aligned meets the tensor maps' refusal
  const uintptr_t all = (uintptr_t)a | (uintptr_t)w | (uintptr_t)ep.x | (uintptr_t)ep.y | (uintptr_t)ep.out16 | (uintptr_t)ep.bias | (uintptr_t)ep.pj.out;
  if (all & 15) return false;
  return ep.mode != EPI_HEADS || !(ep.pj.q_norm || ep.pj.k_norm) || ep.pj.dimp <= 128;
}

int arcb_launch_gemm_mid(const void* a, const void* w, const GemmEpilogue& ep, int K, int act_f16, cudaStream_t stream) {
  switch (ep.mode) {
    case EPI_STORE_F32: return launch<EPI_STORE_F32>(a, w, ep, K, act_f16, stream);
    case EPI_QKV_ROPE: return launch<EPI_QKV_ROPE>(a, w, ep, K, act_f16, stream);
    case EPI_RESID: return launch<EPI_RESID>(a, w, ep, K, act_f16, stream);
    case EPI_SWIGLU: return launch<EPI_SWIGLU>(a, w, ep, K, act_f16, stream);
    case EPI_RELU2: return launch<EPI_RELU2>(a, w, ep, K, act_f16, stream);
    case EPI_HEADS: return launch<EPI_HEADS>(a, w, ep, K, act_f16, stream);
    case EPI_ACT: return launch<EPI_ACT>(a, w, ep, K, act_f16, stream);
    case EPI_GLU: return launch<EPI_GLU>(a, w, ep, K, act_f16, stream);
  }
  return -1;
}
