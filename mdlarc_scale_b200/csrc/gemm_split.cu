// y = A[M,K] * W[N,K]^T of 32-bit operands, with the epilogues of epilogue.cuh, on tcgen05.
//
// Every operand value is the exact sum of three bf16 values (8 significant bits each, rounded to nearest one after the other),
// a = a0 + a1 + a2 with |a1| <= 2^-8 |a|, |a2| <= 2^-16 |a|, so a product is nine products of bf16 values, each exact in 32 bits.
// Six of them are taken; a1 w2, a2 w1 and a2 w2 are below 2^-23 of the product, and of either sign.  The matrix unit's own additions
// do not round to nearest, so sums stay short there: the leading products of 128 columns have an accumulator of their own, the five
// smaller ones another, and both are added in registers to the running 32-bit sum.  A row's order of addition depends on K alone.
// Errors against 64 bits, this / multiply-adds in 32 bits (gemm_simt_wide_kernel): K 1280 1.4e-7 / 6.4e-7 of the result's norm, K 5120
// 2.0e-7 / 1.3e-6, factors spread over e^+-3 1.9e-7 / 6.4e-7; largest of an element 6e-8 / 4e-7 of its sum of magnitudes.  The sums of a
// row of A or W with values that have no such pieces (infinities, NaN, beyond the largest bf16) are multiply-adds instead, those of the
// rows beside it stay as they are; below 2^-110 the pieces lose bits as subnormals.
//
// What bounds it: 24 instructions of 128 x 128 x 16 for 64 columns (12 where the weights are bf16 values, as those of a checkpoint
// in 16 bits are: their other pieces are zeros), and next to them the splitting of 16 k values by 16 warps, 6 to 8 operations each, on
// their way from memory to the two operand stages, with one block of loads ahead: 1.0 to 1.2 us a block of 64 columns, issue slots 61 %
// busy, the tensor pipe 26 % (any weights: 56 %, 48 %).  8 warps with twice the work each: the same.
// B200, us a launch, multiply-adds / here with 16-bit weights (any weights): 1719 rows, 1280 x 1280 151 / 35 (39), 5120 x 1280 470 / 131
// (144), 1280 x 5120 588 / 119 (134); 28 rows, 32000 x 1280 160 / 68 (72); 1 row, 1280 x 1280 82 / 33 (35), 1280 x 5120 316 / 119 (125).
// Registers are at their limit (96): a few more held through the loop for redo_without_pieces cost 3 to 13 % of a launch.
#include <atomic>

#include "common.cuh"
#include "gemm.cuh"
#include "gemm_split.cuh"
#include "launch.cuh"
#include "ptx_sm100.cuh"

using namespace sm100;

namespace {

constexpr int GS_WORKERS = 512, GS_THREADS = GS_WORKERS + 32, GS_WARPS = GS_WORKERS / 32;
constexpr int GS_ITEMS = 1024 / GS_WORKERS;       // runs of 8 values of a block of either operand, a thread
constexpr int GS_COLS = 128 * 128 / GS_WORKERS;  // sums of a row, a thread
constexpr int GS_PLANE = 128 * 128;              // 128 rows of 64 bf16
constexpr int GS_STAGE = 6 * GS_PLANE;           // three planes of A, three of W
constexpr int GS_CHUNK = 2;                      // blocks of 64 columns that the matrix unit adds up
constexpr int GS_PITCH = 132;                    // floats of a row of sums in shared memory
constexpr int GS_SMEM = 2 * GS_STAGE + 1024 + 128;

// two values into their bf16 pieces; `odd` becomes NaN when one of them has none (infinities, NaN, beyond the largest bf16)
__device__ __forceinline__ void split2(float x, float y, uint32_t& p0, uint32_t& p1, uint32_t& p2, uint64_t& odd) {
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p0) : "f"(y), "f"(x));
  const float rx = x - __uint_as_float(p0 << 16), ry = y - __uint_as_float(p0 & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p1) : "f"(ry), "f"(rx));
  const float sx = rx - __uint_as_float(p1 << 16), sy = ry - __uint_as_float(p1 & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p2) : "f"(sy), "f"(sx));
  asm("{.reg .b64 t;\n mov.b64 t, {%1, %2};\n fma.rn.f32x2 %0, t, %3, %0;}" : "+l"(odd) : "f"(sx), "f"(sy), "l"(0ull));
}

// tmem_wait_ld_dep of a 16-column load
__device__ __forceinline__ void tmem_wait_ld_dep16(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}

// Sums of a tile that meet a value without pieces, by multiply-adds in order of K as gemm_simt_wide_kernel takes them: those of such a row
// of A or of W.  All others stay as they are, so that what a neighbour holds changes no bit of a row.  `base_ptr`: the tile's
// sums, then (the operands are done with) blocks of 32 columns of both operands.
__device__ __noinline__ void redo_without_pieces(uint8_t* base_ptr, const float* A, const float* W, int K, size_t lda, int a_row0, int rows_in,
                                                 size_t w_row0) {
  constexpr int PA = 33, PW = 36;
  float* part = reinterpret_cast<float*>(base_ptr);
  float* sa = part + 128 * GS_PITCH;
  float* sw = sa + 128 * PA;
  volatile int* flag = reinterpret_cast<volatile int*>(sw + 128 * PW);      // rows of A, then of W
  static_assert((128 * (GS_PITCH + PA + PW) + 256) * 4 <= 2 * GS_STAGE && 128 * PA % 4 == 0, "shared memory");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < 256) flag[tid] = 0;
  __syncthreads();
  // 512 threads: four values of rows tid / 8 and tid / 8 + 64 of both operands
  const int q = (tid & 7) * 4;
  auto quad = [&](bool of_w, int row, int k) {
    if (of_w) return __ldg(reinterpret_cast<const float4*>(W + (w_row0 + row) * K + k));
    return row < rows_in ? __ldcg(reinterpret_cast<const float4*>(A + (size_t)(a_row0 + row) * lda + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  if (warp < GS_WARPS)
    for (int i = 0; i < 4; ++i) {
      const int row = (tid >> 3) + 64 * (i & 1);
      uint64_t odd = 0ull;
      for (int k = q; k < K; k += 32) {
        const float4 v = quad(i >> 1, row, k);
        uint32_t p[3];
        split2(v.x, v.y, p[0], p[1], p[2], odd);
        split2(v.z, v.w, p[0], p[1], p[2], odd);
      }
      float ox, oy;
      asm("mov.b64 {%0, %1}, %2;" : "=f"(ox), "=f"(oy) : "l"(odd));
      if (!(ox == 0.f && oy == 0.f)) flag[128 * (i >> 1) + row] = 1;
    }
  __syncthreads();
  const int r = (warp & 3) * 32 + lane, c0 = (warp >> 2) * GS_COLS;
  uint32_t cols = 0;
  bool row = false;
  if (warp < GS_WARPS) {
    cols = __ballot_sync(0xffffffffu, flag[128 + c0 + lane] != 0);
    row = flag[r] != 0;
  }
  const bool any = cols || __any_sync(0xffffffffu, row);
  float acc[GS_COLS];
#pragma unroll
  for (int i = 0; i < GS_COLS; ++i) acc[i] = 0.f;
  for (int k0 = 0; k0 < K; k0 += 32) {
    if (warp < GS_WARPS)
      for (int i = 0; i < 2; ++i) {
        const int rr = (tid >> 3) + 64 * i;
        const float4 a = quad(false, rr, k0 + q);
        float* to = sa + rr * PA + q;
        to[0] = a.x; to[1] = a.y; to[2] = a.z; to[3] = a.w;
        *reinterpret_cast<float4*>(sw + rr * PW + q) = quad(true, rr, k0 + q);
      }
    __syncthreads();
    if (any)
      for (int k = 0; k < 32; k += 4) {
        const float a[4] = {sa[r * PA + k], sa[r * PA + k + 1], sa[r * PA + k + 2], sa[r * PA + k + 3]};
#pragma unroll
        for (int i = 0; i < GS_COLS; ++i) {
          const float4 w = *reinterpret_cast<const float4*>(sw + (c0 + i) * PW + k);
          acc[i] = fmaf(a[3], w.w, fmaf(a[2], w.z, fmaf(a[1], w.y, fmaf(a[0], w.x, acc[i]))));
        }
      }
    __syncthreads();
  }
  if (any)
#pragma unroll
    for (int i = 0; i < GS_COLS; ++i)
      if (row || (cols >> i & 1)) part[r * GS_PITCH + c0 + i] = acc[i];
  __syncthreads();
}

template <int MODE>
__global__ void __launch_bounds__(GS_THREADS, 1)
gemm_split_kernel(const float* A, const float* W, GemmEpilogue ep, int K, uint32_t idesc) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  const int m0 = blockIdx.y * 128, n0 = blockIdx.x * 128;
  const GroupArgs& g = ep.grp;
  if (g.n_tiles && (int)blockIdx.y >= *g.n_tiles) return;
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  const uint32_t bars = base + 2 * GS_STAGE;
  const uint32_t full = bars, empty = bars + 16, acc_full = bars + 32, acc_empty = bars + 48;      // two each
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(base_ptr + 2 * GS_STAGE + 64);
  volatile int* w_fine = reinterpret_cast<volatile int*>(base_ptr + 2 * GS_STAGE + 72);      // per stage: 1 + last block with finer weights
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int blocks = K / 64, chunks = (blocks + GS_CHUNK - 1) / GS_CHUNK;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      w_fine[s] = 0;
      mbar_init(full + 8 * s, GS_WORKERS);
      mbar_init(empty + 8 * s, 1);
      mbar_init(acc_full + 8 * s, 1);
      mbar_init(acc_empty + 8 * s, GS_WORKERS);
    }
    mbar_fence_init();
  }
  if (warp == GS_WARPS) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;              // accumulators of chunk c at 256 (c & 1): leading products, smaller ones at + 128

  const int a_row0 = g.tile_src ? g.tile_src[blockIdx.y] : m0;
  int rows_in = (int)min(128ll, (g.a_rows ? g.a_rows : ep.M) - a_row0);      // rows of A in this tile, the others are zeros
  // padding of a group is memory that nothing wrote: no part of it may choose how sums are taken
  if (g.tile_rows) rows_in = min(rows_in, g.tile_rows[blockIdx.y]);
  const size_t lda = g.lda ? g.lda : K;
  const size_t w_row0 = (size_t)n0 + (g.tile_group ? (size_t)g.tile_group[blockIdx.y] * g.group_rows : 0);
  float* part = reinterpret_cast<float*>(base_ptr);
  bool ok = true;
  auto wait_or_flag = [&](uint32_t bar, uint32_t parity, int code) {
    if (ok && !mbar_wait_bounded(bar, parity)) {
      arcb_set_error(ep.err, code);
      ok = false;
    }
  };

  bool odd = false;
  if (warp == GS_WARPS) {
    if (lane == 0) {
      for (int b = 0; ok && b < blocks; ++b) {
        const int c = b / GS_CHUNK, s = b & 1;
        if (b % GS_CHUNK == 0 && c >= 2) wait_or_flag(acc_empty + 8 * (c & 1), ((c >> 1) - 1) & 1, ARCB_DEV_WAIT_TIMEOUT_ACC);
        wait_or_flag(full + 8 * s, (b >> 1) & 1, ARCB_DEV_WAIT_TIMEOUT_TMA);
        if (!ok) break;
        tc_fence_after();
        const bool fine = w_fine[s] == b + 1;    // else these weights are bf16 values: their second and third pieces are zeros
        uint64_t a[3], w[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          a[i] = umma_desc_k_sw128(base + s * GS_STAGE + i * GS_PLANE);
          w[i] = umma_desc_k_sw128(base + s * GS_STAGE + (3 + i) * GS_PLANE);
        }
        const uint32_t lead = tmem + 256 * (c & 1), rest = lead + 128;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t add = (b % GS_CHUNK || k) ? 1u : 0u;
          if (fine) umma_f16(rest, a[1] + 2 * k, w[1] + 2 * k, idesc, add);
          umma_f16(lead, a[0] + 2 * k, w[0] + 2 * k, idesc, add);
          umma_f16(rest, a[2] + 2 * k, w[0] + 2 * k, idesc, fine ? 1u : add);
          if (fine) umma_f16(rest, a[0] + 2 * k, w[2] + 2 * k, idesc, 1u);
          umma_f16(rest, a[1] + 2 * k, w[0] + 2 * k, idesc, 1u);
          if (fine) umma_f16(rest, a[0] + 2 * k, w[1] + 2 * k, idesc, 1u);
        }
        umma_commit(empty + 8 * s);
        if (b % GS_CHUNK == GS_CHUNK - 1 || b == blocks - 1) umma_commit(acc_full + 8 * (c & 1));
      }
    }
    __syncwarp();
  } else {
    // eight neighbouring values of rows r0, r0 + 32, ... of both operands, a block ahead in registers
    const int r0 = threadIdx.x >> 3, q = threadIdx.x & 7;
    float4 ra[GS_ITEMS][2], rw[GS_ITEMS][2];
    auto fetch_a = [&](int b) {
#pragma unroll
      for (int j = 0; j < GS_ITEMS; ++j) {
        const int row = r0 + 128 / GS_ITEMS * j;
        const float4* src = reinterpret_cast<const float4*>(A + (size_t)(a_row0 + row) * lda + b * 64 + q * 8);
        const bool in = row < rows_in;
        ra[j][0] = in ? __ldcg(src) : make_float4(0.f, 0.f, 0.f, 0.f);
        ra[j][1] = in ? __ldcg(src + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    auto fetch_w = [&](int b) {
#pragma unroll
      for (int j = 0; j < GS_ITEMS; ++j) {
        const float4* src = reinterpret_cast<const float4*>(W + (w_row0 + r0 + 128 / GS_ITEMS * j) * K + b * 64 + q * 8);
        rw[j][0] = __ldg(src);
        rw[j][1] = __ldg(src + 1);
      }
    };
    uint64_t sum_odd = 0ull;
    const uint32_t dst0 = base + r0 * 128 + ((q ^ (r0 & 7)) << 4);     // rows 32 apart share the swizzle
    // Pieces that are all zeros (bf16 weights, rows beyond the last) are not written where zeros are already: `dirty` has a bit for
    // each of this thread's places in a stage.
    uint32_t dirty = ~0u;
    auto store = [&](uint32_t at, const float4 (&v)[GS_ITEMS][2], uint32_t place) {
      uint32_t fine = 0;
#pragma unroll
      for (int j = 0; j < GS_ITEMS; ++j) {
        uint32_t p[3][4];
        split2(v[j][0].x, v[j][0].y, p[0][0], p[1][0], p[2][0], sum_odd);
        split2(v[j][0].z, v[j][0].w, p[0][1], p[1][1], p[2][1], sum_odd);
        split2(v[j][1].x, v[j][1].y, p[0][2], p[1][2], p[2][2], sum_odd);
        split2(v[j][1].z, v[j][1].w, p[0][3], p[1][3], p[2][3], sum_odd);
        const uint32_t any = p[1][0] | p[1][1] | p[1][2] | p[1][3] | p[2][0] | p[2][1] | p[2][2] | p[2][3], bit = place << j;
#pragma unroll
        for (int i = 0; i < 3; ++i)
          if (i == 0 || any || (dirty & bit))
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + i * GS_PLANE + j * (128 / GS_ITEMS) * 128), "r"(p[i][0]), "r"(p[i][1]),
                         "r"(p[i][2]), "r"(p[i][3])
                         : "memory");
        dirty = any ? dirty | bit : dirty & ~bit;
        fine |= any;
      }
      return fine != 0;
    };
    float acc[GS_COLS];
#pragma unroll
    for (int i = 0; i < GS_COLS; ++i) acc[i] = 0.f;
    const uint32_t t_acc = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * GS_COLS;
    auto drain = [&](int c) {
      wait_or_flag(acc_full + 8 * (c & 1), (c >> 1) & 1, ARCB_DEV_WAIT_TIMEOUT_ACC);
      __syncwarp();
      tc_fence_after();
#pragma unroll
      for (int h = 0; h < GS_COLS / 16; ++h)
#pragma unroll
        for (int part = 1; part >= 0; --part) {
          uint32_t v[16];
          tmem_ld_32x16(t_acc + 256 * (c & 1) + 128 * part + h * 16, v);
          tmem_wait_ld_dep16(v);
#pragma unroll
          for (int i = 0; i < 16; ++i) acc[h * 16 + i] += __uint_as_float(v[i]);
        }
      tc_fence_before();
      mbar_arrive(acc_empty + 8 * (c & 1));
    };
    fetch_a(0);
    fetch_w(0);
    for (int b = 0; b < blocks; ++b) {
      const int s = b & 1;
      if (b >= 2) wait_or_flag(empty + 8 * s, ((b >> 1) - 1) & 1, ARCB_DEV_WAIT_TIMEOUT_MMA);
      store(dst0 + s * GS_STAGE, ra, 1u << (s * 2 * GS_ITEMS));
      if (b + 1 < blocks) fetch_a(b + 1);
      if (store(dst0 + s * GS_STAGE + 3 * GS_PLANE, rw, 1u << (s * 2 * GS_ITEMS + GS_ITEMS))) w_fine[s] = b + 1;
      if (b + 1 < blocks) fetch_w(b + 1);
      fence_proxy_async_smem();
      mbar_arrive(full + 8 * s);
      if (b % GS_CHUNK == GS_CHUNK - 1 && b >= GS_CHUNK) drain(b / GS_CHUNK - 1);
    }
    if (blocks % GS_CHUNK && chunks > 1) drain(chunks - 2);
    drain(chunks - 1);
    float ox, oy;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(ox), "=f"(oy) : "l"(sum_odd));
    odd = !(ox == 0.f && oy == 0.f);
    float* dst = part + ((warp & 3) * 32 + lane) * GS_PITCH + (warp >> 2) * GS_COLS;
#pragma unroll
    for (int i = 0; i < GS_COLS; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
  }
  if (__syncthreads_or(odd)) redo_without_pieces(base_ptr, A, W, K, lda, a_row0, rows_in, w_row0);
  if (warp < GS_WARPS) {
    constexpr bool PAIRED = MODE == EPI_GLU;
    constexpr int STEP = (PAIRED ? 2 : 1) * GS_WARPS, U = 4;
    const int c = (PAIRED ? lane & 15 : lane) * 4, n = n0 + c;
    for (int r0 = PAIRED ? warp * 2 + (lane >> 4) : warp; r0 < 128; r0 += U * STEP) {
      QuadAhead ahead[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (m0 + r0 + u * STEP < ep.M) ahead[u].template load<MODE>(ep, m0 + r0 + u * STEP, n);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int r = r0 + u * STEP, m = m0 + r;
        if (m >= ep.M) continue;
        const float4 v = *reinterpret_cast<const float4*>(part + r * GS_PITCH + c);
        if constexpr (MODE == EPI_RESID) epi_resid_quad(ep, m, n, v, ahead[u].a, ahead[u].b);
        else if constexpr (MODE == EPI_GLU) epi_glu_quad(ep, m, n, v, *reinterpret_cast<const float4*>(part + r * GS_PITCH + c + 64));
        else if constexpr (MODE == EPI_RELU2) epi_relu2_quad(ep, m, n, v);
        else if constexpr (MODE == EPI_ACT) epi_act_quad(ep, m, n, v);
        else epi_store_quad(ep, m, n, v);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == GS_WARPS) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

template <int MODE>
int launch(const void* a, const void* w, const GemmEpilogue& ep, int K, cudaStream_t stream) {
  static std::atomic<unsigned long long> opted{0};
  cudaError_t e = arcb_opt_in_smem(gemm_split_kernel<MODE>, GS_SMEM, opted);
  if (e == cudaSuccess)
    e = arcb_launch(gemm_split_kernel<MODE>, dim3(ep.N / 128, (ep.M + 127) / 128), dim3(GS_THREADS), GS_SMEM, stream, reinterpret_cast<const float*>(a),
                    reinterpret_cast<const float*>(w), ep, K, umma_idesc_f16(128, 128, 1, 1));
  arcb_count_launch(1);
  return (int)e;
}

}  // namespace

bool arcb_gemm_split_applies(const void* a, const void* w, const GemmEpilogue& ep, int K) {
  if (ep.act_f16 != 2 || ep.M <= 0 || K <= 0 || K % 64 || ep.N % 128 || (ep.M + 127) / 128 > 65535) return false;
  const GroupArgs& g = ep.grp;
  if (g.panels || g.n_group || g.lda % 4) return false;
  const uintptr_t all = (uintptr_t)a | (uintptr_t)w | (uintptr_t)ep.x | (uintptr_t)ep.y | (uintptr_t)ep.out16 | (uintptr_t)ep.bias;
  if (all & 15) return false;
  switch (ep.mode) {
    case EPI_STORE_F32: case EPI_RESID: case EPI_RELU2: case EPI_ACT: case EPI_GLU: return true;
  }
  return false;
}

int arcb_launch_gemm_split(const void* a, const void* w, const GemmEpilogue& ep, int K, cudaStream_t stream) {
  switch (ep.mode) {
    case EPI_STORE_F32: return launch<EPI_STORE_F32>(a, w, ep, K, stream);
    case EPI_RESID: return launch<EPI_RESID>(a, w, ep, K, stream);
    case EPI_RELU2: return launch<EPI_RELU2>(a, w, ep, K, stream);
    case EPI_ACT: return launch<EPI_ACT>(a, w, ep, K, stream);
    case EPI_GLU: return launch<EPI_GLU>(a, w, ep, K, stream);
  }
  return -1;
}
