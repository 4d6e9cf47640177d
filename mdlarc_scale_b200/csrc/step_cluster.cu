// Decode steps of the smallest models (up to 4 rows of 384 columns): any number of steps in one launch of one cluster.
//
// A step of such a model is 28 launches of 1.5 to 3.7 us for four layers, each a chain of loads, one reduction and a store, while
// all weights together stream from L2 in a few microseconds.  Here 16 SMs take the whole loop (on a device that runs no cluster of 16 the
// launches stay): columns of every product are divided among the CTAs, rows of 16 weights at a time on mma.m16n8k16 (the sequences
// are its columns); what the next phase reads (queries, attention records, residual stream, hidden units) is written into every
// CTA's shared memory, and a cluster barrier (five a layer) takes the place of a launch.  A phase's weights are copied into shared
// memory while the phase before it runs.  Norms, embedding and the merge of attention records are repeated in every CTA.
// Rounding points are those of the separate kernels; sums over K and over keys are divided differently.
// What bounds it is latency: of 18 k cycles a layer (width 256, one row) 5.5 k are barriers with the stores they wait for, 3.5 k
// products, 3.3 k their epilogues, 3 k attention, 1.5 k norms.  B200, one row of 168 to 300 cached rows, us a step: launches of
// a graph 70, here 46 in a launch of many steps, 51 in one of a single step (weights through registers 48, by 16-byte asynchronous copies 52).
#include <mutex>

#include "common.cuh"
#include "epilogue.cuh"
#include "gemm.cuh"
#include "greedy_loop.cuh"
#include "launch.cuh"
#include "ptx_sm100.cuh"
#include "step_cluster.cuh"
#include "step_rules.cuh"

using namespace sm100;

namespace {

constexpr int SC_WARPS = 8, SC_THREADS = 32 * SC_WARPS;
constexpr int SC_PITCH = 20, SC_PART = 8 * SC_PITCH;       // a warp's sums of a tile: 8 rows of 16 columns, padded
constexpr int SC_REC = 68;                                 // attention record: 64 sums, maximum, normaliser
constexpr float LOG2E = 1.4426950408889634f;

template <bool F16>
__device__ __forceinline__ void mma16816(float (&c)[4], const uint4& lo, const uint4& hi, const uint4& x) {
  if constexpr (F16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n\t"
                 "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%10,%11,%12,%13}, {%14,%15}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(lo.x), "r"(hi.x), "r"(lo.y), "r"(hi.y), "r"(x.x), "r"(x.y), "r"(lo.z), "r"(hi.z), "r"(lo.w), "r"(hi.w), "r"(x.z), "r"(x.w));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n\t"
                 "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%10,%11,%12,%13}, {%14,%15}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(lo.x), "r"(hi.x), "r"(lo.y), "r"(hi.y), "r"(x.x), "r"(x.y), "r"(lo.z), "r"(hi.z), "r"(lo.w), "r"(hi.w), "r"(x.z), "r"(x.w));
}

__device__ __forceinline__ uint32_t at_rank(uint32_t addr, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  return a;
}
// a value at this shared address of CTA `rank` of the cluster
__device__ __forceinline__ void tell(const void* p, int rank, uint2 v) {
  asm volatile("st.shared::cluster.v2.b32 [%0], {%1, %2};" ::"r"(at_rank(smem_u32(p), rank)), "r"(v.x), "r"(v.y) : "memory");
}
__device__ __forceinline__ void tell(const void* p, int rank, float4 v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at_rank(smem_u32(p), rank)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void tell(const void* p, int rank, int4 v) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at_rank(smem_u32(p), rank)), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// This CTA's column tiles of a product: tile i of the plain products is columns 16 (rank + i cl); of gate/up (paired) tiles 2 i and
// 2 i + 1 are 16 gate columns and their up columns, 64 further, of unit rank + i cl.  A warp takes every eighth block of 32 columns.
struct Part {
  const uint16_t* w;
  int K, tiles;
  bool paired;
};
__device__ __forceinline__ int tile_row(const Part& p, int tile, int rank, int cl) {
  if (!p.paired) return (rank + tile * cl) * 16;
  const int u = rank + (tile >> 1) * cl;
  return (u >> 2) * 128 + (u & 3) * 16 + (tile & 1) * 64;
}

// A part's weights on their way into `buf`: a tile is 16 whole rows, one run of memory.  A lane of every warp asks for the warp's share of
// the tiles: issuing a copy takes 150 cycles.
__device__ __forceinline__ void request(const Part& p, int rank, int cl, uint32_t buf, uint32_t bar) {
  if ((threadIdx.x & 31) != 0) return;
  const int warp = threadIdx.x >> 5, mine = (p.tiles - warp + SC_WARPS - 1) / SC_WARPS;
  const uint32_t bytes = 32 * p.K;
  if (mine > 0) mbar_expect_tx(bar, mine * bytes);
  else mbar_arrive(bar);
  for (int tile = warp; tile < p.tiles; tile += SC_WARPS)
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(buf + tile * bytes),
                 "l"(p.w + (size_t)tile_row(p, tile, rank, cl) * p.K), "r"(bytes), "r"(bar)
                 : "memory");
}

// K of a product is divided into 2^k_parts(K) parts, up to eight, of whole pairs of blocks of 32 columns.
__device__ __forceinline__ int k_parts(int K) { return K >= 512 ? 3 : K >= 256 ? 2 : K >= 128 ? 1 : 0; }

// x: rows of `pitch` bytes; red: [tile][part][SC_PART].  A warp takes a part of three tiles at a time: what takes time is the chain of
// load, products, store.  Rows of weights lie a multiple of 128 bytes apart, so neighbouring rows read the two blocks of a pair
// in opposite order: no two lanes of a quarter warp meet on a bank.  One copy of the code for all products: the loop over layers has
// to stay in the instruction cache.
template <bool F16>
__device__ __noinline__ void multiply(int K, int tiles, const uint8_t* buf, const uint8_t* x, int pitch, float* red) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, lg = k_parts(K), pairs = K / 64;
  const int part = warp & ((1 << lg) - 1), begin = part * pairs >> lg, end = (part + 1) * pairs >> lg;
  const uint8_t* xg = x + g * pitch + t * 16;
  const bool swap = g & 1;
  const uint8_t* w0 = buf + g * 2 * K + t * 16 + (swap ? 64 : 0);
  const int other = swap ? -64 : 64;
  constexpr int G = 3;
  for (int tile = G * (warp >> lg); tile < tiles; tile += G * (SC_WARPS >> lg)) {
    float acc[G][4];
#pragma unroll
    for (int j = 0; j < G; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    for (int b = begin; b < end; ++b) {
      const uint4 x0 = *reinterpret_cast<const uint4*>(xg + b * 128), x1 = *reinterpret_cast<const uint4*>(xg + b * 128 + 64);
#pragma unroll
      for (int j = 0; j < G; ++j) {
        const uint8_t* w = w0 + min(tile + j, tiles - 1) * 32 * K + b * 128;
        const uint4 lo = *reinterpret_cast<const uint4*>(w), hi = *reinterpret_cast<const uint4*>(w + 16 * K);
        const uint4 lo2 = *reinterpret_cast<const uint4*>(w + other), hi2 = *reinterpret_cast<const uint4*>(w + 16 * K + other);
        mma16816<F16>(acc[j], swap ? lo2 : lo, swap ? hi2 : hi, x0);
        mma16816<F16>(acc[j], swap ? lo : lo2, swap ? hi : hi2, x1);
      }
    }
#pragma unroll
    for (int j = 0; j < G; ++j)
      if (tile + j < tiles) {
        float* r = red + (((tile + j) << lg) + part) * SC_PART + 2 * t * SC_PITCH + g;
        r[0] = acc[j][0];
        r[SC_PITCH] = acc[j][1];
        r[8] = acc[j][2];
        r[SC_PITCH + 8] = acc[j][3];
      }
  }
}

// four columns of a row of a tile, over the parts of K in their order
__device__ __forceinline__ float4 total(const float* red, int lg, int tile, int row, int q) {
  const float* r = red + (tile << lg) * SC_PART + row * SC_PITCH + q * 4;
  const int parts = 1 << lg;
  float4 v = *reinterpret_cast<const float4*>(r);
#pragma unroll
  for (int k = 1; k < 8; ++k)
    if (k < parts) {
      const float4 o = *reinterpret_cast<const float4*>(r + k * SC_PART);
      v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
    }
  return v;
}

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

template <bool F16>
__global__ void __launch_bounds__(SC_THREADS, 1)
step_cluster_kernel(DecodeState st, StepArgs a, int cl, StepClusterSmem lay) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) uint8_t sm[];
  // residual stream [8][d], twice: a sublayer reads the one and writes the other
  float* xa = reinterpret_cast<float*>(sm);
  float* xb = xa + 8 * a.d;
  uint8_t* xn = sm + lay.xn;                                         // [8] normed rows, then attention's output
  uint8_t* hs = sm + lay.hs;                                         // [8] hidden units
  uint16_t* qs = reinterpret_cast<uint16_t*>(sm + lay.q);            // [8][d]
  float* recs = reinterpret_cast<float*>(sm + lay.rec);              // [rows * heads * splits][SC_REC]
  float* red = reinterpret_cast<float*>(sm + lay.red);
  float* tokens = reinterpret_cast<float*>(sm + lay.tokens);         // embeddings [vocab][d], then the rows' examples [8][d]
  float* head = reinterpret_cast<float*>(sm + lay.head);             // the final gain [d], then the head [vocab][d]
  const uint32_t even = smem_u32(sm + lay.even), odd = smem_u32(sm + lay.odd);   // weights of QKV and gate/up, of the other two
  __shared__ __align__(16) float s_warp[SC_WARPS][SC_REC];
  __shared__ __align__(16) int s_state[8][8];                        // token, x, y, z, slot, visible keys
  __shared__ float s_dot[8][16];
  __shared__ __align__(16) float2 s_turn[8][32];                      // (cos, sin) of a row's rotary pairs
  __shared__ __align__(8) unsigned long long s_bar[2];
  const uint32_t bar_even = smem_u32(s_bar), bar_odd = bar_even + 8;
  uint32_t turn_even = 0, turn_odd = 0;
  bool ok = true;                                                    // no wait has run out
  const int rank = (int)cluster_ctarank(), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int M = a.rows, d = a.d, H = a.n_heads, T = st.t_max;
  const int xn_pitch = d * 2 + 64, hs_pitch = a.dff * 2 + 64;       // neighbouring rows on the other half of the banks
  const int items = M * H, splits = items < cl ? cl / items : 1;
  constexpr int fmt = F16 ? 1 : 0;
  const int parts_d = k_parts(d), parts_ff = k_parts(a.dff);
  const int tiles_qkv = (3 * d / 16 - rank + cl - 1) / cl, tiles_d = (d / 16 - rank + cl - 1) / cl, units_gu = (a.dff / 16 - rank + cl - 1) / cl;

  if (tid == 0) {
    mbar_init(bar_even, SC_WARPS);
    mbar_init(bar_odd, SC_WARPS);
    mbar_fence_init();
  }
  __syncthreads();
  request(Part{a.layers[0].w_qkv, d, tiles_qkv, false}, rank, cl, even, bar_even);
  for (int i = tid; i < (lay.q - lay.xn) / 16; i += SC_THREADS) reinterpret_cast<uint4*>(xn)[i] = make_uint4(0u, 0u, 0u, 0u);   // rows beyond M
  for (int i = tid; i < a.embed.vocab * d / 4; i += SC_THREADS) reinterpret_cast<float4*>(tokens)[i] = reinterpret_cast<const float4*>(a.embed.token_embed)[i];
  for (int i = tid; i < M * d / 4; i += SC_THREADS) {
    const float* ex = example_row(a.embed, i / (d / 4));
    reinterpret_cast<float4*>(tokens + a.embed.vocab * d)[i] = ex ? reinterpret_cast<const float4*>(ex)[i % (d / 4)] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (rank == 0) {
    for (int i = tid; i < d / 4; i += SC_THREADS) reinterpret_cast<float4*>(head)[i] = reinterpret_cast<const float4*>(a.head.lnf_w)[i];
    for (int i = tid; i < ARCB_VOCAB * d / 4; i += SC_THREADS) reinterpret_cast<float4*>(head + d)[i] = reinterpret_cast<const float4*>(a.head.lm_head)[i];
  }
  // row b's fed token moves the grid state; all CTAs learn what the step needs of it
  auto feed = [&](int b) {
    const int tok = st.cur_tok[b];
    grid_step(st, b, tok);
    const int slot = st.slot[b], len = st.kv_len[b];
    if (slot >= T) arcb_set_error(st.err, ARCB_DEV_BAD_INDEX);
    const int4 lo = make_int4(min(max(tok, 0), a.embed.vocab - 1), min(max(st.pos[3 * b], 0), a.max_x - 1), min(max(st.pos[3 * b + 1], 0), a.max_y - 1),
                              min(max(st.pos[3 * b + 2], 0), a.max_z - 1));
    const int4 hi = make_int4(slot < T ? slot : -1, (a.skip && a.skip[b]) || len < 0 ? 0 : min(len, T), 0, 0);
    for (int r = 0; r < cl; ++r) {
      tell(&s_state[b][0], r, lo);
      tell(&s_state[b][4], r, hi);
    }
  };
  cluster_sync_all();                            // every CTA has started before any writes to another's memory
  if (rank == 0 && tid < M) feed(tid);
  __syncwarp();
  cluster_sync_all();

  // rows of x: norm, gain, 16-bit operand; a warp a row
  auto norm = [&](const float* x, const float* gain) {
    if (warp >= M) return;
    const float* row = x + warp * d;
    constexpr int Q = STEP_CLUSTER_WIDTH / 128;
    float4 v[Q], g[Q];
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
      const int c = (lane + 32 * k) * 4;
      v[k] = c < d ? *reinterpret_cast<const float4*>(row + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      g[k] = c < d ? __ldg(reinterpret_cast<const float4*>(gain + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
      ss += (v[k].x * v[k].x + v[k].y * v[k].y) + (v[k].z * v[k].z + v[k].w * v[k].w);
    }
    const float inv = rsqrtf(warp_sum(ss) / (float)d + a.embed.eps);
#pragma unroll
    for (int k = 0; k < Q; ++k) {
      const int c = (lane + 32 * k) * 4;
      if (c < d)
        *reinterpret_cast<uint2*>(xn + warp * xn_pitch + c * 2) =
            make_uint2(pack2_act((v[k].x * inv) * g[k].x, (v[k].y * inv) * g[k].y, fmt), pack2_act((v[k].z * inv) * g[k].z, (v[k].w * inv) * g[k].w, fmt));
    }
  };
  // this part's weights have landed; nobody else's have to be waited for.  A launch gives up once, and asks for nothing more then.
  auto landed = [&](uint32_t bar, uint32_t& turn) {
    if (!ok) return;
    ok = mbar_wait_bounded(bar, turn);
    if (ok) turn ^= 1;
    else arcb_set_error(st.err, ARCB_DEV_WAIT_TIMEOUT_TMA);
  };
  // Sums of this CTA's tiles to all CTAs: a thread a destination and quad of a row.
  const int cl_bits = 31 - __clz(cl);
  auto each_quad = [&](int tiles, auto&& f) {
    int tile = 0, row = (tid >> cl_bits) >> 2;
    for (int u = tid; u < (tiles * M * 4) << cl_bits; u += SC_THREADS, row += (SC_THREADS >> cl_bits) >> 2) {
      while (row >= M) { row -= M; ++tile; }
      f(tile, row, (u >> cl_bits) & 3, u & (cl - 1));
    }
  };
  auto onto_x = [&](const float* from, float* to, int lg, const float* bias) {
    each_quad(tiles_d, [&](int tile, int row, int q, int dest) {
      const int n = (rank + tile * cl) * 16 + q * 4;
      float4 v = total(red, lg, tile, row, q);
      if (bias) {
        const float4 b = __ldg(reinterpret_cast<const float4*>(bias + n));
        v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
      }
      const float4 old = *reinterpret_cast<const float4*>(from + row * d + n);
      tell(to + row * d + n, dest, make_float4(old.x + v.x, old.y + v.y, old.z + v.z, old.w + v.w));
    });
  };

  for (int s = 0; s < a.n_steps; ++s) {
    for (int u = tid; u < M * d / 4; u += SC_THREADS) {
      const int b = u / (d / 4);
      float4 v = reinterpret_cast<const float4*>(tokens + s_state[b][0] * d)[u - b * (d / 4)];
      if (a.embed.example_ids) {
        const float4 e = reinterpret_cast<const float4*>(tokens + a.embed.vocab * d)[u];
        v.x += e.x; v.y += e.y; v.z += e.z; v.w += e.w;
      }
      reinterpret_cast<float4*>(xa)[u] = v;
    }
    if (tid < M * 32) {
      GemmEpilogue e;
      e.rope = a.rope; e.max_x = a.max_x; e.max_y = a.max_y; e.max_z = a.max_z;
      RopeRow r;
      r.x = s_state[warp][1]; r.y = s_state[warp][2]; r.z = s_state[warp][3];
      s_turn[warp][lane] = rope_cs(e, r, lane);
    }
    __syncthreads();

    for (int l = 0; l < a.n_layers; ++l) {
      const StepLayer L = a.layers[l];
      __nv_bfloat16* kc = a.cache + (size_t)l * 2 * M * H * T * ARCB_HEAD_DIM;
      __nv_bfloat16* vc = kc + (size_t)M * H * T * ARCB_HEAD_DIM;
      if (ok) request(Part{L.w_out, d, tiles_d, false}, rank, cl, odd, bar_odd);
      norm(xa, L.ln1);
      __syncthreads();
      landed(bar_even, turn_even);
      multiply<F16>(d, tiles_qkv, sm + lay.even, xn, xn_pitch, red);
      __syncthreads();
      each_quad(tiles_qkv, [&](int tile, int row, int q, int dest) {
        const int n = (rank + tile * cl) * 16 + q * 4, sec = n / d, c = n - sec * d, h = c >> 6, dim = c & 63;
        if (sec > 0 && dest) return;             // keys and values are stored once
        float4 v = total(red, parts_d, tile, row, q);
        if (sec < 2) {
          v = rotate4(v, *reinterpret_cast<const float4*>(&s_turn[row][dim >> 1]));
        }
        const int slot = s_state[row][4];
        if (sec == 0)
          tell(qs + row * d + c, dest, make_uint2(pack2_act_chk(v.x, v.y, fmt, dest ? nullptr : st.err), pack2_act_chk(v.z, v.w, fmt, dest ? nullptr : st.err)));
        else if (slot >= 0)
          *reinterpret_cast<uint2*>((sec == 1 ? kc : vc) + ((size_t)(row * H + h) * T + slot) * ARCB_HEAD_DIM + dim) =
              make_uint2(pack2_bf16(v.x, v.y), pack2_bf16(v.z, v.w));
      });
      __syncwarp();
      cluster_arrive();
      // this warp's first keys and values, but for the new row, are not waited for
      uint4 k_old[4], v_old[4];
      {
        const int item = min(rank, items * splits - 1) / splits, part = rank - item * splits, b = item / H;
        const int len = s_state[b][5], chunk = ((len + splits - 1) / splits + 15) & ~15, end = min(len, (part + 1) * chunk), fresh = s_state[b][4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int row = part * chunk + warp * 16 + u * 4 + (lane >> 3);
          k_old[u] = v_old[u] = make_uint4(0u, 0u, 0u, 0u);
          if (rank < items * splits && row < end && row != fresh) {
            k_old[u] = __ldcg(reinterpret_cast<const uint4*>(kc + ((size_t)item * T + row) * ARCB_HEAD_DIM) + (lane & 7));
            v_old[u] = __ldcg(reinterpret_cast<const uint4*>(vc + ((size_t)item * T + row) * ARCB_HEAD_DIM) + (lane & 7));
          }
        }
      }
      cluster_wait();

      // attention: a CTA an item (row, head), or a part of its keys
      if (l == 0 && rank == 0 && tid == 0) a.probe[0] = now_ns();
      for (int w = rank; w < items * splits; w += cl) {
        const int item = w / splits, part = w - item * splits, b = item / H, h = item - b * H;
        const int len = s_state[b][5], chunk = ((len + splits - 1) / splits + 15) & ~15, end = min(len, (part + 1) * chunk), fresh = s_state[b][4];
        const int sub = lane >> 3, seg = lane & 7;
        const uint4 raw = *reinterpret_cast<const uint4*>(qs + b * d + h * 64 + seg * 8);
        const float2 f0 = unpack2_act(raw.x, fmt), f1 = unpack2_act(raw.y, fmt), f2 = unpack2_act(raw.z, fmt), f3 = unpack2_act(raw.w, fmt);
        const float sc = 0.125f * LOG2E;
        const float q[8] = {f0.x * sc, f0.y * sc, f1.x * sc, f1.y * sc, f2.x * sc, f2.y * sc, f3.x * sc, f3.y * sc};
        const uint4* Kp = reinterpret_cast<const uint4*>(kc + (size_t)item * T * ARCB_HEAD_DIM) + seg;
        const uint4* Vp = reinterpret_cast<const uint4*>(vc + (size_t)item * T * ARCB_HEAD_DIM) + seg;
        float m = -INFINITY, lsum = 0.f, acc[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = 0.f;
        for (int r0 = part * chunk + warp * 16; r0 < end; r0 += SC_WARPS * 16) {
          uint4 kk[4], vv[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int row = r0 + u * 4 + sub;
            const bool old = w == rank && r0 == part * chunk + warp * 16 && row != fresh;
            kk[u] = old ? k_old[u] : make_uint4(0u, 0u, 0u, 0u);
            vv[u] = old ? v_old[u] : make_uint4(0u, 0u, 0u, 0u);
            if (row < end && !old) {
              kk[u] = __ldcg(Kp + (size_t)row * 8);
              vv[u] = __ldcg(Vp + (size_t)row * 8);
            }
          }
          float sv[4], mx = m;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float2 k0 = unpack2_bf16(kk[u].x), k1 = unpack2_bf16(kk[u].y), k2 = unpack2_bf16(kk[u].z), k3 = unpack2_bf16(kk[u].w);
            float dot = (q[0] * k0.x + q[1] * k0.y) + (q[2] * k1.x + q[3] * k1.y) + ((q[4] * k2.x + q[5] * k2.y) + (q[6] * k3.x + q[7] * k3.y));
            dot += __shfl_xor_sync(0xffffffffu, dot, 1);
            dot += __shfl_xor_sync(0xffffffffu, dot, 2);
            dot += __shfl_xor_sync(0xffffffffu, dot, 4);
            sv[u] = r0 + u * 4 + sub < end ? dot : -INFINITY;
            mx = fmaxf(mx, sv[u]);
          }
          const float safe = mx == -INFINITY ? 0.f : mx, alpha = exp2f(m - safe);
          lsum *= alpha;
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[j] *= alpha;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float p = exp2f(sv[u] - safe);
            lsum += p;
            const float2 v0 = unpack2_bf16(vv[u].x), v1 = unpack2_bf16(vv[u].y), v2 = unpack2_bf16(vv[u].z), v3 = unpack2_bf16(vv[u].w);
            acc[0] = fmaf(p, v0.x, acc[0]); acc[1] = fmaf(p, v0.y, acc[1]);
            acc[2] = fmaf(p, v1.x, acc[2]); acc[3] = fmaf(p, v1.y, acc[3]);
            acc[4] = fmaf(p, v2.x, acc[4]); acc[5] = fmaf(p, v2.y, acc[5]);
            acc[6] = fmaf(p, v3.x, acc[6]); acc[7] = fmaf(p, v3.y, acc[7]);
          }
          m = mx;
        }
#pragma unroll
        for (int o = 8; o <= 16; o <<= 1) {      // the warp's four row groups
          const float mo = __shfl_xor_sync(0xffffffffu, m, o), lo = __shfl_xor_sync(0xffffffffu, lsum, o), mx = fmaxf(m, mo);
          const float safe = mx == -INFINITY ? 0.f : mx, fa = exp2f(m - safe), fb = exp2f(mo - safe);
          lsum = lsum * fa + lo * fb;
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[j] = acc[j] * fa + __shfl_xor_sync(0xffffffffu, acc[j], o) * fb;
          m = mx;
        }
        if (sub == 0) {
          *reinterpret_cast<float4*>(s_warp[warp] + seg * 8) = make_float4(acc[0], acc[1], acc[2], acc[3]);
          *reinterpret_cast<float4*>(s_warp[warp] + seg * 8 + 4) = make_float4(acc[4], acc[5], acc[6], acc[7]);
          if (seg == 0) {
            s_warp[warp][64] = m;
            s_warp[warp][65] = lsum;
          }
        }
        __syncthreads();
        // the warps' records, merged by sixteen threads for each CTA of the cluster
        if (tid < 16 * cl) {
          const int quad = tid & 15, dest = tid >> 4;
          float mt = s_warp[0][64];
#pragma unroll
          for (int j = 1; j < SC_WARPS; ++j) mt = fmaxf(mt, s_warp[j][64]);
          const float safe = mt == -INFINITY ? 0.f : mt;
          float lt = 0.f;
          float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int j = 0; j < SC_WARPS; ++j) {
            const float f = exp2f(s_warp[j][64] - safe);
            const float4 v = *reinterpret_cast<const float4*>(s_warp[j] + quad * 4);
            lt += s_warp[j][65] * f;
            o.x += v.x * f; o.y += v.y * f; o.z += v.z * f; o.w += v.w * f;
          }
          const uint32_t rec = at_rank(smem_u32(recs + w * SC_REC), dest);
          asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(rec + quad * 16), "f"(o.x), "f"(o.y), "f"(o.z), "f"(o.w) : "memory");
          if (quad == 0) asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(rec + 256), "f"(mt), "f"(lt) : "memory");
        }
        __syncthreads();                         // before the next item's records
      }
      cluster_sync_all();
      if (l == 0 && rank == 0 && tid == 0) a.probe[1] = now_ns();
      for (int u = tid; u < items * 16; u += SC_THREADS) {
        const int item = u >> 4, quad = u & 15, b = item / H, h = item - b * H;
        const float* rec = recs + item * splits * SC_REC;
        float mt = -INFINITY, lt = 0.f;
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k0 = 0; k0 < splits; k0 += 4) {           // running merge, four records in flight
          float2 ml[4];
          float4 v[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float* p = rec + min(k0 + k, splits - 1) * SC_REC;
            ml[k] = k0 + k < splits ? *reinterpret_cast<const float2*>(p + 64) : make_float2(-INFINITY, 0.f);
            v[k] = *reinterpret_cast<const float4*>(p + quad * 4);
          }
          const float top = fmaxf(fmaxf(fmaxf(ml[0].x, ml[1].x), fmaxf(ml[2].x, ml[3].x)), mt), safe = top == -INFINITY ? 0.f : top;
          const float keep = exp2f(mt - safe);
          lt *= keep;
          o.x *= keep; o.y *= keep; o.z *= keep; o.w *= keep;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float f = exp2f(ml[k].x - safe);
            lt += ml[k].y * f;
            o.x += v[k].x * f; o.y += v[k].y * f; o.z += v[k].z * f; o.w += v[k].w * f;
          }
          mt = top;
        }
        const float inv = lt > 0.f ? 1.f / lt : 0.f;
        *reinterpret_cast<uint2*>(xn + b * xn_pitch + (h * 64 + quad * 4) * 2) =
            make_uint2(pack2_act(o.x * inv, o.y * inv, fmt), pack2_act(o.z * inv, o.w * inv, fmt));
      }
      __syncthreads();
      const Part gu{L.w_gu, d, 2 * units_gu, true};
      if (ok) request(gu, rank, cl, even, bar_even);
      landed(bar_odd, turn_odd);
      multiply<F16>(d, tiles_d, sm + lay.odd, xn, xn_pitch, red);
      __syncthreads();
      onto_x(xa, xb, parts_d, nullptr);
      __syncwarp();
      cluster_sync_all();

      if (ok) request(Part{L.w_down, a.dff, tiles_d, false}, rank, cl, odd, bar_odd);
      norm(xb, L.ln2);
      __syncthreads();
      landed(bar_even, turn_even);
      multiply<F16>(d, 2 * units_gu, sm + lay.even, xn, xn_pitch, red);
      __syncthreads();
      each_quad(units_gu, [&](int unit, int row, int q, int dest) {
        const int n = tile_row(gu, 2 * unit, rank, cl) + q * 4;
        float4 g = total(red, parts_d, 2 * unit, row, q), up = total(red, parts_d, 2 * unit + 1, row, q);
        const float4 bg = __ldg(reinterpret_cast<const float4*>(L.b_gu + n)), bu = __ldg(reinterpret_cast<const float4*>(L.b_gu + n + 64));
        g.x += bg.x; g.y += bg.y; g.z += bg.z; g.w += bg.w;
        up.x += bu.x; up.y += bu.y; up.z += bu.z; up.w += bu.w;
        const int j = (n >> 7) * 64 + (n & 127);
        int* err = dest ? nullptr : st.err;
        tell(hs + row * hs_pitch + j * 2, dest, make_uint2(pack2_act_chk(silu_f(g.x) * up.x, silu_f(g.y) * up.y, fmt, err),
                                                           pack2_act_chk(silu_f(g.z) * up.z, silu_f(g.w) * up.w, fmt, err)));
      });
      __syncwarp();
      cluster_sync_all();

      if (ok) request(Part{a.layers[l + 1 < a.n_layers ? l + 1 : 0].w_qkv, d, tiles_qkv, false}, rank, cl, even, bar_even);
      landed(bar_odd, turn_odd);
      multiply<F16>(a.dff, tiles_d, sm + lay.odd, hs, hs_pitch, red);
      __syncthreads();
      onto_x(xb, xa, parts_ff, L.b_down);
      __syncwarp();
      cluster_sync_all();
    }

    // logits of every row: sums of squares (15th) and products with the head's rows, a warp each; then the loop's bookkeeping
    if (rank == 0) {
      for (int u = warp; u < M * 15; u += SC_WARPS) {
        const int b = u / 15, v = u - b * 15;
        float sum = 0.f;
        for (int c = lane * 4; c < d; c += 128) {
          const float4 xv = *reinterpret_cast<const float4*>(xa + b * d + c);
          if (v == 14) {
            sum += (xv.x * xv.x + xv.y * xv.y) + (xv.z * xv.z + xv.w * xv.w);
          } else {
            const float4 g = *reinterpret_cast<const float4*>(head + c), w = *reinterpret_cast<const float4*>(head + d + v * d + c);
            sum += ((xv.x * g.x) * w.x + (xv.y * g.y) * w.y) + ((xv.z * g.z) * w.z + (xv.w * g.w) * w.w);
          }
        }
        sum = warp_sum(sum);
        if (lane == 0) s_dot[b][v] = sum;
      }
      __syncthreads();
      if (tid < M) {
        const float inv = rsqrtf(s_dot[tid][14] / (float)d + a.head.eps);
        float logits[ARCB_VOCAB];
#pragma unroll
        for (int v = 0; v < ARCB_VOCAB; ++v) logits[v] = s_dot[tid][v] * inv;
        head_finish(a.head, st, tid, logits);
        if (s + 1 < a.n_steps) feed(tid);
      }
    }
    __syncwarp();
    cluster_sync_all();                          // also: nobody leaves while its memory is written
  }
  landed(bar_even, turn_even);                   // the request behind the last layer
  if (!ok) {                                     // what is still on its way gets another limit each: it writes into this CTA's memory
    mbar_wait_bounded(bar_even, turn_even);
    mbar_wait_bounded(bar_odd, turn_odd);
  }
}

constexpr int SC_DEVICES = 64, SC_CLUSTER = 16;

// Whether a cluster runs on this device, at its most shared memory.
template <bool F16>
bool cluster_runs() {
  static std::mutex mu;
  static int known[SC_DEVICES];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= SC_DEVICES) return false;
  std::lock_guard<std::mutex> lock(mu);
  return asked_once(known[dev], [&](int& n) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = SC_CLUSTER;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(SC_CLUSTER);
    cfg.blockDim = dim3(SC_THREADS);
    cfg.dynamicSmemBytes = STEP_CLUSTER_SMEM_MAX;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const bool ok = cudaFuncSetAttribute(step_cluster_kernel<F16>, cudaFuncAttributeMaxDynamicSharedMemorySize, STEP_CLUSTER_SMEM_MAX) == cudaSuccess &&
                    cudaFuncSetAttribute(step_cluster_kernel<F16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&n, step_cluster_kernel<F16>, &cfg) == cudaSuccess;
    if (!ok) cudaGetLastError();
    return ok;
  }) > 0;
}

}  // namespace

int arcb_step_cluster(int rows, int d, int dff, int n_layers, int t_max) {
  return step_cluster_fits(rows, d, dff, n_layers, t_max, SC_CLUSTER) && cluster_runs<true>() && cluster_runs<false>() ? SC_CLUSTER : 0;
}

int arcb_launch_step_cluster(const DecodeState& st, const StepArgs& a, int cluster, cudaStream_t stream) {
  const StepClusterSmem lay = step_cluster_smem(a.rows, a.d, a.dff, a.n_heads, cluster);
  const cudaError_t e = arcb_launch_cluster(a.embed.act_f16 ? step_cluster_kernel<true> : step_cluster_kernel<false>, cluster, dim3(cluster), dim3(SC_THREADS),
                                            lay.total, stream, st, a, cluster, lay);
  arcb_count_launch(1);
  return (int)e;
}
