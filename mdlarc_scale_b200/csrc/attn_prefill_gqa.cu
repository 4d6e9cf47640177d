// Causal prefill attention of grouped heads on tcgen05 tensor cores with TMEM accumulators, reading keys and
// values straight from the cache (so a portion of a prompt sees what earlier portions left there).
//
// An item = up to 256 consecutive query rows of one sequence (two 128-row Q tiles, A and B) x one query head.
// One CTA an SM takes items from a common counter, a block's heads one after the other (a group's heads share its keys
// in L2): an item alone is a chain of block description, Q and K, scores, softmax, P V, denominators, store, of which most
// is waiting.  Here the producer describes and fetches the next item while this one is worked on, and its first
// scores are computed behind this one's last product.  B200, us a launch, an item a CTA / this: 150 prompts of about 400
// tokens, 16 heads of 128 658 / 556; 48 of about 900, 20 latent heads 199 / 167; 8 of 900 to 1024, 16 latent heads of 128 + 64 172 / 161.
// With 128 value columns in one product a step, 64-byte moves of gates and results and products issued by a warp
// 416 / 139 / 123: what bounds it is the chain of a tile (scores, softmax, P, P V, the next scores) beside 2048 cycles of
// exponentials for a pair of tiles.
// Warps 0-3 are helpers (TMA producer, MMA issuer of A, MMA issuer of B, one idle); warps 4-11 serve tile A
// and warps 12-19 tile B, two threads per query row: thread `half` owns keys [64 half, 64 half + 64) of every
// 128-key tile and half of the output dims.  Per key tile j and Q tile x:
//   TMA        K and V tiles as 128 x 64 boxes, 128-byte swizzle, rings shared by A and B
//   MMA        S_x = Q_x K^T, fp32 in 128 TMEM columns
//   softmax_x  scores to registers; reference maximum (raised only when exceeded by 2^8, O rescaled then);
//              p = exp2(s c - m) in fp32, row sums in fp32; P rounded to the operand format and written over
//              the thread's own score columns
//   MMA        O_x += P_x V (A = P from TMEM), then at once S_x of the next tile
// Both products of a tile are issued by one thread in this order, so S(j + 1) cannot overtake the read of P(j)
// it overwrites, and its completion implies that O(j) is complete.  While one Q tile is in the tensor core the
// other tile's threads do exponentials.  A sink only joins the denominator at the end: rows are normalised by
// l 2^m + 2^(sink log2 e).  The output gate multiplies the normalised row.  Every wait is bounded.
//
// A window hides keys from below: key tiles start at the first key the block's first row sees, and tile B skips
// the tiles that lie ahead of its own first key.  With DR > 0 keys and values are those expanded from cached
// latents: the first DP key columns and the values come from the expansion scratch, the last DR key columns,
// which all heads share, from the latent cache itself.
#include <type_traits>

#include "attn_prefill_gqa.cuh"
#include "flash_common.cuh"
#include "gemm.cuh"
#include "launch.cuh"

using namespace sm100;

namespace {

constexpr int BQ = 128, BKV = 128;
constexpr int THREADS = 640;
constexpr float LOG2E = 1.4426950408889634f;
constexpr float RESCALE_THRESHOLD = 8.f;   // log2 units
constexpr int BOX_BYTES = 128 * 64 * 2;    // one 128-row x 64-column box

// What the producer works out about an item; rows < 0: the list has ended.
struct FgItem { int row0, rows, n_a, n_b, key0, j0_b, head, kv_row, rot_row, pad; };
constexpr int ITEM_SLOTS = 4;

template <int DP, int DR, int VP>
struct FgCfg {
  static constexpr int QB = (DP + DR) / 64;  // boxes of a query (key) row
  static constexpr int Q_BYTES = QB * BOX_BYTES;
  static constexpr int K_BYTES = Q_BYTES;
  static constexpr int V_BYTES = (VP / 64) * BOX_BYTES;
  static constexpr int AVAIL = (DR > 0 ? 224 : 208) * 1024 - 2 * Q_BYTES;
  static constexpr int FIT = AVAIL / (K_BYTES + V_BYTES);
  static constexpr int V_STAGES = FIT > 4 ? 4 : FIT;
  // one more key tile where it fits: the next tile's scores then do not wait for this tile's values
  static constexpr int K_STAGES = V_STAGES < 4 && AVAIL >= (V_STAGES + 1) * K_BYTES + V_STAGES * V_BYTES ? V_STAGES + 1 : V_STAGES;
  static_assert(V_STAGES >= 1, "a key tile and a value tile must fit");
  static constexpr int TILES = 2 * Q_BYTES + K_STAGES * K_BYTES + V_STAGES * V_BYTES;
  // Behind the tiles: barriers, descriptions of items, and what the two threads of a row exchange.  DR = 0: 1 KB of
  // alignment slack, exchange in fp32.  DR > 0 has no room for either: no static shared memory (the dynamic part then starts
  // aligned, which is checked), maxima exchanged as bfloat16, denominators in two halves.
  static constexpr int BAR_BYTES = 384;
  static constexpr int XCHG_BYTES = 2 * 2 * 2 * BQ * (DR > 0 ? 2 : 4);
  static constexpr int SMEM = TILES + BAR_BYTES + ITEM_SLOTS * (int)sizeof(FgItem) + XCHG_BYTES + (DR > 0 ? 0 : 1024);
  static_assert(SMEM <= 227 * 1024, "shared memory of one CTA");
  // S_A [0,128) S_B [128,256) O_A [256,256+VP) O_B; P_x of key half y occupies columns [64 y, 64 y + 32) of S_x
  static constexpr int TMEM_COLS = 512;
};

template <int DP, int DR, int VP, bool F16>
__global__ void __launch_bounds__(THREADS, 1)
attn_prefill_gqa_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                        const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_r,
                        AttnPrefillGqaArgs a, uint32_t idesc_qk, uint32_t idesc_pv) {
  using C = FgCfg<DP, DR, VP>;
  pdl_launch_dependents();
  pdl_wait();   // the prologue below already reads the work list from global memory
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  using XT = typename std::conditional<(DR > 0), uint16_t, float>::type;
  if constexpr (DR > 0) {
    if (smem_u32(smem_raw) & 1023u) {
      if (threadIdx.x == 0) arcb_set_error(a.err, ARCB_DEV_BAD_INDEX);
      return;
    }
  }
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  const uint32_t q_smem = base;
  const uint32_t k_smem = base + 2 * C::Q_BYTES;
  const uint32_t v_smem = k_smem + C::K_STAGES * C::K_BYTES;
  const uint32_t bar0 = base + C::TILES;
  const uint32_t b_full = bar0, b_empty = b_full + 8 * ITEM_SLOTS,                 // descriptions of items
                 b_q = b_empty + 8 * ITEM_SLOTS, b_qfree = b_q + 16,               // Q tile A, B
                 b_kfull = b_qfree + 16, b_kempty = b_kfull + 8 * C::K_STAGES, b_vfull = b_kempty + 8 * C::K_STAGES,
                 b_vempty = b_vfull + 8 * C::V_STAGES, b_s = b_vempty + 8 * C::V_STAGES,
                 b_p = b_s + 16, b_o = b_p + 16, b_x = b_o + 16;     // b_x: 8 barriers, one per pair of warps of a row
  static_assert(16 * ITEM_SLOTS + 32 + 16 * (C::K_STAGES + C::V_STAGES) + 48 + 64 <= C::BAR_BYTES - 8, "barriers");
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(base_ptr + C::TILES + C::BAR_BYTES - 8);
  FgItem* s_item = reinterpret_cast<FgItem*>(base_ptr + C::TILES + C::BAR_BYTES);
  XT (*s_xchg)[2][2][BQ] =                // [parity of the exchange][Q tile][half][row]
      reinterpret_cast<XT (*)[2][2][BQ]>(base_ptr + C::TILES + C::BAR_BYTES + ITEM_SLOTS * sizeof(FgItem));

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // known to be the same in a warp
  const int wg = (warp >> 2) - 1;
  const int grp = wg >> 1;
  const int half = wg & 1;
  const int quarter = warp & 3;
  const int r = quarter * 32 + lane;
  if (threadIdx.x == 0) {
    for (int s = 0; s < ITEM_SLOTS; ++s) {
      mbar_init(b_full + 8 * s, 1);
      mbar_init(b_empty + 8 * s, 18);     // two issuers, sixteen softmax warps
    }
    for (int s = 0; s < C::K_STAGES; ++s) {
      mbar_init(b_kfull + 8 * s, 1);
      mbar_init(b_kempty + 8 * s, 2);
    }
    for (int s = 0; s < C::V_STAGES; ++s) {
      mbar_init(b_vfull + 8 * s, 1);
      mbar_init(b_vempty + 8 * s, 2);
    }
    for (int x = 0; x < 2; ++x) {
      mbar_init(b_q + 8 * x, 1);
      mbar_init(b_qfree + 8 * x, 1);
      mbar_init(b_s + 8 * x, 1);
      mbar_init(b_p + 8 * x, 256);
      mbar_init(b_o + 8 * x, 1);
    }
    for (int i = 0; i < 8; ++i) mbar_init(b_x + 8 * i, 64);
    mbar_fence_init();
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    if (DR > 0) tma_prefetch_desc(&tmap_r);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  if (warp < 4) {
    reg_dealloc_32();
    if (warp == 0) {
      // ---- TMA producer: the whole warp, lane 0 issues ----
      const int total = a.n_qblocks * a.n_heads;
      auto wait = [&](uint32_t bar, uint32_t parity) -> bool {
        const bool good = __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity));
        if (!good && lane == 0) arcb_set_error(a.err, ARCB_DEV_WAIT_TIMEOUT_MMA);
        return good;
      };
      // description k of this CTA
      auto describe = [&](int k, int item) -> bool {
        FgItem it{};
        it.rows = -1;
        if (item < total) {
          const int blk = item / a.n_heads;
          it.head = item - blk * a.n_heads;
          it.row0 = a.qblock_row0[blk];
          it.rows = a.qblock_rows[blk];           // 1..256
          const int seq = a.seq[it.row0];
          const bool seq_ok = seq >= 0 && seq < a.n_seqs;
          int first[2] = {0, 0}, most[2] = {0, 0};  // of tiles A and B: the first row's visible keys, and the most
          if (seq_ok) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int cnt = i * 32 + lane < it.rows ? a.kv_count[it.row0 + i * 32 + lane] : 0;
              if (i % 4 == 0) first[i >> 2] = __shfl_sync(0xffffffffu, cnt, 0);
              if (cnt <= a.t_max) most[i >> 2] = max(most[i >> 2], cnt);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
              most[0] = max(most[0], __shfl_xor_sync(0xffffffffu, most[0], o));
              most[1] = max(most[1], __shfl_xor_sync(0xffffffffu, most[1], o));
            }
          } else if (lane == 0) {
            arcb_set_error(a.err, ARCB_DEV_BAD_INDEX);
          }
          // first key tile, and the first one tile B reads (rows of a block are consecutive positions)
          it.key0 = a.window > 0 ? max(0, first[0] - a.window) : 0;
          it.j0_b = a.window > 0 && it.rows > BQ ? max(0, max(0, first[1] - a.window) - it.key0) / BKV : 0;
          it.n_a = (max(most[0] - it.key0, 0) + BKV - 1) / BKV;
          it.n_b = (max(most[1] - it.key0, 0) + BKV - 1) / BKV;
          it.kv_row = DR > 0 ? a.kv0[blk] + it.key0 : (seq * a.n_kv + it.head / (a.n_heads / a.n_kv)) * a.t_max + it.key0;
          it.rot_row = DR > 0 ? (seq * a.rot_panels + a.rot_panel) * a.t_max + it.key0 : 0;
        }
        const int slot = k % ITEM_SLOTS;
        if (!wait(b_empty + 8 * slot, ((k / ITEM_SLOTS) & 1) ^ 1)) return false;
        if (lane == 0) {
          s_item[slot] = it;
          mbar_arrive(b_full + 8 * slot);
        }
        __syncwarp();
        return true;
      };
      int item = blockIdx.x, tile = 0, used[2] = {0, 0};   // key tiles and Q tiles of all items so far
      bool ok = describe(0, item);
      for (int k = 0; ok && item < total; ++k) {
        int next = 0;
        if (lane == 0) {
          next = atomicAdd(a.next, 1);
          // `total` fetches a launch (every CTA's last one finds nothing): the last of them leaves the counter as it was
          if (next == total - 1) *a.next = 0;
        }
        const FgItem* it = s_item + k % ITEM_SLOTS;
        const int n_tiles = max(it->n_a, it->n_b), ahead = min(n_tiles, 2);
        auto load_q = [&](int x) -> bool {
          if (x ? it->n_b <= it->j0_b : it->n_a <= 0) return true;
          if (!wait(b_qfree + 8 * x, (used[x] & 1) ^ 1)) return false;
          ++used[x];
          if (lane == 0) {
            mbar_expect_tx(b_q + 8 * x, C::Q_BYTES);
#pragma unroll
            for (int c = 0; c < C::QB; ++c)
              tma_load_2d(q_smem + x * C::Q_BYTES + c * BOX_BYTES, &tmap_q, a.q_col + it->head * (DP + DR) + c * 64, it->row0 + x * BQ, b_q + 8 * x);
          }
          return true;
        };
        for (int j = 0;; ++j) {
          // the next item, once this one's first tiles are on their way
          if (j == ahead) {
            item = __shfl_sync(0xffffffffu, next, 0) + (int)gridDim.x;
            ok = describe(k + 1, item);
          }
          if (!ok || j >= n_tiles) break;
          const int s = tile % C::K_STAGES, t = tile % C::V_STAGES;
          if (j == 0) ok = load_q(0);
          ok = ok && wait(b_kempty + 8 * s, ((tile / C::K_STAGES) & 1) ^ 1);
          if (!ok) break;
          if (lane == 0) {
            const uint32_t dst = k_smem + s * C::K_BYTES;
            const int k_col = DR > 0 ? it->head * DP : 0;
            mbar_expect_tx(b_kfull + 8 * s, C::K_BYTES);
#pragma unroll
            for (int c = 0; c < DP / 64; ++c) tma_load_2d(dst + c * BOX_BYTES, &tmap_k, k_col + c * 64, it->kv_row + j * BKV, b_kfull + 8 * s);
#pragma unroll
            for (int c = 0; c < DR / 64; ++c)
              tma_load_2d(dst + (DP / 64 + c) * BOX_BYTES, &tmap_r, 0, it->rot_row + c * a.t_max + j * BKV, b_kfull + 8 * s);
          }
          if (j == 0) ok = load_q(1);
          ok = ok && wait(b_vempty + 8 * t, ((tile / C::V_STAGES) & 1) ^ 1);
          if (!ok) break;
          if (lane == 0) {
            const int v_col = DR > 0 ? a.v_col + it->head * VP : 0;
            mbar_expect_tx(b_vfull + 8 * t, C::V_BYTES);
#pragma unroll
            for (int c = 0; c < VP / 64; ++c)
              tma_load_2d(v_smem + t * C::V_BYTES + c * BOX_BYTES, &tmap_v, v_col + c * 64, it->kv_row + j * BKV, b_vfull + 8 * t);
          }
          ++tile;
        }
      }
    } else if (warp == 1 || warp == 2) {
      // ---- MMA issuer of Q tile x: the whole warp runs this with one elected lane, so that operands stay in uniform
      // registers.  One thread alone needed about 1000 cycles to issue 8 products and their commits: 502 / 170 / 158 us a
      // launch of the three above, against 416 / 139 / 123.
      const int x = warp - 1;
      const uint32_t el = elect_one();
      bool ok = true;
      auto wait_or_flag = [&](uint32_t bar, uint32_t parity, int code) {
        if (ok && !__all_sync(0xffffffffu, mbar_wait_bounded(bar, parity))) {
          arcb_set_error(a.err, code);
          ok = false;
        }
      };
      const uint32_t t_s = tmem_base + x * 128, t_o = tmem_base + 256 + x * VP;
      int tile = 0, done = 0, used = 0;    // of the items before: key tiles, this Q tile's products, items that had this Q tile
      for (int k = 0;; ++k) {
        const int slot = k % ITEM_SLOTS;
        wait_or_flag(b_full + 8 * slot, (k / ITEM_SLOTS) & 1, ARCB_DEV_WAIT_TIMEOUT_TMA);
        if (!ok) break;
        auto field = [&](int v) { return __shfl_sync(0xffffffffu, v, 0); };
        const int rows = field(s_item[slot].rows), n_a = field(s_item[slot].n_a), n_b = field(s_item[slot].n_b), j0_b = field(s_item[slot].j0_b);
        if (rows < 0) break;
        const int n_x = x ? n_b : n_a, n_tiles = max(n_a, n_b), j0 = x ? j0_b : 0;
        if (el) mbar_arrive(b_empty + 8 * slot);
        auto k_stage = [&](int j) { return (tile + j) % C::K_STAGES; };
        auto v_stage = [&](int j) { return (tile + j) % C::V_STAGES; };
        auto mma_s = [&](int j) {
          const uint32_t kst = k_smem + k_stage(j) * C::K_BYTES;
#pragma unroll
          for (int c = 0; c < C::QB; ++c) {
            const uint64_t dq = umma_desc_k_sw128(q_smem + x * C::Q_BYTES + c * BOX_BYTES);
            const uint64_t dk = umma_desc_k_sw128(kst + c * BOX_BYTES);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) umma_f16_if(el, t_s, dq + 2 * ks, dk + 2 * ks, idesc_qk, (c | ks) ? 1u : 0u);
          }
          umma_commit_if(el, b_s + 8 * x);
          umma_commit_if(el, b_kempty + 8 * k_stage(j));
          if (j == n_x - 1) umma_commit_if(el, b_qfree + 8 * x);
        };
        auto mma_o = [&](int j) {
          const uint32_t vst = v_smem + v_stage(j) * C::V_BYTES;
          const uint64_t dv = umma_desc_mn_sw128(vst, BOX_BYTES);
#pragma unroll
          for (int ks = 0; ks < BKV / 16; ++ks)
            umma_f16_ts_if(el, t_o, t_s + (ks >> 2) * 64 + (ks & 3) * 8, dv + (uint64_t)(ks * (2048 >> 4)), idesc_pv, (j > j0 || ks) ? 1u : 0u);
          umma_commit_if(el, b_vempty + 8 * v_stage(j));
        };
        auto wait_v = [&](int j) { wait_or_flag(b_vfull + 8 * v_stage(j), ((tile + j) / C::V_STAGES) & 1, ARCB_DEV_WAIT_TIMEOUT_TMA); };
        auto wait_k = [&](int j) { wait_or_flag(b_kfull + 8 * k_stage(j), ((tile + j) / C::K_STAGES) & 1, ARCB_DEV_WAIT_TIMEOUT_TMA); };
        // stages only the other tile uses: give them back in order as they land
        auto pass = [&](int from, int to) {
          for (int j = from; ok && j < to; ++j) {
            wait_k(j);
            if (ok && el) mbar_arrive(b_kempty + 8 * k_stage(j));
            wait_v(j);
            if (ok && el) mbar_arrive(b_vempty + 8 * v_stage(j));
          }
        };
        if (n_x > j0) {
          pass(0, j0);
          wait_or_flag(b_q + 8 * x, used & 1, ARCB_DEV_WAIT_TIMEOUT_TMA);
          // scores j, behind probabilities j - 1 times values (which they overwrite)
          for (int j = j0; ok && j <= n_x; ++j) {
            if (j > j0) {
              wait_or_flag(b_p + 8 * x, (done + j - 1 - j0) & 1, ARCB_DEV_WAIT_TIMEOUT_ACC);
              wait_v(j - 1);
              if (!ok) break;
              tc_fence_after();
              mma_o(j - 1);
            }
            if (j == n_x) break;
            wait_k(j);
            if (!ok) break;
            tc_fence_after();
            mma_s(j);
          }
          if (ok) umma_commit_if(el, b_o + 8 * x);
          pass(n_x, n_tiles);
          done += n_x - j0;
          ++used;
        } else {
          pass(0, n_tiles);
        }
        if (!ok) break;
        tile += n_tiles;
      }
    }
  } else {
    reg_alloc_112();
    // ---- softmax / output threads: row r of Q tile grp, key half `half` ----
    const uint32_t t_lane = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t t_s = t_lane + grp * 128 + half * 64;
    const uint32_t t_o = t_lane + 256 + grp * VP + half * (VP / 2);
    const uint32_t xbar = b_x + 8 * (grp * 4 + quarter);
    const float sc = a.scale * LOG2E;
    const int qr = grp * BQ + r;
    bool ok = true;
    uint32_t xphase = 0;
    // hands `mine` to the row's other thread; consecutive exchanges use the buffer's two parts in turn
    auto swap = [&](XT mine, XT& theirs) -> bool {
      s_xchg[xphase][grp][half][r] = mine;
      tc_fence_before();
      mbar_arrive(xbar);
      const bool good = mbar_wait_bounded(xbar, xphase);
      tc_fence_after();
      theirs = s_xchg[xphase][grp][half ^ 1][r];
      xphase ^= 1u;
      return good;
    };
    // maxima: as bfloat16 both sides go on with the rounded values
    auto exchange_max = [&](float& mine, float& theirs) -> bool {
      if constexpr (DR > 0) {
        const __nv_bfloat16 sent = (__nv_bfloat16)mine;
        mine = (float)sent;
        uint16_t got;
        const bool good = swap(__bfloat16_as_ushort(sent), got);
        theirs = (float)__ushort_as_bfloat16(got);
        return good;
      } else {
        return swap(mine, theirs);
      }
    };
    // all 32 bits
    auto exchange_sum = [&](float mine, float& theirs) -> bool {
      if constexpr (DR > 0) {
        uint16_t hi, lo;
        bool good = swap((uint16_t)(__float_as_uint(mine) >> 16), hi);
        good = swap((uint16_t)(__float_as_uint(mine) & 0xffffu), lo) && good;
        theirs = __uint_as_float((uint32_t)hi << 16 | lo);
        return good;
      } else {
        return swap(mine, theirs);
      }
    };
    // waits for description k and requests its row's visible keys
    auto await_item = [&](int k, int& cnt) {
      const int slot = k % ITEM_SLOTS;
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(b_full + 8 * slot, (k / ITEM_SLOTS) & 1))) {
        arcb_set_error(a.err, ARCB_DEV_WAIT_TIMEOUT_TMA);
        ok = false;
        return;
      }
      cnt = qr < s_item[slot].rows ? a.kv_count[s_item[slot].row0 + qr] : 0;
    };
    int done = 0, used = 0, cnt = 0;       // of the items before: key tiles, and items with rows here; this item's visible keys
    await_item(0, cnt);
    for (int k = 0; ok; ++k) {
    const FgItem& it = s_item[k % ITEM_SLOTS];
    const int row0 = it.row0, n_rows = it.rows, h = it.head, key0 = it.key0, n_mine = grp ? it.n_b : it.n_a, j0 = grp ? it.j0_b : 0;
    if (n_rows < 0) break;
    __syncwarp();
    if (lane == 0) mbar_arrive(b_empty + 8 * (k % ITEM_SLOTS));
    const int my_cnt = cnt > a.t_max ? 0 : cnt;
    const int my_lo = a.window > 0 ? max(0, my_cnt - a.window) : 0;
    float m_ref = -INFINITY, l = 0.f;
    for (int j = j0; j < n_mine; ++j) {
      if (ok && !mbar_wait_bounded(b_s + 8 * grp, (done + j - j0) & 1)) {
        arcb_set_error(a.err, ARCB_DEV_WAIT_TIMEOUT_ACC);
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const int tile_key = key0 + j * BKV + half * 64;            // visible: [v_lo, v_hi) of the thread's 64 keys
      const int v_hi = my_cnt - tile_key, v_lo = my_lo - tile_key;
      const bool full = __all_sync(0xffffffffu, v_hi >= 64 && v_lo <= 0);
      // 32 of the thread's 64 scores; hidden keys become -inf, whose exp2 is exactly 0
      auto load_scores = [&](int c, uint32_t (&sv)[32]) {
        tmem_ld_32x32(t_s + c * 32, sv);
        tmem_wait_ld_dep(sv);
        if (!full) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i >= v_hi || c * 32 + i < v_lo) sv[i] = 0xff800000u;
        }
      };
      // the scores are read twice (maximum, then exponentials): tensor memory is quicker to read again than
      // 64 registers are to hold
      float raw_mx = -INFINITY;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t sv[32];
        load_scores(c, sv);
        float mx2 = fmaxf(__uint_as_float(sv[0]), __uint_as_float(sv[1]));
#pragma unroll
        for (int i = 2; i < 32; i += 2) mx2 = max3_f32(mx2, __uint_as_float(sv[i]), __uint_as_float(sv[i + 1]));
        raw_mx = fmaxf(raw_mx, mx2);
      }
      float mine = raw_mx == -INFINITY ? -INFINITY : raw_mx * sc;
      float other;
      bool good = exchange_max(mine, other);
      if (!good) arcb_set_error(a.err, ARCB_DEV_WAIT_TIMEOUT_ACC);
      ok = __all_sync(0xffffffffu, good);
      if (!ok) break;
      const float mx = fmaxf(mine, other);
      float alpha = 1.f;
      if (mx > m_ref + RESCALE_THRESHOLD) {  // also the first visible tile (m_ref = -inf)
        alpha = (m_ref == -INFINITY) ? 0.f : ex2_fast(m_ref - mx);
        m_ref = mx;
      }
      l *= alpha;
      const float m_safe = (m_ref == -INFINITY) ? 0.f : m_ref;
      const uint64_t sc2 = pack_f32x2(sc, sc), nm2 = pack_f32x2(-m_safe, -m_safe);
      if (j > j0 && __any_sync(0xffffffffu, alpha != 1.f)) {
        // S(j) was issued after P V(j - 1): O is complete and may be rescaled
#pragma unroll
        for (int c = 0; c < VP / 64; ++c) {
          uint32_t oreg[32];
          tmem_ld_32x32(t_o + c * 32, oreg);
          tmem_wait_ld_dep(oreg);
#pragma unroll
          for (int i = 0; i < 32; ++i) oreg[i] = __float_as_uint(__uint_as_float(oreg[i]) * alpha);
          tmem_st_32x32(t_o + c * 32, oreg);
        }
      }
      float ls0 = 0.f, ls1 = 0.f;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t sv[32];
        load_scores(c, sv);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          uint32_t pr[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            float t0, t1;
            shift2_f32(sv[g * 16 + 2 * e], sv[g * 16 + 2 * e + 1], sc2, nm2, t0, t1);
            t0 = ex2_fast(t0);
            t1 = ex2_fast(t1);
            ls0 += t0;
            ls1 += t1;
            pr[e] = pack2_prob(t0, t1, F16 ? 1 : 0);
          }
          tmem_st_32x8(t_s + (c * 2 + g) * 8, pr);   // over scores this thread has already read
        }
      }
      l += ls0 + ls1;
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(b_p + 8 * grp);
    }
    // the next item's description has been there for long; this one's gates travel while its last product runs
    int next_cnt = 0;
    if (ok) await_item(k + 1, next_cnt);
    // Rows lie far apart: a quad of lanes moves 64 consecutive bytes of each of its four rows (lane q piece q), not
    // every lane 16 bytes of its own (32 lines an access).
    const int piece = lane & 3, quad_row = qr - piece;
    uint16_t* dst = reinterpret_cast<uint16_t*>(a.out) + (((size_t)row0 + quad_row) * a.n_heads + h) * VP + half * (VP / 2) + piece * 8;
    const uint16_t* gt = reinterpret_cast<const uint16_t*>(a.gate) + ((size_t)row0 + quad_row) * a.gate_pitch + (size_t)h * VP + half * (VP / 2) + piece * 8;
    uint4 gates[4];
    auto load_gates = [&](int c) {
      if (a.gate)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          gates[i] = quad_row + i < n_rows ? __ldg(reinterpret_cast<const uint4*>(gt + i * a.gate_pitch + c * 32)) : make_uint4(0u, 0u, 0u, 0u);
    };
    load_gates(0);
    float l_other = 0.f;
    if (ok && n_mine > j0) {
      bool good = exchange_sum(l, l_other);
      good = mbar_wait_bounded(b_o + 8 * grp, used & 1) && good;
      if (!good) arcb_set_error(a.err, ARCB_DEV_WAIT_TIMEOUT_ACC);
      ok = __all_sync(0xffffffffu, good);
    }
    float l_row = half ? l_other + l : l + l_other;   // same order of addition in both threads
    float num = 1.f;
    if (a.sink && m_ref > -INFINITY) {
      const float d = __ldg(a.sink + h) * LOG2E - m_ref;
      if (d > 0.f) {      // bring both terms to the larger reference
        num = exp2f(-d);
        l_row = l_row * num + 1.f;
      } else {
        l_row += exp2f(d);
      }
    }
    const float inv = (ok && l_row > 0.f) ? num / l_row : 0.f;
#pragma unroll
    for (int c = 0; c < VP / 64; ++c) {
      if (c > 0) load_gates(c);
      if (a.gate) quad_transpose(gates, lane);
      uint32_t oreg[32];
      if (ok && n_mine > j0) {
        tc_fence_after();
        tmem_ld_32x32(t_o + c * 32, oreg);
        tmem_wait_ld_dep(oreg);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) oreg[i] = 0u;
      }
      uint4 res[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(oreg[i * 8 + e]) * inv;
        if (a.gate) {
          const uint32_t gw[4] = {gates[i].x, gates[i].y, gates[i].z, gates[i].w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 g2 = unpack2_act(gw[e], F16 ? 1 : 0);
            f[2 * e] *= g2.x;
            f[2 * e + 1] *= g2.y;
          }
        }
        res[i] = make_uint4(pack2_act(f[0], f[1], F16 ? 1 : 0), pack2_act(f[2], f[3], F16 ? 1 : 0),
                            pack2_act(f[4], f[5], F16 ? 1 : 0), pack2_act(f[6], f[7], F16 ? 1 : 0));
      }
      quad_transpose(res, lane);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (quad_row + i < n_rows) *reinterpret_cast<uint4*>(dst + (size_t)i * a.n_heads * VP + c * 32) = res[i];
    }
    if (n_mine > j0) {
      done += n_mine - j0;
      ++used;
    }
    cnt = next_cnt;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

template <int DP, int DR, int VP>
cudaError_t set_attr() {
  cudaError_t e = cudaFuncSetAttribute(attn_prefill_gqa_kernel<DP, DR, VP, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, FgCfg<DP, DR, VP>::SMEM);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(attn_prefill_gqa_kernel<DP, DR, VP, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, FgCfg<DP, DR, VP>::SMEM);
}

template <int DP, int DR, int VP>
int launch(const AttnPrefillGqaArgs& a, cudaStream_t stream) {
  using C = FgCfg<DP, DR, VP>;
  CUtensorMap tq, tk, tv;
  const uint64_t cache_rows = (uint64_t)a.n_seqs * a.n_kv * a.t_max;
  const uint64_t kv_rows = DR > 0 ? (uint64_t)a.kv_rows : cache_rows;
  int r = arcb_make_tmap_2d_16b(&tq, a.q, (uint64_t)a.n_rows, (uint64_t)a.q_pitch, BQ, 64, a.act_f16);
  if (r) return 1000 + r;
  r = arcb_make_tmap_2d_16b(&tk, a.k, kv_rows, DR > 0 ? (uint64_t)a.kv_pitch : DP, BKV, 64, a.act_f16);
  if (r) return 1000 + r;
  r = arcb_make_tmap_2d_16b(&tv, a.v, kv_rows, DR > 0 ? (uint64_t)a.kv_pitch : VP, BKV, 64, a.act_f16);
  if (r) return 1000 + r;
  CUtensorMap tr = tk;
  if (DR > 0) {
    r = arcb_make_tmap_2d_16b(&tr, a.k_rot, (uint64_t)a.n_seqs * a.rot_panels * a.t_max, 64, BKV, 64, a.act_f16);
    if (r) return 1000 + r;
  }
  const int fmt = a.act_f16 ? 0 : 1;
  const uint32_t idesc_qk = umma_idesc_f16(BQ, BKV, fmt, fmt, 0, 0);
  const uint32_t idesc_pv = umma_idesc_f16(BQ, VP, fmt, fmt, 0, 1);   // V is MN-major
  const long long items = (long long)a.n_heads * a.n_qblocks;
  if (items > 0x7fffffffll - 1024) return -1;
  const dim3 grid((unsigned)(items < arcb_num_sms() ? items : arcb_num_sms()));
  const cudaError_t e =
      a.act_f16 ? arcb_launch(attn_prefill_gqa_kernel<DP, DR, VP, true>, grid, dim3(THREADS), C::SMEM, stream, tq, tk, tv, tr, a, idesc_qk, idesc_pv)
                : arcb_launch(attn_prefill_gqa_kernel<DP, DR, VP, false>, grid, dim3(THREADS), C::SMEM, stream, tq, tk, tv, tr, a, idesc_qk, idesc_pv);
  arcb_count_launch(1);
  return (int)e;
}

}  // namespace

bool arcb_attn_prefill_gqa_supported(int dimp, int vdimp, int n_seqs, int n_kv, int t_max, float scale) {
  // the reference maximum follows the largest raw score, which needs a positive scale
  return scale > 0.f && dimp <= 128 && vdimp <= 128 && (long long)n_seqs * n_kv * t_max < (1ll << 31) - 256;
}

bool arcb_attn_prefill_latent_supported(int dimp, int rotp, int vdimp, int panels, int n_seqs, int t_max, float scale) {
  return scale > 0.f && dimp <= 128 && rotp == 64 && vdimp <= 128 && (long long)n_seqs * panels * t_max < (1ll << 31) - 256;
}

int arcb_attn_prefill_gqa_init() {
  cudaError_t e;
  if ((e = set_attr<64, 0, 64>()) != cudaSuccess) return (int)e;
  if ((e = set_attr<64, 0, 128>()) != cudaSuccess) return (int)e;
  if ((e = set_attr<128, 0, 64>()) != cudaSuccess) return (int)e;
  if ((e = set_attr<128, 0, 128>()) != cudaSuccess) return (int)e;
  if ((e = set_attr<64, 64, 64>()) != cudaSuccess) return (int)e;
  if ((e = set_attr<64, 64, 128>()) != cudaSuccess) return (int)e;
  if ((e = set_attr<128, 64, 64>()) != cudaSuccess) return (int)e;
  if ((e = set_attr<128, 64, 128>()) != cudaSuccess) return (int)e;
  return 0;
}

int arcb_launch_attn_prefill_gqa(const AttnPrefillGqaArgs& a, cudaStream_t stream) {
  if (a.n_qblocks <= 0) return 0;
  if (a.n_rows <= 0 || a.n_kv <= 0 || a.n_heads % a.n_kv || a.n_qblocks > 65535 || !a.next) return -1;
  if (a.kv0) {
    if (a.rotp != 64) return -1;
    switch (a.dimp * 1000 + a.vdimp) {
      case 64064: return launch<64, 64, 64>(a, stream);
      case 64128: return launch<64, 64, 128>(a, stream);
      case 128064: return launch<128, 64, 64>(a, stream);
      case 128128: return launch<128, 64, 128>(a, stream);
    }
    return -1;
  }
  switch (a.dimp * 1000 + a.vdimp) {
    case 64064: return launch<64, 0, 64>(a, stream);
    case 64128: return launch<64, 0, 128>(a, stream);
    case 128064: return launch<128, 0, 64>(a, stream);
    case 128128: return launch<128, 0, 128>(a, stream);
  }
  return -1;
}
