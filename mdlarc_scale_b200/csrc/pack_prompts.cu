// Padded prompts (tokens, positions, mask) to the arrays of one prefill call, on the device: packed rows in the order of the
// sequences, cache slots, visible keys, and what the first generated token needs.  Bound by the launch (a batch of 1024 puzzles
// is 14 MB in and 8 MB out); on the host the same arrays take 25 ns a position and their copies wait for the prefill before.
#include "../../include/arcb200.h"
#include "engine.cuh"
#include "launch.cuh"

namespace {

constexpr int PK_THREADS = 256, PK_SPAN = 4 * PK_THREADS;      // positions of one CTA

__device__ __forceinline__ long long ld_int(const void* p, size_t i, int bytes) {
  return bytes == 8 ? reinterpret_cast<const long long*>(p)[i] : (long long)reinterpret_cast<const int*>(p)[i];
}

// sum over the CTA; every thread gets it
__device__ __forceinline__ int cta_sum(int v, int* sm) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  int sum = 0;
#pragma unroll
  for (int w = 0; w < PK_THREADS / 32; ++w) sum += sm[w];
  __syncthreads();
  return sum;
}

// Row r of a call: its length, whether its index max(len - 1, 0) is a real token, and one more than its last real index.
__global__ void __launch_bounds__(PK_THREADS) mask_stats_kernel(const uint8_t* mask, int S, int* out) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ int sm[PK_THREADS / 32];
  const uint8_t* m = mask + (size_t)blockIdx.x * S;
  int n = 0, end = 0;
  for (int s = threadIdx.x; s < S; s += PK_THREADS)
    if (m[s]) { ++n; end = s + 1; }
  n = cta_sum(n, sm);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) end = max(end, __shfl_xor_sync(0xffffffffu, end, o));
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = end;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < PK_THREADS / 32; ++w) end = max(end, sm[w]);
    out[3 * blockIdx.x] = n;
    out[3 * blockIdx.x + 1] = m[max(n - 1, 0)] != 0;
    out[3 * blockIdx.x + 2] = end;
  }
}

__device__ __forceinline__ void store_row(const arcb_pack_args& a, int row, int seq, size_t at, int slot, int count, int kv_row) {
  a.d_token_ids[row] = (int)ld_int(a.d_ids, at, a.id_bytes);
#pragma unroll
  for (int c = 0; c < 3; ++c) a.d_pos_xyz[3 * (size_t)row + c] = (int)ld_int(a.d_pos, 3 * at + c, a.pos_bytes);
  a.d_seq[row] = seq;
  a.d_kv_slot[row] = slot;
  a.d_kv_count[row] = count;
  a.d_kv_row[row] = kv_row;
}

// CTA (sequence of the call, chunk of positions)
__global__ void __launch_bounds__(PK_THREADS) pack_prompts_kernel(arcb_pack_args a) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ int sm[PK_THREADS / 32];
  const int i = blockIdx.x, S = a.seq_len, s0 = blockIdx.y * PK_SPAN, seq = a.d_rows[i], len = a.d_len[i];
  const size_t base = (size_t)seq * S;
  const uint8_t* m = a.d_mask ? a.d_mask + base : nullptr;
  int before = 0;                                // real tokens ahead of this CTA's positions
  if (m) {
    for (int s = threadIdx.x; s < s0; s += PK_THREADS) before += m[s] != 0;
    before = cta_sum(before, sm);
  } else {
    before = s0;
  }
  const int last = max(len - 1, 0);
  const int row0 = a.d_row_start[i], kv0 = a.d_kv_start[i];
  for (int k = 0; k < PK_SPAN; k += PK_THREADS) {
    const int s = s0 + k + threadIdx.x;
    const bool valid = s < S && (!m || m[s]);
    const unsigned votes = __ballot_sync(0xffffffffu, valid);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = __popc(votes);
    __syncthreads();
    int upto = before + __popc(votes & (0xffffffffu >> (31 - (threadIdx.x & 31))));     // real tokens at or ahead of s
#pragma unroll
    for (int w = 0; w < PK_THREADS / 32; ++w) {
      if (w < (int)(threadIdx.x >> 5)) upto += sm[w];
      before += sm[w];
    }
    __syncthreads();
    if (s >= S) continue;
    const int count = a.causal ? upto : len;
    if (valid || a.all_positions)
      store_row(a, row0 + (a.all_positions ? s : upto - 1), seq, base + s, valid ? upto - 1 : -1, count, valid ? kv0 + upto - 1 : -1);
    if (a.with_first && s == last) {
      int first = row0 + (a.all_positions ? s : upto - 1);
      if (!valid && !a.all_positions) {          // a padded position: a query-only row of its own
        first = a.d_extra[i];
        store_row(a, first, seq, base + s, -1, count, -1);
      }
      a.d_first_row[i] = first;
      a.d_first_seq[i] = seq;
      a.d_prompt_len[i] = len;
      // grid state behind the prompt (src/inference.py:171-221)
      const long long tok = ld_int(a.d_ids, base + s, a.id_bytes);
      long long x = ld_int(a.d_pos, 3 * (base + s), a.pos_bytes), y = ld_int(a.d_pos, 3 * (base + s) + 1, a.pos_bytes);
      bool out = ld_int(a.d_pos, 3 * (base + s) + 2, a.pos_bytes) >= 3;
      if (tok == TOK_START) out = false;
      if (tok == TOK_IOSEP) out = true;
      if (tok == TOK_START || tok == TOK_IOSEP) x = y = 0;
      if (tok == TOK_NEWLINE) { x = 0; y = min(y + 1, 29ll); }
      if (tok < 10) x = min(x + 1, 30ll);
      a.d_grid_x[i] = len > 0 ? (int)min(max(x, 0ll), 30ll) : 0;
      a.d_grid_y[i] = len > 0 ? (int)min(max(y, 0ll), 29ll) : 0;
      a.d_grid_in_output[i] = len > 0 ? (int)out : 1;
    }
  }
}

}  // namespace

extern "C" int arcb_mask_stats(const uint8_t* d_mask, int32_t n_rows, int32_t seq_len, int32_t* d_out, void* stream) {
  if (!d_mask || !d_out || n_rows <= 0 || seq_len <= 0) return arcb_fail(ARCB_E_ARG, "bad mask arguments");
  const cudaError_t e = arcb_launch(mask_stats_kernel, dim3(n_rows), dim3(PK_THREADS), 0, (cudaStream_t)stream, d_mask, (int)seq_len, d_out);
  arcb_count_launch(1);
  return e == cudaSuccess ? ARCB_OK : arcb_fail_cuda(e, "mask stats");
}

extern "C" int arcb_pack_prompts(const arcb_pack_args* a, void* stream) {
  if (!a) return arcb_fail(ARCB_E_ARG, "null argument");
  if (a->n_seqs <= 0 || a->seq_len <= 0 || a->seq_len > 65535 * PK_SPAN) return arcb_fail(ARCB_E_ARG, "bad batch sizes");
  if ((a->id_bytes != 4 && a->id_bytes != 8) || (a->pos_bytes != 4 && a->pos_bytes != 8)) return arcb_fail(ARCB_E_ARG, "tokens and positions are int32 or int64");
  if (!a->d_ids || !a->d_pos || !a->d_rows || !a->d_len || !a->d_row_start || !a->d_kv_start || !a->d_token_ids || !a->d_pos_xyz || !a->d_seq ||
      !a->d_kv_slot || !a->d_kv_count || !a->d_kv_row)
    return arcb_fail(ARCB_E_ARG, "null array");
  if (a->with_first && (!a->d_extra || !a->d_first_row || !a->d_first_seq || !a->d_prompt_len || !a->d_grid_x || !a->d_grid_y || !a->d_grid_in_output))
    return arcb_fail(ARCB_E_ARG, "null first-token array");
  const cudaError_t e = arcb_launch(pack_prompts_kernel, dim3(a->n_seqs, (a->seq_len + PK_SPAN - 1) / PK_SPAN), dim3(PK_THREADS), 0,
                                    (cudaStream_t)stream, *a);
  arcb_count_launch(1);
  return e == cudaSuccess ? ARCB_OK : arcb_fail_cuda(e, "pack prompts");
}
