// The greedy loop's state on the device: what a fed token does to it, and what becomes of a row's logits.
#pragma once
#include "rowops.cuh"

namespace {

// GridStateUpdater.update (src/inference.py:127-168) for sequence b after token tok.
__device__ __forceinline__ void grid_step(const DecodeState& st, int b, int tok) {
  int x = st.gx[b], y = st.gy[b], in_out = st.gin[b];
  const bool is_start = tok == TOK_START, is_sep = tok == TOK_IOSEP, is_end = tok == TOK_END,
             is_nl = tok == TOK_NEWLINE, is_color = tok < 10;
  int z = in_out ? 3 : 1;
  if (is_start) z = 0;
  if (is_sep) z = 2;
  if (is_end) z = 4;
  const int xc = min(max(x, 0), 30), yc = min(max(y, 0), 29);
  st.pos[3 * b + 0] = (is_start || is_sep || is_end || is_nl) ? 0 : xc;
  st.pos[3 * b + 1] = (is_start || is_sep || is_end) ? 0 : yc;
  st.pos[3 * b + 2] = z;
  if (is_start || is_sep) { x = 0; y = 0; }
  if (is_start) in_out = 0;
  if (is_sep) in_out = 1;
  if (is_nl) { x = 0; y = min(y + 1, 29); }
  if (is_color) x = min(x + 1, 30);
  st.gx[b] = min(max(x, 0), 30);
  st.gy[b] = min(max(y, 0), 29);
  st.gin[b] = in_out;
  const int len = st.cur_len[b];
  if (len >= st.t_max) {
    // cache row is full: drop the key and attend to what is there
    arcb_set_error(st.err, ARCB_DEV_BAD_INDEX);
    st.slot[b] = -1;
    st.kv_len[b] = st.t_max;
  } else {
    st.slot[b] = len;
    st.kv_len[b] = len + 1;
  }
}

__device__ __forceinline__ const float* example_row(const EmbedArgs& a, int b) {
  if (!a.example_ids) return nullptr;
  const int ex = min(max(a.example_ids[b], 0), a.num_examples - 1);
  return a.example_embed + (size_t)ex * a.d;
}

// Argmax, and in the generating modes the bookkeeping of row i; one thread.
__device__ __forceinline__ void head_finish(const HeadArgs& a, const DecodeState& st, int i, const float (&acc)[ARCB_VOCAB]) {
  int best = 0;
  float bv = acc[0];
#pragma unroll
  for (int v = 1; v < ARCB_VOCAB; ++v)
    if (acc[v] > bv) { bv = acc[v]; best = v; }  // strict '>' keeps the first maximum (argmax semantics)
  if (a.logits) {
#pragma unroll
    for (int v = 0; v < ARCB_VOCAB; ++v) a.logits[(size_t)i * ARCB_VOCAB + v] = acc[v];
  }
  if (a.argmax) a.argmax[i] = best;
  if (a.mode == HEAD_PLAIN) return;

  // ---- greedy-loop bookkeeping (src/inference.py:573-590, 609-626) ----
  const int b = (a.mode == HEAD_FIRST) ? a.first_seq[i] : i;
  if (b < 0 || b >= st.n_seqs) { arcb_set_error(st.err, ARCB_DEV_BAD_INDEX); return; }
  int out_idx;
  if (a.mode == HEAD_FIRST) {
    const int plen = a.prompt_len[i];
    st.len0[b] = plen;
    st.cur_len[b] = plen;
    st.gx[b] = a.grid_x[i];
    st.gy[b] = a.grid_y[i];
    st.gin[b] = a.grid_in_output[i];
    if (st.finished[b]) { st.finished[b] = 0; atomicSub(st.n_finished, 1); }
    out_idx = 0;
  } else {
    out_idx = st.cur_len[b] - st.len0[b] + 1;
    st.cur_len[b] = min(st.cur_len[b] + 1, st.t_max);
  }
  // Soft constraints (src/inference.py:285-364) act on a copy of the logits, using the grid state
  // after the last fed token (st.gx / st.gy were advanced by decode_begin, or armed just above).
  if (st.disallow_mask || st.palette_mask || st.target_shape || st.temperature > 0.f) {
    float adj[ARCB_VOCAB];
#pragma unroll
    for (int v = 0; v < ARCB_VOCAB; ++v) adj[v] = ((st.disallow_mask >> v) & 1u) ? -INFINITY : acc[v];
    if (st.palette_mask) {
#pragma unroll
      for (int c = 0; c < 10; ++c)
        if (!st.palette_mask[(size_t)b * 10 + c]) adj[c] -= st.palette_penalty;
    }
    if (st.target_shape) {
      const int th = st.target_shape[2 * b], tw = st.target_shape[2 * b + 1];
      if (th >= 0 && tw >= 0) {
        const int gx = st.gx[b], gy = st.gy[b];
        const bool row_full = gx >= tw, past_end = gy >= th;
        if (row_full) {
#pragma unroll
          for (int c = 0; c < 10; ++c) adj[c] -= st.shape_penalty;
        } else {
          adj[TOK_NEWLINE] -= st.shape_penalty;
        }
        if (past_end) {
#pragma unroll
          for (int c = 0; c < 10; ++c) adj[c] -= st.shape_penalty;
          adj[TOK_NEWLINE] -= st.shape_penalty;
        }
      }
    }
    best = 0;
    float bv2 = adj[0];
#pragma unroll
    for (int v = 1; v < ARCB_VOCAB; ++v)
      if (adj[v] > bv2) { bv2 = adj[v]; best = v; }
    if (st.temperature > 0.f) {
      // temperature / top-k sampling (src/inference.py:575-583): softmax of the kept logits, inverse CDF
      const float inv_t = 1.f / fmaxf(st.temperature, 1e-6f);
      const int kk = (st.top_k > 0 && st.top_k < ARCB_VOCAB) ? st.top_k : ARCB_VOCAB;
      float p[ARCB_VOCAB];
      float total = 0.f;
#pragma unroll
      for (int v = 0; v < ARCB_VOCAB; ++v) {
        int rank = 0;  // logits ahead of v: larger, or equal with a smaller index
#pragma unroll
        for (int w = 0; w < ARCB_VOCAB; ++w) rank += (adj[w] > adj[v] || (adj[w] == adj[v] && w < v)) ? 1 : 0;
        p[v] = (rank < kk) ? __expf((adj[v] - bv2) * inv_t) : 0.f;
        total += p[v];
      }
      // counter-based uniform number: splitmix64 of (seed, stream id, generated index)
      const unsigned long long sid = st.sample_stream ? (unsigned long long)(unsigned int)st.sample_stream[b]
                                                      : (unsigned long long)b;
      unsigned long long z = st.sample_seed + 0x9E3779B97F4A7C15ull * (sid + 1) +
                             0xD1B54A32D192ED03ull * (unsigned long long)(out_idx + 1);
      z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
      z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
      z ^= z >> 31;
      const float u = (float)(z >> 40) * (1.f / 16777216.f) * total;
      float run = 0.f;
      int pick = best;
      bool found = false;
#pragma unroll
      for (int v = 0; v < ARCB_VOCAB; ++v) {
        run += p[v];
        if (!found && p[v] > 0.f && u < run) { pick = v; found = true; }
      }
      best = pick;
    }
  }
  int tok = best;
  const bool in_range = out_idx >= 0 && out_idx < st.max_new;
  if (st.forced && in_range) tok = st.forced[(size_t)b * st.max_new + out_idx];
  else if (st.stop_on_end == 1 && st.finished[b]) tok = TOK_END;  // frozen row keeps emitting END (mode 2: keeps decoding)
  if (in_range) {
    st.out_tokens[(size_t)b * st.max_new + out_idx] = tok;
    if (st.step_logits) {
#pragma unroll
      for (int v = 0; v < ARCB_VOCAB; ++v)
        st.step_logits[((size_t)b * st.max_new + out_idx) * ARCB_VOCAB + v] = acc[v];
    }
  }
  if (st.stop_on_end && tok == TOK_END && !st.finished[b]) {
    st.finished[b] = 1;
    atomicAdd(st.n_finished, 1);
  }
  st.cur_tok[b] = tok;
}

}  // namespace
