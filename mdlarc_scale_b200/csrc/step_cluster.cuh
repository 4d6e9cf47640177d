// Decode steps of the smallest models inside one cluster; see step_cluster.cu.
#pragma once
#include "rowops.cuh"

// One layer's weights, as the engine packs them.
struct StepLayer {
  const float* ln1;
  const uint16_t* w_qkv;
  const uint16_t* w_out;
  const float* ln2;
  const uint16_t* w_gu;
  const float* b_gu;
  const uint16_t* w_down;
  const float* b_down;
};

struct StepArgs {
  const StepLayer* layers;     // device array
  int n_layers, rows, d, dff, n_heads, n_steps;
  EmbedArgs embed;
  HeadArgs head;
  const float* rope;
  int max_x, max_y, max_z;
  __nv_bfloat16* cache;        // [layer][K, V][row][head][t_max][64]
  const unsigned char* skip;   // finished rows whose attention is left out, or null
  unsigned long long* probe;   // begin and end of layer 0's attention in nanoseconds
};

// CTAs of the cluster that a session's steps run in, 0: none.
int arcb_step_cluster(int rows, int d, int dff, int n_layers, int t_max);
int arcb_launch_step_cluster(const DecodeState& st, const StepArgs& a, int cluster, cudaStream_t stream);
