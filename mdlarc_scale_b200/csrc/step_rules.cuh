// Rules that choose kernels and splits of decode steps from sizes and from the number of SMs: host code without CUDA, so that
// they are tested on any machine.
#pragma once

constexpr int ATTN_CLUSTER_MAX = 8;      // splits of decode attention that are merged inside the launch

// One split of decode attention, or more of them than a cluster merges, has a CTA an item (or a warp): from two CTAs an SM on
// the former.
inline bool attn_cta_per_item(long long n_work, int sms) { return n_work >= 2LL * sms; }

// Split count of decode attention for `work` items (sequences x heads) over a cache of t_max rows: up to eight splits of at least
// two CTA iterations (256 rows), which one launch merges in clusters.  An SM holds four of its CTAs, so a launch takes as long as
// its waves of 4 CTAs an SM times the rows of a split: the count with the shortest such time is taken, within the first wave if
// that is 10 % less than with fewer splits, beyond it only if it is 30 % less (148 SMs, 2048 items: 39 us unsplit, 48 in two
// splits).
// Few items over a long cache leave most of the machine idle in eight splits: more of them, 2.7 CTAs an SM, and a merge launch.
// It costs 5 us, and a split of eight 1 us for every 128 rows: B200, us a layer, eight splits / more: 12 heads over 10 k rows
// 14.0 / 14.2, 12 k 16.3 / 14.9, 32 k 36.5 / 24.3; 16 heads 14.9 / 15.3, 17.6 / 15.6, 40.6 / 28.0; 20 heads 15.8 / 16.6, 18.4 / 18.1,
// 41.9 / 33.1; 24 heads 16.5 / 16.9, 19.1 / 18.8, 43.7 / 36.9; 28 heads 17.0 / 19.4, 20.1 / 21.9, 45.8 / 42.8.
inline int attn_splits(long long work, int t_max, int sms) {
  if (t_max > 12288 && work * ATTN_CLUSTER_MAX <= sms * 13 / 10) {
    const long long s = (sms * 27 / 10 + work - 1) / work;
    const int many = s < 64 ? (int)s : 64;
    if (many > ATTN_CLUSTER_MAX && attn_cta_per_item(work * many, sms)) return many;
  }
  int best = 1;
  double best_time = 0.;
  for (int s = 1; s <= ATTN_CLUSTER_MAX && (s == 1 || 256LL * s <= t_max); ++s) {
    const double time = (double)((work * s + 4 * sms - 1) / (4 * sms)) / s;
    if (s == 1 || time < (work * s <= 4 * sms ? 0.9 : 0.7) * best_time) { best = s; best_time = time; }
  }
  return best;
}

// Splits that a session's scratch is made for: the caller's choice, or the most that any cache is given; 1: none.
inline int attn_scratch_splits(long long work, int requested, int sms) {
  if (requested > 0) return requested > 64 ? 64 : requested;
  const int s = attn_splits(work, 0x7fffffff, sms);
  return s > ATTN_CLUSTER_MAX ? s : 1;
}

// Few-row products: 32 columns a CTA once 16 make more CTAs than run at once (two an SM), for 9 rows and more some earlier, where
// re-reading the activations counts.  B200 (148 SMs), us a launch, 16 / 32 columns: 1 row, 4608 x 1280 4.2 / 4.6, 5120 x 1280
// 5.7 / 5.0, 8192 x 2048 9.0 / 7.7; 16 rows, 1280 x 1280 3.5 / 4.2, 3200 x 1280 4.8 / 4.6, 5120 x 1280 7.2 / 5.8.
inline bool rows_wide_columns(int M, int N, int sms) { return M <= 16 && N / 16 > (M <= 8 ? 2 * sms : sms * 13 / 10); }

// Transposed products instead of few-row ones.  Fewer rows are quicker on gemm_rows.cu up to 32 (us a launch transposed / there: 32
// rows, 1280 x 1280 6.6 / 5.4, 5504 x 1024 8.7 / 7.0; 48 rows, 7.0 / 7.5 and 8.0 / 9.7), unless a CTA there has long sums of its
// own (24 rows, 1280 x 3456 7.8 / 10.5) or every SM several of its CTAs (16 rows, 32000 x 1280 17 / 24)
inline bool mid_transposes(int M, int N, int K, int sms) { return M <= 256 && (M > 32 || (M > 16 && K >= 2560) || N / 128 > sms); }

constexpr int GM_W_BYTES = 128 * 128;            // 128 weight rows x 64 columns
constexpr int GM_SMEM_MAX = 222 * 1024, GM_SMEM_HALF = 111 * 1024;
constexpr int GM_SPLIT_MAX = 8;

struct GmShape {
  int rows;          // rows of A, rounded up to 16: columns of the instruction
  int splits;        // CTAs of a cluster
  int stages;
  // Never less than lets CTAs of an SM outgrow its tensor memory: with one of a cluster waiting for columns that another
  // cluster holds, whose peer waits in turn, neither would end.
  int smem() const {
    const int ring = stages * (GM_W_BYTES + rows * 128), part = rows * 512, least = (rows > 128 ? 100 : 58) * 1024;
    const int need = (ring > part ? ring : part) + 1024 + 16 * stages + 64;
    return need > least ? need : least;
  }
};

// A device query that is asked until it succeeds: `slot` is 0 before that and the answer + 1 from then on.  query(n) says whether n
// was written; the answer of one that fails is 0 for this time only.
template <typename F>
int asked_once(int& slot, F&& query) {
  if (slot) return slot - 1;
  int n = 0;
  if (!query(n)) return 0;
  slot = n + 1;
  return n;
}

// The split with the shortest time: a launch's and a tile's fixed cost (about 4 us a wave), operands at one SM's 110 KB a us,
// and 2 us for the exchange, as long as all clusters run at once.  Tiles beyond one wave run two CTAs an SM where shared
// memory allows it.  clusters_at_once(s): clusters of s CTAs that run at once.
template <typename F>
GmShape gm_shape(int M, int N, int K, int sms, F&& clusters_at_once) {
  GmShape best{};
  best.rows = (M + 15) / 16 * 16;
  const int tiles = N / 128, num_k = K / 64, stage = GM_W_BYTES + best.rows * 128;
  const bool two = tiles > sms && 2 * stage + 2048 <= GM_SMEM_HALF && best.rows * 512 + 2048 <= GM_SMEM_HALF;
  best.splits = 1;
  double best_time = 0.;
  for (int s = 1; s <= GM_SPLIT_MAX && s <= num_k; ++s) {
    if (s > 1 && (tiles * s > sms || tiles > clusters_at_once(s))) continue;
    const int at_once = s == 1 && two ? 2 * sms : sms, waves = s > 1 ? 1 : (tiles + at_once - 1) / at_once;
    const double time = waves * (4. + (num_k + s - 1) / s * (stage / 110e3) * (two ? 2 : 1)) + (s > 1 ? 2. : 0.);
    if (s == 1 || time < best_time) { best.splits = s; best_time = time; }
  }
  const int share = (num_k + best.splits - 1) / best.splits, room = ((two ? GM_SMEM_HALF : GM_SMEM_MAX) - 2048) / stage;
  best.stages = share < room ? share : room;
  return best;
}

// Steps inside one cluster (step_cluster.cu): shared memory of a CTA, in bytes from its start.
struct StepClusterSmem {
  int xn, hs, q, rec, red, tokens, head, even, odd, total;
};
constexpr int STEP_CLUSTER_SMEM_MAX = 220 * 1024;

inline StepClusterSmem step_cluster_smem(int rows, int d, int dff, int heads, int cl) {
  const int items = rows * heads, records = items < cl ? cl : items;
  const int qkv = (3 * d / 16 + cl - 1) / cl, gu = 2 * ((dff / 16 + cl - 1) / cl), wide = qkv > gu ? qkv : gu, narrow = (d / 16 + cl - 1) / cl;
  const int long_k = d > dff ? d : dff;
  StepClusterSmem s;
  s.xn = 2 * 8 * d * 4;
  s.hs = s.xn + 8 * (d * 2 + 64);
  s.q = s.hs + 8 * (dff * 2 + 64);
  s.rec = s.q + 8 * d * 2;
  s.red = s.rec + records * 68 * 4;
  s.tokens = s.red + wide * 8 * 160 * 4;
  s.head = s.tokens + (14 + 8) * d * 4;
  s.even = (s.head + 15 * d * 4 + 127) / 128 * 128;
  s.odd = s.even + wide * 32 * d;                                    // 16 rows a tile
  s.total = s.odd + narrow * 32 * long_k;
  return s;
}

// Whether the cluster is the quicker of the two, from what both were measured to take (B200, 199 sizes of 128 to 384 columns, 1 to 4
// rows, 1 to 12 layers, 100 to 30 k cached rows; deviations 1.2 and 2.1 us).  us a step of a launch of one step: the cluster 11 and a layer
// 7.3, 1.1 a MB of its weights, 0.6 a row and 0.26 a row and MB, 4.4 a thousand keys that one CTA reads and 1.8 where CTAs take a second
// (row, head) item; launches of a graph 16 and a layer 13.3, 0.6 a thousand cached rows, 0.7 a million of all rows' columns.  A launch of many
// steps spares the cluster 5.6 us a step, and a first launch the recording of a graph, hence the 2 us.  Graph / one step a launch / 16:
// 256 columns, 4 layers: one row over 300 rows 70 / 51 / 46, over 2400 76 / 60 / 55, four over 600 76 / 74 / 68; one layer: one row over 10 k 37 / 31 /
// 25, four over 1200 31 / 29 / 24, over 2400 31 / 35 / 30; 384 columns, 4 layers: two rows over 300 72 / 66 / 60; not taken: four over 300 72 / 82 / 76, one
// layer, four over 2400 31 / 48 / 42.  Weights and cached rows beyond 16 MB a step are for the whole machine.
// Shared memory holds a layer of 384 columns up to d_ff 448, of 256 up to 1024 and of 128 up to 1536 (16 CTAs); none of 512.
constexpr int STEP_CLUSTER_ROWS = 4, STEP_CLUSTER_WIDTH = 384;
inline bool step_cluster_fits(int rows, int d, int dff, int n_layers, int t_max, int cl) {
  if (rows < 1 || rows > STEP_CLUSTER_ROWS || d > STEP_CLUSTER_WIDTH || d % 128 || dff % 64) return false;
  if (step_cluster_smem(rows, d, dff, d / 64, cl).total > STEP_CLUSTER_SMEM_MAX) return false;
  const long long weights = 2LL * (4LL * d * d + 3LL * d * dff), cached = 4LL * d * rows * t_max;      // bytes of a layer
  if (n_layers * (weights + cached) > 16LL << 20) return false;
  const int items = rows * (d / 64), splits = items < cl ? cl / items : 1, turns = (items * splits + cl - 1) / cl;
  const double mb = weights * 1e-6, kt = t_max * 1e-3;
  const double cluster = 11. + n_layers * (7.3 + 1.1 * mb + rows * (0.6 + 0.26 * mb) + 4.4 * turns * kt / splits + 1.8 * (turns - 1));
  const double graph = 16. + n_layers * (13.3 + 0.6 * kt + 0.7 * rows * d * kt * 1e-3);
  return cluster <= graph + 2.;
}
