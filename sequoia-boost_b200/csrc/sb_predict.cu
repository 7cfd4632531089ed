// sb_predict.cu — ensemble prediction (K9): the device copy of a model, margins,
// predict and predict_leaf. TreeSHAP (K10) is in sb_shap.cu.
//
// Replaces BoostedModel::predict_margin_limited (learner/model.rs:231-285),
// predict (:291-300, with pred_transform of objective/classification.rs:
// :73-77 and multiclass.rs:93-99), predict_leaf (:330-341) and
// node_mean_value (learner/shap.rs:288-302).
//
// Margins: k_leaf_values routes every (row, tree) pair, k_margin_sum adds each
// (row, class) over its trees in tree order, so margins are bit-identical.
#include <cmath>
#include <cstring>
#include <functional>

#include "sb_internal.cuh"

namespace sb {
namespace {

constexpr uint32_t NF_DEFAULT_LEFT = 1u << 30;
constexpr uint32_t NF_CATEGORICAL = 1u << 31;
constexpr uint32_t NF_FEATURE = (1u << 30) - 1;

// A node in 8 bytes, for ensembles of numeric splits whose children sit side
// by side: {condition or leaf value, NodeBits}. x / y as in uint2.
enum : uint32_t { CN_LEFT = 0xFFFFu, CN_FEATURE_SHIFT = 16, CN_FEATURE = 0x3FFFu, CN_DEFAULT_LEFT = 1u << 30, CN_LEAF = 1u << 31 };

struct PredDev {
  const int4* nodes;        // {feat|flags, cond (leaf value for leaves / cat_begin), left, right}
  const int* cat_end;       // per node (categorical nodes only)
  const int64_t* tree_off;  // [n_trees + 1]
  const uint32_t* cats;     // global category pool
  const float* weights;
  int n_trees;
  const uint2* cnodes;      // the nodes in 8 bytes, or null when they have no such form
};

__device__ __forceinline__ bool is_missing_d(float v, float missing, bool miss_nan) {
  return miss_nan ? isnan(v) : (v == missing);
}

// RegTree::leaf_id_with over a dense row (regtree.rs:213-242) whose value of
// feature f is value(f): the leaf's node index, and its packed node in *leaf.
template <typename Value>
__device__ __forceinline__ int route_to_leaf(const PredDev& P, int t, float missing, bool miss_nan, Value value,
                                             int4* leaf) {
  const int4* nd = P.nodes + P.tree_off[t];
  int nid = 0;
  for (;;) {
    int4 x = __ldg(nd + nid);
    if (x.z < 0) {
      *leaf = x;
      return nid;
    }
    uint32_t ff = (uint32_t)x.x;
    float v = value(ff & NF_FEATURE);
    bool go_left;
    if (is_missing_d(v, missing, miss_nan)) {
      go_left = (ff & NF_DEFAULT_LEFT) != 0;
    } else if (ff & NF_CATEGORICAL) {
      uint32_t c = f32_as_u32(v);
      go_left = false;
      for (int i = x.y; i < P.cat_end[P.tree_off[t] + nid]; ++i)
        if (P.cats[i] == c) {
          go_left = true;
          break;
        }
    } else {
      go_left = v < __int_as_float(x.y);
    }
    nid = go_left ? x.z : x.w;
  }
}

// predict_leaf (model.rs:330-341): out [n][T] leaf node ids, one thread per
// (row, tree) with the tree index fastest, so the stores are coalesced and a
// warp reads one row.
__global__ void k_leaf_ids(PredDev P, const float* __restrict__ X, size_t n, int F, float missing,
                           uint32_t* __restrict__ out) {
  const size_t T = (size_t)P.n_trees;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * T) return;
  const size_t r = i / T;
  const int t = (int)(i - r * T);
  const float* row = X + r * F;
  int4 x;
  out[i] = (uint32_t)route_to_leaf(P, t, missing, isnan(missing), [&](uint32_t f) { return row[f]; }, &x);
}

// The leaf value of a tree in compact nodes `nd` for a row whose value of
// feature f is value(f).
template <typename Value>
__device__ __forceinline__ float route_compact(const uint2* nd, float missing, bool miss_nan, Value value) {
  uint2 x = nd[0];
  while (!(x.y & CN_LEAF)) {
    const float v = value((x.y >> CN_FEATURE_SHIFT) & CN_FEATURE);
    const bool left = is_missing_d(v, missing, miss_nan) ? (x.y & CN_DEFAULT_LEFT) != 0 : v < __uint_as_float(x.x);
    x = nd[(x.y & CN_LEFT) + (left ? 0 : 1)];
  }
  return __uint_as_float(x.x);
}

// What is added to a row's margin before the trees' values, by output.
struct MarginStart {
  float base;
  const float* base_margin;  // [n][K] (kind 1) or [n] (kind 2), or null
  int kind;
};
__device__ __forceinline__ float margin_start(const MarginStart& m, size_t r, int K, int c) {
  if (m.kind == 1) return m.base_margin[r * K + c];
  if (m.kind == 2) return m.base_margin[r];
  return m.base;
}

// Margins in two phases. Phase 1: the leaf value of every (row, tree),
// tree-major. A block takes 2^lr rows, up to 32, and a tree per remaining
// thread, so that all trees of a small request are walked at once: its time is
// one tree's chain of dependent loads. With many rows a thread takes up to 8
// trees and the block's rows are staged in shared memory (read row by row from
// global memory they cost a sector per value); the time is then the gathers of
// nodes, 8 bytes each (16 rows x 1000 trees of depth 8: 8.9 -> 5.2 us; 65,536
// rows: 1.85 -> 0.86 ms; one kernel that streams the nodes through shared memory
// and adds in place took 0.85 ms for both phases there and 0.12 ms for any small
// request). Which rows are staged: leaf_plan.
constexpr int LEAF_THREADS = 128;
__global__ void __launch_bounds__(LEAF_THREADS) k_leaf_values(PredDev P, const float* __restrict__ X, size_t n, int F,
                                                              float missing, int limit, int lr, int staged,
                                                              int per_thread, float* __restrict__ buf) {
  extern __shared__ float s_rows[];  // [F][2^lr + 1]
  const int rows = 1 << lr, row = threadIdx.x & (rows - 1);
  const size_t r0 = (size_t)blockIdx.x * rows, r = r0 + row;
  const int tpb = LEAF_THREADS >> lr;  // trees at once
  const int t0 = blockIdx.y * tpb * per_thread + (threadIdx.x >> lr);
  const bool miss_nan = isnan(missing);
  if (staged) {
    const int nr = (int)min((size_t)rows, n - r0);
    for (int i = threadIdx.x; i < nr * F; i += LEAF_THREADS) {
      const int q = i / F;
      s_rows[(i - q * F) * (rows + 1) + q] = X[r0 * F + i];
    }
    __syncthreads();
  }
  if (r >= n) return;
  const float* own = X + r * F;
  auto global = [&](uint32_t f) { return own[f]; };
  for (int i = 0; i < per_thread; ++i) {
    const int t = t0 + i * tpb;
    if (t >= limit) return;
    float v;
    if (staged) {
      v = route_compact(P.cnodes + P.tree_off[t], missing, miss_nan,
                        [&](uint32_t f) { return s_rows[f * (rows + 1) + row]; });
    } else if (P.cnodes) {
      v = route_compact(P.cnodes + P.tree_off[t], missing, miss_nan, global);
    } else {
      int4 x;
      route_to_leaf(P, t, missing, miss_nan, global, &x);
      v = __int_as_float(x.y);
    }
    buf[(size_t)t * n + r] = v;
  }
}

// Phase 2: a block adds 32 rows' leaf values in tree order, with separate f32
// multiply and add, which is the reference's accumulation. All its
// warps bring the next chunk's weighted values into shared memory while the
// first min(K, SUM_WARPS) add the current one (warp w takes the classes c with
// c % SUM_WARPS == w; lane = row; with more classes than warps the sums wait in
// `out` between chunks).
// 16 warps and 64 KB where there is more than one chunk of values to bring; 4
// warps and 16 KB
//  - in the serving loop: beside a batch of explanations an SM frees little at a
//    time, and blocks of 16 warps waited for it behind that batch (mixed stream,
//    requests of at most 4096 rows: p99 24 ms, 0.9 with these);
//  - for up to 64 trees, which are one of their chunks, of up to 4 classes: an SM
//    holds four times as many such blocks (1M rows x 20 features, 5 trees, pinned,
//    whole call 2.40 -> 2.21 ms; 100,000 rows, 60 trees 0.356 -> 0.340).
constexpr int SUM_ROWS = 32;
template <int SUM_WARPS>
__global__ void __launch_bounds__(SUM_ROWS * SUM_WARPS)
    k_margin_sum(PredDev P, const float* __restrict__ buf, size_t n, int K, int limit, MarginStart start, int objective,
                 float* __restrict__ out) {
  constexpr int SUM_CHUNK = 16 * SUM_WARPS;
  extern __shared__ float sum_sm[];  // [2][SUM_CHUNK][SUM_ROWS]
  auto s_leaf = reinterpret_cast<float(*)[SUM_CHUNK][SUM_ROWS]>(sum_sm);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t r = (size_t)blockIdx.x * SUM_ROWS + lane;
  const bool in = r < n;
  constexpr int PER = SUM_CHUNK / SUM_WARPS;
  float v[PER];
  auto load = [&](int t0) {
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int t = t0 + warp + i * SUM_WARPS;
      v[i] = in && t < limit ? __fmul_rn(P.weights ? P.weights[t] : 1.0f, buf[(size_t)t * n + r]) : 0.0f;
    }
  };
  float acc = 0.0f;  // the class of this warp
  const bool in_regs = K <= SUM_WARPS;
  if (in && in_regs && warp < K) acc = margin_start(start, r, K, warp);
  if (!in_regs && in)
    for (int c = warp; c < K; c += SUM_WARPS) out[r * K + c] = margin_start(start, r, K, c);
  load(0);
  for (int t0 = 0, b = 0; t0 < limit; t0 += SUM_CHUNK, b ^= 1) {
#pragma unroll
    for (int i = 0; i < PER; ++i) s_leaf[b][warp + i * SUM_WARPS][lane] = v[i];
    __syncthreads();
    load(t0 + SUM_CHUNK);
    const int cnt = min(SUM_CHUNK, limit - t0);
    if (K == 1) {
      if (warp == 0) {
        int t = 0;
        for (; t + 32 <= cnt; t += 32) {
          float x[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) x[j] = s_leaf[b][t + j][lane];
#pragma unroll
          for (int j = 0; j < 32; ++j) acc = __fadd_rn(acc, x[j]);
        }
        for (; t < cnt; ++t) acc = __fadd_rn(acc, s_leaf[b][t][lane]);
      }
    } else {
      for (int c = warp; c < K; c += SUM_WARPS) {
        float a = in_regs ? acc : in ? out[r * K + c] : 0.0f;
        for (int t = (c - t0 % K + K) % K; t < cnt; t += K) a = __fadd_rn(a, s_leaf[b][t][lane]);
        if (in_regs) acc = a;
        else if (in) out[r * K + c] = a;
      }
    }
  }
  if (!in || !in_regs) return;
  if (K == 1) {
    if (warp == 0) {
      pred_transform_row(&acc, 1, objective);
      out[r] = acc;
    }
    return;
  }
  if (warp < K) out[r * K + warp] = acc;
}

// Rows and trees of a k_leaf_values block.
struct LeafPlan {
  int lr, staged, per_thread;
  size_t smem;
};
// Staged rows are paid for by what is read of them: a copy of all F values
// against about a path of each of the block's trees. Whole calls, staged /
// read from global memory, us: 4096 rows x 100 features x 1000 trees of depth 8
// (32 trees to a block) 206 / 227; 300 rows (4 trees) 86 / 75; 1000 rows x 360
// features x 500 trees of depth 6 194 / 139. 16-byte nodes read from global
// memory at any size, since their walk leaves L1 to the rows (4096 rows x 100
// features, 500 trees of depth 8 with categorical splits: 464 staged, 362 not).
// Without staging a thread takes one tree: more of them only leave an uneven
// last wave (the same call: 362 at up to 8 trees, 301 at one). A warp has one
// tree of 16-byte nodes however few the rows: lanes wait for one another's
// category lists, and trees in one warp meet theirs at different steps (one row,
// 100 trees of lists of some 100 categories: 128 with 32 trees to a warp, 68).
LeafPlan leaf_plan(size_t n, size_t F, size_t limit, bool compact, int num_sms) {
  LeafPlan p{0, 0, 1, 0};
  while (p.lr < 5 && (!compact || ((size_t)1 << p.lr) < n)) ++p.lr;
  // one tree per thread while all fit the chip at once, up to 8
  const size_t pairs = n * limit, chip = (size_t)num_sms * 2048;
  const int many = (int)std::max<size_t>(1, std::min<size_t>(8, pairs / chip));
  const size_t sm = F * sizeof(float) * ((1 << p.lr) + 1), trees = (size_t)(LEAF_THREADS >> p.lr) * many;
  if (compact && sm <= 48 * 1024 && F <= 4 * trees) {
    p.staged = 1;
    p.per_thread = many;
    p.smem = sm;
  }
  const size_t at_once = (size_t)(LEAF_THREADS >> p.lr) * 65535;  // a grid's rows of blocks
  p.per_thread = std::max(p.per_thread, (int)((limit + at_once - 1) / at_once));
  return p;
}

// n rows' margins on a stream; with transform_objective >= 0 a single output
// is put through pred_transform as well. d_buf holds chunk * T floats. `serving`:
// beside other kernels, in small blocks.
int margins(sb_ctx* ctx, cudaStream_t st, const PredDev& P, const float* d_X, size_t n, size_t F, float missing,
            int K, int limit, float base, const float* d_bm, int bm_kind, float* d_buf, size_t chunk, float* d_out,
            int transform_objective, bool serving) {
  const int objective = K == 1 && transform_objective >= 0 ? transform_objective : (int)SB_OBJ_SQUARED_ERROR;
  for (size_t r0 = 0; r0 < n; r0 += chunk) {
    const size_t nb = std::min(chunk, n - r0);
    if (limit > 0) {
      const LeafPlan L = leaf_plan(nb, F, (size_t)limit, P.cnodes != nullptr, ctx->num_sms);
      const int per = (LEAF_THREADS >> L.lr) * L.per_thread;
      dim3 grid((unsigned)((nb + (1 << L.lr) - 1) >> L.lr), (unsigned)((limit + per - 1) / per));
      SB_LAUNCH_ON(ctx, st, k_leaf_values, grid, LEAF_THREADS, L.smem, P, d_X + r0 * F, nb, (int)F, missing, limit, L.lr,
                   L.staged, L.per_thread, d_buf);
    }
    const float* bm = d_bm ? d_bm + (bm_kind == 1 ? r0 * K : r0) : nullptr;
    const int warps = serving || (limit <= 64 && K <= 4) ? 4 : 16;
    const size_t sum_smem = 2 * 16 * warps * SUM_ROWS * sizeof(float);
    auto sum = warps == 4 ? k_margin_sum<4> : k_margin_sum<16>;
    SB_TRY(raise_smem_limit((const void*)sum, sum_smem));
    SB_LAUNCH_ON(ctx, st, sum, (unsigned)((nb + SUM_ROWS - 1) / SUM_ROWS), SUM_ROWS * warps, sum_smem, P, d_buf, nb, K,
                 limit, MarginStart{base, bm, bm ? bm_kind : 0}, objective, d_out + r0 * K);
  }
  return SB_OK;
}

// The 8-byte form of packed nodes that have one.
__global__ void k_compact_nodes(const int4* __restrict__ nodes, size_t n, uint2* __restrict__ out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int4 x = nodes[i];
  const uint32_t f = (uint32_t)x.x;
  out[i] = make_uint2((uint32_t)x.y, x.z < 0 ? (uint32_t)CN_LEAF
                                             : (uint32_t)x.z | ((f & CN_FEATURE) << CN_FEATURE_SHIFT) |
                                                   ((f & NF_DEFAULT_LEFT) ? (uint32_t)CN_DEFAULT_LEFT : 0u));
}

__global__ void k_transform(float* __restrict__ v, size_t n, int K, int objective) {
  size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  pred_transform_row(v + r * K, K, objective);
}

}  // namespace

int tree_depth(const HostTree& t) {
  std::vector<int> depth(t.nodes.size(), 0);
  int mx = 0;
  for (size_t i = 0; i < t.nodes.size(); ++i) {
    const sb_node& nd = t.nodes[i];
    if (nd.left >= 0) {
      depth[nd.left] = depth[i] + 1;
      depth[nd.right] = depth[i] + 1;
      mx = std::max(mx, depth[i] + 1);
    }
  }
  return mx;
}

double node_mean_value(const HostTree& t, int id) {  // shap.rs:288-302
  const sb_node& nd = t.nodes[id];
  if (nd.left < 0) return (double)nd.leaf_value;
  double cover = (double)nd.sum_hess;
  if (cover <= 0.0) return 0.0;
  double lc = (double)t.nodes[nd.left].sum_hess, rc = (double)t.nodes[nd.right].sum_hess;
  return (lc * node_mean_value(t, nd.left) + rc * node_mean_value(t, nd.right)) / cover;
}

int model_upload(sb_model* m) {
  if (m->dev_valid) return SB_OK;
  sb_ctx* ctx = m->ctx;
  DevEnsemble& D = m->dev;
  const int T = (int)m->trees.size();
  std::vector<int64_t> off(T + 1, 0);
  for (int t = 0; t < T; ++t) off[t + 1] = off[t] + (int64_t)m->trees[t].nodes.size();
  std::vector<int4> packed(off[T]);
  std::vector<int> catend;  // empty without categorical nodes: nothing reads it then
  std::vector<uint32_t> cats;
  int maxd = 0;
  bool compact = off[T] > 0;  // every tree has the 8-byte form (CN_*)
  for (int t = 0; t < T; ++t) {
    const HostTree& tr = m->trees[t];
    int cat_base = (int)cats.size();
    cats.insert(cats.end(), tr.cats.begin(), tr.cats.end());
    compact = compact && !tr.nodes.empty() && tr.nodes.size() <= CN_LEFT;
    for (size_t i = 0; i < tr.nodes.size(); ++i) {
      const sb_node& nd = tr.nodes[i];
      int4 x;
      uint32_t ff = nd.split_feature & NF_FEATURE;
      if (nd.default_left) ff |= NF_DEFAULT_LEFT;
      if (nd.is_categorical && nd.left >= 0) ff |= NF_CATEGORICAL;
      x.x = (int)ff;
      if (nd.left < 0) {
        float lv = nd.leaf_value;
        std::memcpy(&x.y, &lv, 4);
      } else if (nd.is_categorical) {
        x.y = cat_base + (int)nd.cat_begin;
        if (catend.empty()) catend.resize(off[T], 0);
        catend[off[t] + i] = cat_base + (int)nd.cat_end;
      } else {
        float c = nd.split_cond;
        std::memcpy(&x.y, &c, 4);
      }
      x.z = nd.left;
      x.w = nd.right;
      if (nd.left >= 0 && (nd.is_categorical || nd.right != nd.left + 1 || nd.split_feature > CN_FEATURE ||
                           (size_t)nd.right >= tr.nodes.size()))
        compact = false;
      packed[off[t] + i] = x;
    }
    maxd = std::max(maxd, tree_depth(tr));
  }
  SB_TRY(D.nodes.alloc(ctx, std::max<size_t>(packed.size(), 1)));
  SB_TRY(D.tree_off.alloc(ctx, T + 1));
  SB_TRY(D.cats.alloc(ctx, std::max<size_t>(cats.size(), 1)));
  SB_TRY(D.weights.alloc(ctx, std::max(T, 1)));
  cudaStream_t st = ctx->stream;
  if (!packed.empty()) {
    SB_CUDA(cudaMemcpyAsync(D.nodes.p, packed.data(), packed.size() * 16, cudaMemcpyHostToDevice, st));
  }
  D.compact = compact;
  if (compact) {
    SB_TRY(D.cnodes.alloc(ctx, packed.size()));
    SB_LAUNCH(ctx, k_compact_nodes, (unsigned)((packed.size() + 255) / 256), 256, 0, D.nodes.p, packed.size(), D.cnodes.p);
  }
  SB_CUDA(cudaMemcpyAsync(D.tree_off.p, off.data(), (T + 1) * 8, cudaMemcpyHostToDevice, st));
  if (!cats.empty()) SB_CUDA(cudaMemcpyAsync(D.cats.p, cats.data(), cats.size() * 4, cudaMemcpyHostToDevice, st));
  if (T) SB_CUDA(cudaMemcpyAsync(D.weights.p, m->weights.data(), T * 4, cudaMemcpyHostToDevice, st));
  SB_TRY(D.cat_end.alloc(ctx, std::max<size_t>(catend.size(), 1)));
  if (!catend.empty())
    SB_CUDA(cudaMemcpyAsync(D.cat_end.p, catend.data(), catend.size() * 4, cudaMemcpyHostToDevice, st));
  SB_CUDA(cudaStreamSynchronize(st));
  D.n_trees = T;
  D.max_depth = maxd;
  m->dev_valid = true;
  return SB_OK;
}

static PredDev pred_dev(const sb_model* m) {
  PredDev P;
  P.nodes = m->dev.nodes.p;
  P.cat_end = m->dev.cat_end.p;
  P.tree_off = m->dev.tree_off.p;
  P.cats = m->dev.cats.p;
  P.weights = m->dev.weights.p;
  P.n_trees = m->dev.n_trees;
  P.cnodes = m->dev.compact ? m->dev.cnodes.p : nullptr;
  return P;
}

// Rows per phase-1 chunk, so that the tree-major leaf buffer stays <= 64 MB.
size_t margin_chunk_rows(const sb_model* m) {
  const size_t T = (size_t)std::max(m->dev.n_trees, 1);
  return std::max<size_t>(1024, (size_t)(64ull << 20) / (T * 4));
}

int predict_margin_device(sb_model* m, const float* d_X, size_t n, size_t F, float missing,
                          const float* d_base_margin, int bm_kind, size_t ntree_limit, float* d_out,
                          int transform_objective) {
  sb_ctx* ctx = m->ctx;
  SB_TRY(model_upload(m));
  const int Kc = m->num_class >= 2 ? m->num_class : 1;
  const int T = m->dev.n_trees;
  const int limit = ntree_limit == 0 ? T : (int)std::min<size_t>(ntree_limit, (size_t)T);
  const PredDev P = pred_dev(m);
  if (n == 0) return SB_OK;
  const size_t chunk = std::min(n, margin_chunk_rows(m));  // leaf buffer <= 64 MB
  DBuf<float> buf;
  if (limit > 0) SB_TRY(buf.alloc(ctx, (size_t)limit * chunk));
  return margins(ctx, ctx->stream, P, d_X, n, F, missing, Kc, limit, m->base_score, d_base_margin, bm_kind, buf.p,
                 chunk, d_out, transform_objective, false);
}

// The margins of n host rows, through their device buffer d_X. Large requests
// go in parts, each copied on a second stream while the part before is computed
// (65,536 rows x 100 features, 1000 trees: 0.48 ms of copies beside 0.97 ms of
// kernels). The stream, its event and the parts cost 0.05 to 0.15 ms, by the
// host, so that both the copy and the walk have to take longer than that: from 4 MB
// and 10 million (row, tree) pairs on. Whole calls in one part / in parts, ms:
// 100,000 rows x 20, 60 trees 0.35 / 0.41; 20,000 rows x 100, 500 trees 0.61 / 0.56
// on one host and 0.59 / 0.68 on another; 1000 trees 0.77 / 0.71; 65,536 rows x 20,
// 500 trees 0.70 / 0.63; 1M rows x 20, 5 trees, pinned 2.4 / 2.9 (8192 rows to a
// part). Eight parts at most: each copy starts anew (1M rows x 20, 300 trees: 122
// parts 7.3, 8 parts 6.9).
// The context's stream waits for every copy, so the buffers' order of use and
// release on it is as with one stream.
constexpr size_t PART_ROWS = 8192, MAX_PARTS = 8;
constexpr size_t SPLIT_BYTES = 4000000, SPLIT_PAIRS = 10000000;
static int margins_from_host(sb_model* m, const float* X, float* d_X, size_t n, size_t F, float missing,
                             const float* d_base_margin, size_t ntree_limit, float* d_out, int transform_objective) {
  sb_ctx* ctx = m->ctx;
  const int K = m->num_class >= 2 ? m->num_class : 1;
  SB_TRY(model_upload(m));
  const size_t trees = (size_t)m->dev.n_trees, limit = ntree_limit ? std::min(ntree_limit, trees) : trees;
  if (n < 2 * PART_ROWS || n * F * sizeof(float) < SPLIT_BYTES || n * limit < SPLIT_PAIRS) {
    SB_CUDA(cudaMemcpyAsync(d_X, X, n * F * sizeof(float), cudaMemcpyHostToDevice, ctx->stream));
    return predict_margin_device(m, d_X, n, F, missing, d_base_margin, 1, ntree_limit, d_out, transform_objective);
  }
  struct Second {  // the copies' stream and event; waited for before they go
    cudaStream_t st = nullptr;
    cudaEvent_t ev = nullptr;
    ~Second() {
      if (st) {
        cudaStreamSynchronize(st);
        cudaStreamDestroy(st);
      }
      if (ev) cudaEventDestroy(ev);
    }
  } s;
  SB_CUDA(cudaStreamCreateWithFlags(&s.st, cudaStreamNonBlocking));
  SB_CUDA(cudaEventCreateWithFlags(&s.ev, cudaEventDisableTiming));
  SB_CUDA(cudaEventRecord(s.ev, ctx->stream));  // d_X's allocation is ordered on the context's stream
  SB_CUDA(cudaStreamWaitEvent(s.st, s.ev, 0));
  const size_t part = std::max(PART_ROWS, (n + MAX_PARTS - 1) / MAX_PARTS);
  for (size_t r0 = 0; r0 < n; r0 += part) {
    const size_t nb = std::min(part, n - r0);
    SB_CUDA(cudaMemcpyAsync(d_X + r0 * F, X + r0 * F, nb * F * sizeof(float), cudaMemcpyHostToDevice, s.st));
    SB_CUDA(cudaEventRecord(s.ev, s.st));
    SB_CUDA(cudaStreamWaitEvent(ctx->stream, s.ev, 0));
    SB_TRY(predict_margin_device(m, d_X + r0 * F, nb, F, missing, d_base_margin ? d_base_margin + r0 * K : nullptr, 1,
                                 ntree_limit, d_out + r0 * K, transform_objective));
  }
  return SB_OK;
}

// ---- batch launchers on an explicit stream with caller-owned buffers (used
// by the serving loop; the model must be resident, see model_upload)

int margin_batch(sb_model* m, cudaStream_t st, const float* d_X, size_t n, size_t F, float missing,
                 float* d_buf, size_t buf_rows, float* d_out) {
  sb_ctx* ctx = m->ctx;
  const int Kc = m->num_class >= 2 ? m->num_class : 1;
  const PredDev P = pred_dev(m);
  if (n == 0) return SB_OK;
  return margins(ctx, st, P, d_X, n, F, missing, Kc, m->dev.n_trees, m->base_score, nullptr, 0, d_buf, buf_rows,
                 d_out, -1, true);
}

}  // namespace sb

extern "C" {

int sb_predict_margin(sb_model* m, const float* X, size_t n_rows, size_t n_cols, float missing,
                      const float* base_margin, size_t ntree_limit, float* out) {
  using namespace sb;
  SB_REQUIRE(m && out && (X || n_rows == 0), SB_ERR_INVALID_ARG, "NULL argument");
  SB_REQUIRE(n_cols == (size_t)m->n_features, SB_ERR_DIMENSION,
             "dimension mismatch: expected %d features, got %zu", m->n_features, n_cols);
  if (n_rows == 0) return SB_OK;
  sb_ctx* ctx = m->ctx;
  SB_CUDA(cudaSetDevice(ctx->device));
  const int K = m->num_class >= 2 ? m->num_class : 1;
  DBuf<float> dX, dbm, dout;
  SB_TRY(dX.alloc(ctx, n_rows * n_cols));
  SB_TRY(dout.alloc(ctx, n_rows * K));
  if (base_margin) {
    SB_TRY(dbm.alloc(ctx, n_rows * K));
    SB_CUDA(cudaMemcpyAsync(dbm.p, base_margin, dbm.bytes(), cudaMemcpyHostToDevice, ctx->stream));
  }
  SB_TRY(margins_from_host(m, X, dX.p, n_rows, n_cols, missing, dbm.p, ntree_limit, dout.p, -1));
  SB_CUDA(cudaMemcpyAsync(out, dout.p, dout.bytes(), cudaMemcpyDeviceToHost, ctx->stream));
  SB_CUDA(cudaStreamSynchronize(ctx->stream));
  return SB_OK;
}

int sb_predict(sb_model* m, const float* X, size_t n_rows, size_t n_cols, float missing,
               const float* base_margin, float* out) {
  using namespace sb;
  SB_REQUIRE(m && out && (X || n_rows == 0), SB_ERR_INVALID_ARG, "NULL argument");
  SB_REQUIRE(n_cols == (size_t)m->n_features, SB_ERR_DIMENSION,
             "dimension mismatch: expected %d features, got %zu", m->n_features, n_cols);
  if (n_rows == 0) return SB_OK;
  sb_ctx* ctx = m->ctx;
  SB_CUDA(cudaSetDevice(ctx->device));
  const int K = m->num_class >= 2 ? m->num_class : 1;
  DBuf<float> dX, dbm, dout;
  SB_TRY(dX.alloc(ctx, n_rows * n_cols));
  SB_TRY(dout.alloc(ctx, n_rows * K));
  if (base_margin) {
    SB_TRY(dbm.alloc(ctx, n_rows * K));
    SB_CUDA(cudaMemcpyAsync(dbm.p, base_margin, dbm.bytes(), cudaMemcpyHostToDevice, ctx->stream));
  }
  // predict uses the effective tree count: (best_iteration + 1) * K after
  // early stopping, else all trees (model.rs:213-219)
  const size_t limit = m->best_iteration >= 0 ? (size_t)(m->best_iteration + 1) * K : 0;
  SB_TRY(margins_from_host(m, X, dX.p, n_rows, n_cols, missing, dbm.p, limit, dout.p, m->objective));
  if (K > 1) SB_LAUNCH(ctx, k_transform, (unsigned)((n_rows + 255) / 256), 256, 0, dout.p, n_rows, K, m->objective);
  SB_CUDA(cudaMemcpyAsync(out, dout.p, dout.bytes(), cudaMemcpyDeviceToHost, ctx->stream));
  SB_CUDA(cudaStreamSynchronize(ctx->stream));
  return SB_OK;
}

int sb_predict_contribs(sb_model* m, const float* X, size_t n_rows, size_t n_cols, float missing,
                        float* out) {
  using namespace sb;
  SB_REQUIRE(m && out && (X || n_rows == 0), SB_ERR_INVALID_ARG, "NULL argument");
  SB_REQUIRE(n_cols == (size_t)m->n_features, SB_ERR_DIMENSION,
             "dimension mismatch: expected %d features, got %zu", m->n_features, n_cols);
  if (n_rows == 0) return SB_OK;
  sb_ctx* ctx = m->ctx;
  SB_CUDA(cudaSetDevice(ctx->device));
  const int K = m->num_class >= 2 ? m->num_class : 1;
  DBuf<float> dX, dout;
  SB_TRY(dX.alloc(ctx, n_rows * n_cols));
  SB_TRY(dout.alloc(ctx, n_rows * K * (n_cols + 1)));
  SB_CUDA(cudaMemcpyAsync(dX.p, X, dX.bytes(), cudaMemcpyHostToDevice, ctx->stream));
  SB_TRY(predict_contribs_device(m, dX.p, n_rows, n_cols, missing, dout.p));
  SB_CUDA(cudaMemcpyAsync(out, dout.p, dout.bytes(), cudaMemcpyDeviceToHost, ctx->stream));
  SB_CUDA(cudaStreamSynchronize(ctx->stream));
  return SB_OK;
}

int sb_predict_leaf(sb_model* m, const float* X, size_t n_rows, size_t n_cols, float missing, uint32_t* out) {
  using namespace sb;
  SB_REQUIRE(m && (out || n_rows == 0) && (X || n_rows == 0), SB_ERR_INVALID_ARG, "NULL argument");
  SB_REQUIRE(n_cols == (size_t)m->n_features, SB_ERR_DIMENSION,
             "dimension mismatch: expected %d features, got %zu", m->n_features, n_cols);
  sb_ctx* ctx = m->ctx;
  SB_CUDA(cudaSetDevice(ctx->device));
  SB_TRY(model_upload(m));
  const size_t T = (size_t)m->dev.n_trees;
  if (n_rows == 0 || T == 0) return SB_OK;
  const PredDev P = pred_dev(m);
  DBuf<float> dX;
  DBuf<uint32_t> dout;
  SB_TRY(dX.alloc(ctx, n_rows * n_cols));
  SB_TRY(dout.alloc(ctx, n_rows * T));
  SB_CUDA(cudaMemcpyAsync(dX.p, X, dX.bytes(), cudaMemcpyHostToDevice, ctx->stream));
  const size_t tot = n_rows * T;
  SB_REQUIRE((tot + 255) / 256 < (1ull << 31), SB_ERR_UNSUPPORTED, "predict_leaf: %zu outputs exceed one launch", tot);
  SB_LAUNCH(ctx, k_leaf_ids, (unsigned)((tot + 255) / 256), 256, 0, P, dX.p, n_rows, (int)n_cols, missing, dout.p);
  SB_CUDA(cudaMemcpyAsync(out, dout.p, dout.bytes(), cudaMemcpyDeviceToHost, ctx->stream));
  SB_CUDA(cudaStreamSynchronize(ctx->stream));
  return SB_OK;
}

int sb_predict_interactions(sb_model* m, const float* X, size_t n_rows, size_t n_cols, float missing, float* out) {
  using namespace sb;
  SB_REQUIRE(m && (out || n_rows == 0) && (X || n_rows == 0), SB_ERR_INVALID_ARG, "NULL argument");
  SB_REQUIRE(n_cols == (size_t)m->n_features, SB_ERR_DIMENSION,
             "dimension mismatch: expected %d features, got %zu", m->n_features, n_cols);
  if (n_rows == 0) return SB_OK;
  sb_ctx* ctx = m->ctx;
  SB_CUDA(cudaSetDevice(ctx->device));
  const int K = m->num_class >= 2 ? m->num_class : 1;
  const size_t WW = (n_cols + 1) * (n_cols + 1);
  DBuf<float> dX, dout;
  SB_TRY(dX.alloc(ctx, n_rows * n_cols));
  SB_TRY(dout.alloc(ctx, n_rows * K * WW));
  SB_CUDA(cudaMemcpyAsync(dX.p, X, dX.bytes(), cudaMemcpyHostToDevice, ctx->stream));
  SB_TRY(predict_interactions_device(m, dX.p, n_rows, n_cols, missing, dout.p));
  SB_CUDA(cudaMemcpyAsync(out, dout.p, dout.bytes(), cudaMemcpyDeviceToHost, ctx->stream));
  SB_CUDA(cudaStreamSynchronize(ctx->stream));
  return SB_OK;
}

}  // extern "C"
