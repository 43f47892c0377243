// Training-loop kernels for sm_103a (everything except the histogram build).
//
//   gradients      ComputeObjectiveGradients + ApplySampleWeights (trainer.cpp:178-216),
//                  FP64 math rounded once to FP32 pairs, plus per-tree max|g| / max h for
//                  the fixed-point scales.
//                  The last CTA sets the round up: fixed-point exponents, root nodes,
//                  level-0 build list.
//   zero_slots     clears a level's histogram slots; root slots start from the count and
//                  hessian histograms that root_cache kept from a fit's first round
//                  (objectives whose hessian does not depend on the prediction).
//   root_stats     root statistics from the root histogram; root leaf value
//                  (TreeTrainingAccess::Create, tree_structure.cpp:104-116), where the
//                  root's split scan does not form them.
//   subtract       SubtractHistograms (tree_histogram.cpp:16-66): exact int64 in fixed
//                  mode, FP64 with the Hessian clamp in float mode.
//   split_screen, split_exact, split_scan
//                  FindBestSplit (tree_split.cpp:142-234): prefix sums over a feature's
//                  slots, FP64 gains with both missing directions, random threshold,
//                  monotone and interaction rules; where an FP32 screen can rule candidates
//                  out, in two launches (screen, then the FP64 gains of what is left).
//   finalize       the per-level bookkeeping of TrainLevelWiseRegressionTree
//                  (tree.cpp:67-145): acceptance under max_leaves, ApplySplit
//                  (tree_structure.cpp:118-148), smaller-child selection, next level.
//   partition      PrepareSplitRows' stable partition (tree_split.cpp:273-289) as a
//                  ballot/popc compaction: count, per-node scan, scatter, in one cluster
//                  launch for small levels.
//   apply_leaves, apply_steps
//                  predictions += lr * leaf (trainer.cpp:256-262) from the final row
//                  segments: no tree traversal; the round's trees into the model.
#include <algorithm>
#include <cfloat>
#include <type_traits>

#include "device.cuh"
#include "kernels.h"

namespace mpsb {
namespace {

__device__ __forceinline__ void raise(Control* ctl, uint32_t bits) { atomicOr(&ctl->error, bits); }

__device__ __forceinline__ uint32_t ceil_div(uint32_t a, uint32_t b) { return (a + b - 1) / b; }

// The dataset's feature behind a tree's feature f (compact forests number a tree's own).
__device__ __forceinline__ uint32_t dataset_feature(const TrainerDev& a, uint32_t tree, uint32_t f) {
  return a.feature_of ? a.feature_of[size_t(tree) * a.features + f] : f;
}

constexpr uint64_t kLongItemRows = 12288;

// Work items per SM a level is cut into. u8 datasets: three, two while the level has fewer
// than eight nodes. Wide ones: one, because each of an item's passes zeroes and flushes
// 200 KB whatever its rows (three items: 12.5 -> 10.2 ms for 1,000,000 x 64 at 1,024 bins
// with one, 18.7 -> 15.7 at 2,000, 8.3 -> 7.7 at 300, each before the whole waves below).
__device__ __forceinline__ uint32_t level_items_per_sm(const TrainerDev& a, uint32_t nodes) {
  const uint32_t base = a.items_per_sm ? a.items_per_sm : default_items_per_sm(a.slots);
  return nodes < 8 && base > 2 ? base - 1 : base;
}

// Rows per histogram work item for a level that builds `rows` rows of `nodes` nodes: about
// per_sm items per SM, a multiple of 512, within [1024, item_rows_max]. Every node's last item
// is cut short, by half on average, so that many items fewer are aimed at: without that a
// level overshoots its multiple of the SM count and ends in a wave of a few items
// (one-vs-rest of ten classes 15.1 -> 14.5 ms, 1,024 bins 9.9 -> 9.4). One more per SM from
// eight nodes on where the items still hold kLongItemRows rows: a large level ends more evenly
// with more of them, and their flushes hardly count (20 trees of 10,000,000 x 128 77.26 ms
// without, 76.54 with; 8,000,000 x 128 unweighted 51.75 and 51.35, 6,000,000 x 100 53.53 and
// 53.40, one-vs-rest of ten classes 14.72 and 14.62, of eight on 700,000 rows 11.77 and 11.88;
// each the median of four runs in turn). Where the upper end forces more items, their number is
// raised to the next multiple of the SM count, so that the persistent CTAs end the level
// together. At the lower end an item's
// reductions (about 1.5 us) weigh as much as its flush: 100,000 x 32, depth 6, 50 trees
// take 17.5, 17.3, 17.7 and 18.7 ms with items of 512, 1,024, 2,048 and 4,096 rows.
__device__ __forceinline__ uint32_t adaptive_item_rows(uint64_t rows, const TrainerDev& a, uint32_t per_sm,
                                                      uint32_t nodes) {
  const uint64_t n_sm = a.sm_count ? a.sm_count : 152;
  const uint32_t nfb = a.nfb;
  const uint32_t most = a.item_rows_max ? a.item_rows_max : kItemRowsMax;
  if (a.slots == uint32_t(kSlots) && nodes >= 8 && rows * nfb >= kLongItemRows * n_sm * (per_sm + 1)) ++per_sm;
  uint64_t target = n_sm * per_sm;
  if (uint64_t(nodes) * nfb <= target) target -= uint64_t(nodes) * nfb / 2;
  const uint64_t min_items = (rows * nfb + most - 1) / most;
  if (target < min_items) target = (min_items + n_sm - 1) / n_sm * n_sm;
  uint64_t per = (rows * nfb + target - 1) / target;
  per = (per + 511) / 512 * 512;
  if (per < 1024) per = 1024;
  if (per > most) per = most;
  return uint32_t(per);
}

// Exponent e with x < 2^e (frexp convention) of a positive finite float.
__device__ __forceinline__ int exponent_above(float x) {
  const uint32_t bits = __float_as_uint(x), field = bits >> 23;
  return field ? int(field) - 126 : 32 - __clz(int(bits)) - 149;
}

// 2^k for -1022 <= k <= 1023.
__device__ __forceinline__ double exp2_int(int k) {
  return __longlong_as_double((long long)(1023 + k) << 52);
}

// Block-wide exclusive scan of N values per thread. `sh` holds >= 33*N words.
template <int N>
__device__ void block_scan(uint32_t (&v)[N], uint32_t (&total)[N], uint32_t* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  uint32_t incl[N];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    uint32_t x = v[k];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
      if (lane >= off) x += y;
    }
    incl[k] = x;
    if (lane == 31) sh[warp * N + k] = x;
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      uint32_t x = lane < nwarps ? sh[lane * N + k] : 0u;
      const uint32_t own = x;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
      }
      if (lane < nwarps) sh[lane * N + k] = x - own;
      if (lane == 31) sh[32 * N + k] = x;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; ++k) {
    total[k] = sh[32 * N + k];
    v[k] = sh[warp * N + k] + incl[k] - v[k];
  }
  __syncthreads();
}

// ------------------------------------------------------------------------------------
// Gradients and round setup
// ------------------------------------------------------------------------------------
__device__ __forceinline__ double logistic_probability(double m) {  // objective.cpp:309-317
  if (m >= 0.0) {
    const double e = exp(-m);
    return __ddiv_rn(1.0, __dadd_rn(1.0, e));
  }
  const double e = exp(m);
  return __ddiv_rn(e, __dadd_rn(1.0, e));
}

// Objective gradient of one row (objective.cpp:290-429). Returns false on a reference
// TrainingError condition. Finiteness tests read the exponent bits (integer pipe); the
// FP64 pipe does only the arithmetic the reference rounds.
__device__ __forceinline__ bool objective_pair(uint32_t objective, double y, double p,
                                               const TreeParams& prm, double* g, double* h) {
  if (!f64_finite(y) || !f64_finite(p)) return false;
  switch (objective) {
    case 0:
      *g = __dadd_rn(p, -y);
      *h = 1.0;
      return f64_finite(*g);
    case 1: {
      if (y != 0.0 && y != 1.0) return false;
      const double t = __longlong_as_double(__double_as_longlong(p) & 0x7FFFFFFFFFFFFFFFll);  // |p|
      if (t <= kExpFixedMax) {
        // The label's side needs no subtraction: g = prob or -(1 - prob).
        double small, big;
        logistic_fixed(t, &small, &big, h);
        const bool negative = __double_as_longlong(p) < 0;
        *g = y == 0.0 ? (negative ? small : big) : (negative ? -big : -small);
        return true;
      }
      const double prob = logistic_probability(p);
      *g = __dadd_rn(prob, -y);
      *h = __dmul_rn(prob, __dadd_rn(1.0, -prob));
      return isfinite(*g) && isfinite(*h) && *h >= 0.0;
    }
    case 2:
      *g = p < y ? -prm.objective_alpha : __dadd_rn(1.0, -prm.objective_alpha);
      *h = 1.0;
      return true;
    case 3: {
      if (y < 0.0 || p > 709.0) return false;
      const double mean = exp(p);
      *g = __dadd_rn(mean, -y);
      *h = mean;
      return isfinite(*g) && isfinite(*h) && *h > 0.0;
    }
    case 4: {
      const double rho = prm.tweedie_variance_power;
      const double a1 = __dmul_rn(__dadd_rn(2.0, -rho), p);
      const double a2 = __dmul_rn(__dadd_rn(1.0, -rho), p);
      if (y < 0.0 || a1 > 709.0 || a2 > 709.0) return false;
      const double first = exp(a1), second = exp(a2);
      *g = __dadd_rn(first, -__dmul_rn(y, second));
      *h = __dadd_rn(__dmul_rn(__dadd_rn(2.0, -rho), first),
                     -__dmul_rn(__dmul_rn(__dadd_rn(1.0, -rho), y), second));
      return isfinite(*g) && isfinite(*h) && *h > 0.0;
    }
    default:
      return false;
  }
}

// ComputeMulticlassSoftmaxGradients for one row (objective.cpp:130-152, 242-287): the
// class probability from the row's K margins (exp of each margin minus the maximum,
// normalized by their sum in class order), g = p - [label == target], h = p (1 - p).
__device__ __forceinline__ bool softmax_pair(const TrainerDev& a, double label, uint32_t row,
                                             uint32_t target, double* g, double* h) {
  const uint32_t K = a.n_classes;
  if (!f64_finite(label) || floor(label) != label || label < 0.0 || label >= double(K)) return false;
  double maximum = -INFINITY;
  for (uint32_t k = 0; k < K; ++k) {
    const double m = a.preds[size_t(k) * a.n_rows + row];
    if (!f64_finite(m)) return false;
    maximum = fmax(maximum, m);
  }
  double normalizer = 0.0, target_exp = 0.0;
  for (uint32_t k = 0; k < K; ++k) {
    const double e = exp_neg(__dadd_rn(maximum, -a.preds[size_t(k) * a.n_rows + row]));
    normalizer = __dadd_rn(normalizer, e);
    if (k == target) target_exp = e;
  }
  if (!f64_finite(normalizer) || normalizer <= 0.0) return false;
  const double p = __ddiv_rn(target_exp, normalizer);
  *g = __dadd_rn(p, uint32_t(label) == target ? -1.0 : 0.0);
  *h = __dmul_rn(p, __dadd_rn(1.0, -p));
  return f64_finite(*g) && f64_finite(*h) && *h >= 0.0;
}

// x / y for the split screen: the fast reciprocal division (within 2 ulp) where the
// divisor is a normal float below 2^125, the IEEE division elsewhere.
__device__ __forceinline__ float screen_div(float x, float y) {
  return (y > 0x1p-125f && y < 0x1p125f) ? __fdividef(x, y) : __fdiv_rn(x, y);
}

// True for a double with the sign bit set and a non-zero magnitude (x < 0).
__device__ __forceinline__ bool f64_negative(double x) {
  const long long b = __double_as_longlong(x);
  return b < 0 && (b & 0x7FFFFFFFFFFFFFFFll) != 0;
}

__device__ __forceinline__ uint32_t root_rows(const TrainerDev& a, uint32_t t) {
  return a.sample_rows ? a.sample_count[t] : a.n_rows;
}

// The round's start, by one CTA once every gradient is known: fixed-point exponents, slots,
// root nodes and the level-0 build list. Tree t's root takes slot t. g_only: the roots'
// count and hessian histograms come from the fit's first round.
__device__ __noinline__ void round_setup(const TrainerDev& a, bool g_only) {
  for (uint32_t i = threadIdx.x; i < a.n_slots; i += blockDim.x) a.free_stack[i] = a.n_slots - 1 - i;
  if (threadIdx.x == 0) {  // trees are few: serial prefix of the roots' work items
    uint64_t total = 0;
    for (uint32_t t = 0; t < a.n_trees; ++t) total += root_rows(a, t);
    const uint32_t item_rows =
        a.item_rows ? a.item_rows : adaptive_item_rows(total, a, a.items_per_sm ? a.items_per_sm : default_items_per_sm(a.slots), a.n_trees);
    uint32_t acc = 0;
    for (uint32_t t = 0; t < a.n_trees; ++t) {
      a.build_prefix[t] = acc;
      acc += ceil_div(root_rows(a, t), item_rows);
    }
    a.build_prefix[a.n_trees] = acc;
    a.ctl->free_top = a.n_slots - a.n_trees;
    a.ctl->n_leafseg = 0;
    a.ctl->leaf_chunks = 0;
    a.leaf_prefix[0] = 0;
    a.ctl->round = *a.round_counter;
    a.ctl->n_nodes = a.n_trees;
    a.ctl->n_build = a.n_trees;
    a.ctl->n_sub = 0;
    a.ctl->n_part = 0;
    a.ctl->hist_items = acc * a.nfb;
    a.ctl->hist_counter = 0;
    a.ctl->item_rows = item_rows;
  }
  if (threadIdx.x >= 32) {  // beside warp 0's work items
    for (uint32_t t = threadIdx.x - 32; t < a.n_trees; t += blockDim.x - 32) {
      TreeState& s = a.trees[t];
      const float mg = __uint_as_float(__ldcg(&s.max_abs_g_bits)), mh = __uint_as_float(__ldcg(&s.max_h_bits));
      s.max_abs_g_bits = s.max_h_bits = 0;  // the next round's maxima start here
      s.n_tree_nodes = 1;
      s.leaf_count = 1;
      // every row's |q| <= 2^30: the histogram's 32-bit limb sums cannot overflow
      s.kg = mg > 0.0f ? 30 - exponent_above(mg) : 0;
      s.kh = mh > 0.0f ? 30 - exponent_above(mh) : 0;
      s.inv_g = exp2_int(-s.kg);  // |k| <= 179: a float's exponent and the 30 bits
      s.inv_h = exp2_int(-s.kh);
      if (g_only && a.root_cache_kh[t] != s.kh) raise(a.ctl, kErrRootCache);
      const uint32_t slot = t;
      const uint32_t cnt = root_rows(a, t);
      NodeRec r;
      r.seg_off = 0;
      r.seg_cnt = cnt;
      r.node_index = 0;
      r.slot = slot;
      r.count = 0;
      r.qg = r.qh = 0;
      r.g = r.h = 0.0;
      r.lo = -INFINITY;
      r.hi = INFINITY;
      r.tree = t;
      r.depth = 0;
      r.sub_from = 0;
      a.nodes[0][t] = r;
      for (uint32_t w = 0; w < a.params.path_words; ++w) {
        uint32_t allowed = 0xffffffffu;
        if (a.params.n_groups > 0) {  // empty path: any group containing the feature
          allowed = 0;
          for (uint32_t g = 0; g < a.params.n_groups; ++g)
            allowed |= a.group_masks[g * a.params.path_words + w];
        }
        if (a.tree_feature_masks != nullptr)
          allowed &= a.tree_feature_masks[t * a.params.path_words + w];
        a.node_path[0][t * a.params.path_words + w] = 0;
        a.node_allowed[0][t * a.params.path_words + w] = allowed;
      }
      BuildEntry e;
      e.tree = t;
      e.parity = 0;
      e.seg_off = 0;
      e.seg_cnt = cnt;
      e.slot = slot;
      e.pad = 0;
      a.build[t] = e;
    }
  }
}

// grid = (x, n_trees): blockIdx.y is the tree, so a block's maxima belong to one tree.
// SQ: squared error without softmax classes only; the instantiation leaves out the other
// objectives' code, so it needs fewer registers and more rows are in flight per SM.
// The last CTA to finish sets the round up.
template <bool SQ>
__global__ void __launch_bounds__(256, SQ ? 8 : 4) gradients_kernel(const __grid_constant__ TrainerDev a, bool g_only) {
  __shared__ uint32_t sg[8], shh[8], s_last;
  const uint32_t t = blockIdx.y;
  const size_t tree_off = size_t(t) * a.n_rows;
  // Squared error and quantile have h = 1, so h * w = w exactly.
  const bool unit_h = !a.n_classes && (a.objective == 0 || a.objective == 2);
  const long long class_bits = __double_as_longlong(double(t));
  uint32_t mg = 0, mh = 0, bad = 0;
  // Position p of the tree's root segment holds row i: the identity for boosting, the
  // tree's sample for a forest.
  const uint32_t count = a.sample_rows ? a.sample_count[t] : a.n_rows;
  const size_t pos_off = size_t(t) * 2 * a.seg_stride;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < count; p += gridDim.x * blockDim.x) {
    const uint32_t i = a.sample_rows ? a.sample_rows[size_t(t) * a.seg_stride + p] : p;
    if (i >= a.n_rows) {
      bad = 1;
      continue;
    }
    double y = a.labels[i];
    if (a.ovr) {  // y == t (class ids are non-negative integers; -0.0 equals class 0)
      const long long yb = __double_as_longlong(y);
      y = (yb == class_bits || (t == 0 && (yb << 1) == 0)) ? 1.0 : 0.0;
    }
    double g = 0.0, h = 0.0;
    if (SQ || (a.objective == 0 && !a.n_classes)) {
      // Squared error (the objective_pair case 0 then the weight products): g = w (p - y),
      // h = w; two FP64 operations per row on the narrow FP64 pipe.
      const double pred = a.preds ? a.preds[tree_off + i] : a.tree_base[t];
      g = __dsub_rn(pred, y);  // p + (-y): negation is exact
      if (!f64_finite(y) || !f64_finite(pred) || !f64_finite(g)) bad = 1;
      h = 1.0;
      if (a.weights != nullptr) {
        const double w = a.weights_per_tree ? a.weights[tree_off + i] : a.weights[i];
        g = __dmul_rn(g, w);
        h = w;
        if (!f64_finite(g) || !f64_finite(h) || f64_negative(h)) bad = 1;
      }
    } else if constexpr (!SQ) {
      if (a.n_classes) {
        if (!softmax_pair(a, y, i, *a.round_counter % a.n_classes, &g, &h)) bad = 1;
      } else {
        const double pred = a.preds ? a.preds[tree_off + i] : a.tree_base[t];
        if (!objective_pair(a.objective, y, pred, a.params, &g, &h)) bad = 1;
      }
      if (a.weights != nullptr) {
        const double w = a.weights_per_tree ? a.weights[tree_off + i] : a.weights[i];
        g = __dmul_rn(g, w);
        h = unit_h ? w : __dmul_rn(h, w);
        if (!f64_finite(g) || !f64_finite(h) || f64_negative(h)) bad = 1;
      }
    }
    const float g32 = f64_to_f32_rn(g), h32 = f64_to_f32_rn(h);
    if (!isfinite(g32) || !isfinite(h32)) bad = 1;
    a.gh[pos_off + p] = make_float2(g32, h32);  // parity 0 = the root segment's order
    a.rows[pos_off + p] = i;
    mg = max(mg, __float_as_uint(fabsf(g32)));
    mh = max(mh, __float_as_uint(fmaxf(h32, 0.0f)));
  }
  for (int off = 16; off > 0; off >>= 1) {
    mg = max(mg, __shfl_xor_sync(0xffffffffu, mg, off));
    mh = max(mh, __shfl_xor_sync(0xffffffffu, mh, off));
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    sg[warp] = mg;
    shh[warp] = mh;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < int(blockDim.x >> 5); ++w) {
      mg = max(mg, sg[w]);
      mh = max(mh, shh[w]);
    }
    atomicMax(&a.trees[t].max_abs_g_bits, mg);
    atomicMax(&a.trees[t].max_h_bits, mh);
    __threadfence();
    s_last = atomicAdd(&a.ctl->grad_ticket, 1u) == gridDim.x * gridDim.y - 1 ? 1u : 0u;
  }
  if (bad) raise(a.ctl, kErrGradient);
  __syncthreads();
  if (s_last) {
    __threadfence();
    if (threadIdx.x == 0) a.ctl->grad_ticket = 0;
    round_setup(a, g_only);
  }
}

// Clears the histogram slots of the current build list (kZeroBuilt) or of the trees' roots
// (kZeroRoots: tree t's slot t, before the round's lists exist, beside the gradients).
// kRestoreRoots: the root of every tree holds all rows in every round, so its count
// histogram never changes, and when the hessian does not depend on the prediction (squared
// error and quantile: h = weight) neither does its hessian histogram, nor the hessian scale.
// The first round of a fit builds the roots in full and saves those two words per cell;
// later rounds start the roots from them and build only the gradient limbs. The hessian
// scale is checked by the round's setup.
enum : int { kZeroBuilt = 0, kZeroRoots = 1, kRestoreRoots = 2 };

__global__ void zero_slots_kernel(TrainerDev a, int what) {
  // The level's split scan publishes node maxima into node_screen: clear them first.
  if (a.node_screen)
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.max_level_nodes; i += gridDim.x * blockDim.x)
      a.node_screen[i] = 0u;
  const uint64_t words_per_slot = uint64_t(a.features) * a.slots * 3;
  if (what == kRestoreRoots) {
    // Pairs of cells: their two {count, hessian} words each, into 48 bytes.
    const uint64_t total = uint64_t(a.n_trees) * (words_per_slot / 6);
    for (uint64_t idx = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; idx < total;
         idx += uint64_t(gridDim.x) * blockDim.x) {
      const ulonglong2* cache = reinterpret_cast<const ulonglong2*>(a.root_cache + idx * 4);
      const ulonglong2 c0 = cache[0], c1 = cache[1];
      ulonglong2* out = reinterpret_cast<ulonglong2*>(a.hist + idx * 6);  // tree t's root slot is t
      out[0] = make_ulonglong2(c0.x, 0);
      out[1] = make_ulonglong2(c0.y, c1.x);
      out[2] = make_ulonglong2(0, c1.y);
    }
    return;
  }
  const uint64_t total = uint64_t(what == kZeroBuilt ? a.ctl->n_build : a.n_trees) * (words_per_slot / 2);
  for (uint64_t idx = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; idx < total;
       idx += uint64_t(gridDim.x) * blockDim.x) {
    const uint32_t e = uint32_t(idx / (words_per_slot / 2));
    const uint64_t w = idx - e * (words_per_slot / 2);
    // A node of one row chunk is stored by its work items, not added.
    if (what == kZeroBuilt && a.store_single && a.build_prefix[e + 1] - a.build_prefix[e] == 1) continue;
    if (a.tree_feature_masks) {
      // A forest tree reads only its own features' histograms (and feature 0's, for the
      // root statistics): the others are neither cleared nor subtracted nor scanned.
      const uint32_t f = uint32_t(w * 2 / (a.slots * 3));
      const uint32_t tree = what == kZeroBuilt ? a.build[e].tree : e;
      const uint32_t mask = a.tree_feature_masks[size_t(tree) * a.params.path_words + (f >> 5)];
      if (f != 0 && !((mask >> (f & 31)) & 1u)) continue;
    }
    const uint32_t slot = what == kZeroBuilt ? a.build[e].slot : e;
    reinterpret_cast<ulonglong2*>(a.hist + slot * words_per_slot)[w] = make_ulonglong2(0, 0);
  }
}

// Saves the roots' count and hessian words of a fit's first round (kRestoreRoots).
__global__ void root_cache_kernel(TrainerDev a) {
  const uint64_t per_tree = uint64_t(a.features) * a.slots;
  const uint64_t total = per_tree * a.n_trees;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < total;
       i += uint64_t(gridDim.x) * blockDim.x) {
    const unsigned long long* slot = a.hist + i * 3;  // tree t's root slot is t
    a.root_cache[i * 2] = slot[0];
    a.root_cache[i * 2 + 1] = slot[2];
    if (i % per_tree == 0) a.root_cache_kh[i / per_tree] = a.trees[i / per_tree].kh;
  }
}

// The root's leaf: tree t's node 0 (TreeTrainingAccess::Create, tree_structure.cpp:104-116).
__device__ __forceinline__ void write_root_leaf(const TrainerDev& a, uint32_t t, double g, double h) {
  double leaf = 0.0;
  if (!leaf_weight(g, h, a.params, &leaf)) raise(a.ctl, kErrNonFinite);
  TreeNodeOut n;
  n.feature_index = 0;
  n.threshold_bin = 0;
  n.left_child = 0xffffffffu;
  n.right_child = 0xffffffffu;
  n.leaf_value = leaf;
  n.gain = 0.0;
  n.default_left = 1;
  n.flags = 1;
  for (int k = 0; k < 6; ++k) n.reserved[k] = 0;
  a.tree_nodes[size_t(t) * a.max_tree_nodes] = n;
}

// Root statistics: the total of feature 0's slots (all rows, exact in fixed mode), where
// the root's split scan does not form them itself.
__global__ void root_stats_kernel(TrainerDev a) {
  const int lane = threadIdx.x & 31;
  for (uint32_t t = threadIdx.x >> 5; t < a.n_trees; t += blockDim.x >> 5) {
    NodeRec& r = a.nodes[0][t];
    const unsigned long long* base = a.hist + size_t(r.slot) * a.features * a.slots * 3;
    unsigned long long cnt = 0;
    long long qg = 0, qh = 0;
    for (uint32_t s = lane; s < a.slots; s += 32) {
      cnt += base[s * 3 + 0];
      qg += (long long)base[s * 3 + 1];
      qh += (long long)base[s * 3 + 2];
    }
    for (int off = 16; off > 0; off >>= 1) {
      cnt += __shfl_xor_sync(0xffffffffu, cnt, off);
      qg += __shfl_xor_sync(0xffffffffu, qg, off);
      qh += __shfl_xor_sync(0xffffffffu, qh, off);
    }
    if (lane == 0) {
      const TreeState& st = a.trees[t];
      r.count = cnt;
      if (a.mode == kModeFixed) {
        r.qg = qg;
        r.qh = qh;
        r.g = q_image(qg, st.inv_g);
        r.h = q_image(qh, st.inv_h);
      } else {  // FP64 total in slot order
        double g = 0.0, h = 0.0;
        for (uint32_t s = 0; s < a.slots; ++s) {
          g = __dadd_rn(g, __longlong_as_double((long long)base[s * 3 + 1]));
          h = __dadd_rn(h, __longlong_as_double((long long)base[s * 3 + 2]));
        }
        r.g = g;
        r.h = h;
      }
      if (cnt != r.seg_cnt) raise(a.ctl, kErrCountMismatch);
      write_root_leaf(a, t, r.g, r.h);
    }
  }
}

// slot_parent := slot_parent - slot_built for every pair (the parent slot becomes the
// sibling's histogram).
__global__ void subtract_kernel(TrainerDev a) {
  const uint64_t bins_per_slot = uint64_t(a.features) * a.slots;
  const uint64_t total = uint64_t(a.ctl->n_sub) * bins_per_slot;
  uint32_t err = 0;
  for (uint64_t idx = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; idx < total;
       idx += uint64_t(gridDim.x) * blockDim.x) {
    const SubEntry e = a.sub[idx / bins_per_slot];
    const uint64_t b = idx % bins_per_slot;
    if (a.tree_feature_masks) {  // a forest tree's own features only (sub[k] pairs build[k])
      const uint32_t f = uint32_t(b / a.slots);
      const uint32_t mask =
          a.tree_feature_masks[size_t(a.build[idx / bins_per_slot].tree) * a.params.path_words + (f >> 5)];
      if (!((mask >> (f & 31)) & 1u)) continue;
    }
    unsigned long long* p = a.hist + (e.parent_slot * bins_per_slot + b) * 3;
    const unsigned long long* c = a.hist + (e.built_slot * bins_per_slot + b) * 3;
    const unsigned long long pc = p[0], cc = c[0];
    if (cc > pc) err |= kErrSubtraction;
    p[0] = pc - cc;
    if (a.mode == kModeFixed) {
      p[1] = p[1] - c[1];
      p[2] = p[2] - c[2];
    } else {
      const double pg = __longlong_as_double((long long)p[1]);
      const double cg = __longlong_as_double((long long)c[1]);
      const double g = __dadd_rn(pg, -cg);
      if (!isfinite(pg) || !isfinite(cg) || !isfinite(g)) err |= kErrNonFinite;
      const double ph = __longlong_as_double((long long)p[2]);
      const double ch = __longlong_as_double((long long)c[2]);
      if (!isfinite(ph) || !isfinite(ch) || ph < 0.0 || ch < 0.0) err |= kErrHessian;
      const double diff = __dadd_rn(ph, -ch);
      const double tol = __dmul_rn(1e-5, fmax(1.0, fmax(fabs(ph), fabs(ch))));
      if (diff < -tol) err |= kErrSubtraction;
      p[1] = (unsigned long long)__double_as_longlong(g);
      p[2] = (unsigned long long)__double_as_longlong(diff < 0.0 ? 0.0 : diff);
    }
  }
  if (err) raise(a.ctl, err);
}

// ------------------------------------------------------------------------------------
// Split scan
// ------------------------------------------------------------------------------------
// Node statistics of the scan: exact int64 (fixed) or FP64 (float).
template <bool FIXED>
struct Stat {
  using V = typename std::conditional<FIXED, long long, double>::type;
  uint32_t count;  // a node holds fewer than 2^32 rows
  V g, h;
};

template <bool FIXED>
__device__ __forceinline__ Stat<FIXED> stat_zero() {
  Stat<FIXED> r;
  r.count = 0;
  r.g = 0;
  r.h = 0;
  return r;
}

template <bool FIXED>
__device__ __forceinline__ Stat<FIXED> stat_add(Stat<FIXED> x, Stat<FIXED> y) {
  Stat<FIXED> r;
  r.count = x.count + y.count;
  if constexpr (FIXED) {
    r.g = x.g + y.g;
    r.h = x.h + y.h;
  } else {
    r.g = __dadd_rn(x.g, y.g);
    r.h = __dadd_rn(x.h, y.h);
  }
  return r;
}

template <bool FIXED>
__device__ __forceinline__ Stat<FIXED> stat_sub(Stat<FIXED> x, Stat<FIXED> y) {
  Stat<FIXED> r;
  r.count = x.count - y.count;
  if constexpr (FIXED) {
    r.g = x.g - y.g;
    r.h = x.h - y.h;
  } else {
    r.g = __dadd_rn(x.g, -y.g);
    r.h = __dadd_rn(x.h, -y.h);
  }
  return r;
}

template <bool FIXED>
__device__ __forceinline__ Stat<FIXED> shfl_up_stat(Stat<FIXED> s, int off) {
  Stat<FIXED> r;
  r.count = __shfl_up_sync(0xffffffffu, s.count, off);
  r.g = __shfl_up_sync(0xffffffffu, s.g, off);
  r.h = __shfl_up_sync(0xffffffffu, s.h, off);
  return r;
}

template <bool FIXED>
__device__ __forceinline__ Stat<FIXED> shfl_stat(Stat<FIXED> s, int src) {
  Stat<FIXED> r;
  r.count = __shfl_sync(0xffffffffu, s.count, src);
  r.g = __shfl_sync(0xffffffffu, s.g, src);
  r.h = __shfl_sync(0xffffffffu, s.h, src);
  return r;
}

// q_image(x) > q_image(y), out of line: the FP64 conversions are not speculated into
// the common case.
static __device__ __noinline__ bool images_above(long long x, long long y, double inv) {
  return q_image(x, inv) > q_image(y, inv);
}

template <bool FIXED>
__device__ __forceinline__ double image(typename Stat<FIXED>::V v, double inv) {
  if constexpr (FIXED) return q_image(v, inv);
  else return v;
}

// ConsiderMissingDirection (tree_split.cpp:65-115): the FP64 gain of one candidate; false
// where the reference rejects it.
template <bool FIXED>
__device__ __forceinline__ bool exact_gain(const TreeParams& p, const Stat<FIXED>& cl,
                                           const Stat<FIXED>& cr, double inv_g, double inv_h,
                                           int8_t mono, double plo, double phi, double* gain_out,
                                           uint32_t& err) {
  if (cl.count < p.min_samples_leaf || cr.count < p.min_samples_leaf) return false;
  const double lh = image<FIXED>(cl.h, inv_h), rh = image<FIXED>(cr.h, inv_h);
  if (lh < p.min_child_weight || rh < p.min_child_weight || lh <= 0.0 || rh <= 0.0) return false;
  const double lg = image<FIXED>(cl.g, inv_g), rg = image<FIXED>(cr.g, inv_g);
  double gain;
  if (!split_gain(lg, lh, rg, rh, p, &gain)) {
    err |= kErrNonFinite;
    return false;
  }
  if (gain <= 0.0 || gain < p.min_gain_to_split) return false;
  if (mono != 0) {
    double lv, rv;
    if (!leaf_weight(lg, lh, p, &lv) || !leaf_weight(rg, rh, p, &rv)) {
      err |= kErrNonFinite;
      return false;
    }
    lv = clamp_bounds(lv, plo, phi);
    rv = clamp_bounds(rv, plo, phi);
    if (mono > 0 ? lv > rv : lv < rv) return false;
  }
  *gain_out = gain;
  return true;
}

// The record of an accepted candidate, with MonotonicBoundsForSplit (tree_monotonic.cpp:
// 12-58); the leaf weights repeat exact_gain's operations.
template <bool FIXED>
__device__ __forceinline__ SplitRec split_record(const TreeParams& p, const Stat<FIXED>& cl,
                                                 const Stat<FIXED>& cr, double inv_g, double inv_h,
                                                 int8_t mono, double plo, double phi, double gain,
                                                 uint32_t feature, uint32_t threshold,
                                                 uint32_t default_left) {
  SplitRec c;
  c.gain = gain;
  c.valid = 1;
  c.feature = feature;
  c.threshold = threshold;
  c.default_left = default_left;
  c.lcount = cl.count;
  c.rcount = cr.count;
  if constexpr (FIXED) {
    c.lqg = cl.g;
    c.lqh = cl.h;
    c.rqg = cr.g;
    c.rqh = cr.h;
  } else {
    c.lqg = c.lqh = c.rqg = c.rqh = 0;
  }
  c.lg = image<FIXED>(cl.g, inv_g);
  c.lh = image<FIXED>(cl.h, inv_h);
  c.rg = image<FIXED>(cr.g, inv_g);
  c.rh = image<FIXED>(cr.h, inv_h);
  c.ll = c.rl = plo;
  c.lu = c.ru = phi;
  if (mono != 0) {
    double lv = 0.0, rv = 0.0;
    leaf_weight(c.lg, c.lh, p, &lv);
    leaf_weight(c.rg, c.rh, p, &rv);
    lv = clamp_bounds(lv, plo, phi);
    rv = clamp_bounds(rv, plo, phi);
    if (mono > 0) {
      c.lu = (rv < c.lu) ? rv : c.lu;  // std::min(lu, rv)
      c.rl = (c.rl < lv) ? lv : c.rl;  // std::max(rl, lv)
    } else {
      c.ll = (c.ll < rv) ? rv : c.ll;  // std::max(ll, rv)
      c.ru = (lv < c.ru) ? lv : c.ru;  // std::min(ru, lv)
    }
  }
  return c;
}

template <bool FIXED>
__device__ __forceinline__ void consider(const TreeParams& p, const Stat<FIXED>& cl,
                                         const Stat<FIXED>& cr, double inv_g, double inv_h,
                                         int8_t mono, double plo, double phi, uint32_t feature,
                                         uint32_t threshold, uint32_t default_left,
                                         SplitRec& best, uint32_t& err) {
  double gain;
  if (!exact_gain<FIXED>(p, cl, cr, inv_g, inv_h, mono, plo, phi, &gain, err)) return;
  const SplitRec c = split_record<FIXED>(p, cl, cr, inv_g, inv_h, mono, plo, phi, gain, feature,
                                         threshold, default_left);
  if (better_split(c, best)) best = c;
}

// ---- FP32 screen ---------------------------------------------------------------------
// Every eligible candidate's score S = gL^2/(hL+lambda) + gR^2/(hR+lambda) is computed in
// FP32 with relative error <= 15u (u = 2^-24; each int64 -> FP32 conversion below is within
// 3u, lambda is rounded once, the approximate reciprocal is within 2u). A candidate whose
// FP32 score is below M(1 - 2^-18), M the best FP32 score of a certainly eligible candidate
// of the node, then has an exact score at least 30u*M below that candidate's, far outside
// the FP64 evaluation's own rounding (a few 2^-53 * M, the parent score included), so its
// FP64 gain is strictly lower and it cannot win. Only the rest -- and candidates whose
// min_child_weight test or score is too close to call in FP32 -- run the FP64 evaluation of
// the reference. The score is quadratic only without reg_alpha, the admissible set monotone
// in it only without monotone constraints, and random thresholds leave one candidate: the
// screen is off for those, and where lambda in hessian quanta leaves a safe range.
//
// Fixed point scores the quantized sums themselves: with lambda and min_child_weight taken
// times 2^kh (a power of two: no rounding), every score of a node is the real one times the
// same power of two, so the comparisons are the same and no sum is scaled. Sums stay below
// 2^62 and an eligible hessian sum is at least 1, so no square, reciprocal or sum leaves the
// FP32 normal range (a zero gradient scores 0).
struct ScreenScale {
  bool on;  // the screen applies to this feature of this node
  float lambda, mcw_lo, mcw_hi;
};

template <bool FIXED>
__device__ __forceinline__ ScreenScale screen_scale(const TreeParams& P, int8_t mono, int kh) {
  ScreenScale s;
  s.on = P.screen_params != 0 && mono == 0;
  float unit = 1.0f;
  if constexpr (FIXED) {
    s.on = s.on && kh >= -120 && kh <= 120;
    unit = s.on ? __int_as_float((127 + kh) << 23) : 1.0f;
  }
  s.lambda = P.screen_lambda * unit;
  if (FIXED && !(s.lambda <= 0x1p100f)) s.on = false;
  // Without a minimum no sum is rejected or close to it.
  s.mcw_lo = P.screen_mcw_on ? P.screen_mcw_lo * unit : -1.0f;
  s.mcw_hi = P.screen_mcw_on ? P.screen_mcw_hi * unit : -1.0f;
  return s;
}

// m as hi * 2^32 + lo: float(hi) and float(lo) are each within u, and the fused
// multiply-add rounds once more, so the result is within 3u (no cancellation: both parts
// are non-negative). The conversions run on the FP32 pipe.
__device__ __forceinline__ float u64_to_f32_3u(unsigned long long m) {
  return __fmaf_rn(u32_to_f32_rn(uint32_t(m >> 32)), 4294967296.0f, u32_to_f32_rn(uint32_t(m)));
}

// 1/y within 2u for a normal y below 2^126.
__device__ __forceinline__ float rcp_approx(float y) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  return r;
}

// 0: rejected by the FP64 test before any arithmetic (no error flag either);
// 1: admissible, FP32 score in *s32; 2: too close to call. msl: min_samples_leaf, at most
// 2^32 - 1 (no node holds more rows).
template <bool FIXED>
__device__ __forceinline__ int screen_classify(uint32_t msl, const ScreenScale& sc,
                                               const Stat<FIXED>& cl, const Stat<FIXED>& cr,
                                               float* s32) {
  if (min(cl.count, cr.count) < msl) return 0;
  if constexpr (FIXED) {
    if (!(cl.h > 0) || !(cr.h > 0)) return 0;  // image > 0 iff q > 0
    const float lh = u64_to_f32_3u((unsigned long long)cl.h), rh = u64_to_f32_3u((unsigned long long)cr.h);
    const float least = fminf(lh, rh);
    if (least < sc.mcw_lo) return 0;
    const float lg = u64_to_f32_3u((unsigned long long)(cl.g < 0 ? -cl.g : cl.g));
    const float rg = u64_to_f32_3u((unsigned long long)(cr.g < 0 ? -cr.g : cr.g));
    *s32 = __fmaf_rn(lg * lg, rcp_approx(lh + sc.lambda), (rg * rg) * rcp_approx(rh + sc.lambda));
    return least <= sc.mcw_hi ? 2 : 1;
  } else {
    if (!f64_finite(cl.h) || !f64_finite(cr.h) || !f64_finite(cl.g) || !f64_finite(cr.g)) return 2;
    if (!(cl.h > 0) || !(cr.h > 0)) return 0;
    const float lh = f64_to_f32_rn(cl.h), rh = f64_to_f32_rn(cr.h);
    const float least = fminf(lh, rh);
    if (least < sc.mcw_lo) return 0;
    const float lg = f64_to_f32_rn(cl.g), rg = f64_to_f32_rn(cr.g);
    const float score = screen_div(lg * lg, lh + sc.lambda) + screen_div(rg * rg, rh + sc.lambda);
    *s32 = score;
    return (least <= sc.mcw_hi || !isfinite(score)) ? 2 : 1;
  }
}

__device__ __forceinline__ uint32_t min_leaf_rows(const TreeParams& P) {
  return uint32_t(P.min_samples_leaf < 0xFFFFFFFFull ? P.min_samples_leaf : 0xFFFFFFFFull);
}

__device__ __forceinline__ SplitRec no_split() {
  SplitRec b;
  b.gain = 0.0;
  b.valid = 0;
  b.feature = b.threshold = 0;
  b.default_left = 1;
  return b;
}

// One warp per (node, feature); a CTA covers one node and blockDim/32 features and
// writes the best split of its features to partial[node][chunk].
constexpr int kScanThreadsMax = 512;
constexpr uint32_t kScanQueue = 32;  // FP64 candidates queued per warp

// A candidate waiting for the exact FP64 evaluation.
template <bool FIXED>
struct ScanCand {
  Stat<FIXED> cl, cr;
  uint32_t threshold, default_left;
};

// A feature's histogram staged in shared memory, [word][k][lane] for slot lane * 8 + k
// (word 0 count, 1 g, 2 h): the lane's eight slots read conflict-free.
constexpr size_t kScanHistBytes = size_t(kSlots) * 3 * sizeof(unsigned long long);

// Shared memory per warp: its best split, its staged histogram and its FP64 queue.
template <bool FIXED>
constexpr size_t scan_smem_per_warp() {
  return sizeof(SplitRec) + kScanHistBytes + kScanQueue * sizeof(ScanCand<FIXED>);
}

// Copies a feature's histogram (kSlots x {count, g, h} 64-bit words, 6 KB, 16-byte
// aligned) into the warp's staging area with coalesced 16-byte loads, all in flight
// together.
__device__ __forceinline__ void stage_feature_hist(const unsigned long long* src,
                                                   unsigned long long* dst, int lane) {
  constexpr int kChunks = int(kScanHistBytes / 16);  // 384
  constexpr int kPerLane = kChunks / 32;              // 12
  constexpr int kBatch = 4;
  const ulonglong2* s2 = reinterpret_cast<const ulonglong2*>(src);
#pragma unroll 1
  for (int part = 0; part < kPerLane / kBatch; ++part) {
    ulonglong2 v[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) v[j] = __ldg(s2 + (part * kBatch + j) * 32 + lane);
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const uint32_t w0 = uint32_t((part * kBatch + j) * 32 + lane) * 2u;
#pragma unroll
      for (uint32_t q = 0; q < 2; ++q) {
        const uint32_t w = w0 + q, slot = w / 3u, word = w - slot * 3u;
        dst[(word * 8u + (slot & 7u)) * 32u + (slot >> 3)] = q ? v[j].y : v[j].x;
      }
    }
  }
  __syncwarp();
}

// One word of a sibling's slot: parent minus built child, with subtract_kernel's checks
// (word 0 count, 1 g, 2 h; count underflow; float mode: finite sums, non-negative hessians, the
// hessian difference clamped at 0 within 1e-5).
template <bool FIXED>
__device__ __forceinline__ unsigned long long sibling_word(unsigned long long pw, unsigned long long cw,
                                                           uint32_t word, uint32_t& err) {
  if (word == 0 || FIXED) {
    if (word == 0 && cw > pw) err |= kErrSubtraction;
    return pw - cw;
  }
  const double pd = __longlong_as_double((long long)pw), cd = __longlong_as_double((long long)cw);
  if (word == 1) {
    const double g = __dadd_rn(pd, -cd);
    if (!isfinite(pd) || !isfinite(cd) || !isfinite(g)) err |= kErrNonFinite;
    return (unsigned long long)__double_as_longlong(g);
  }
  if (!isfinite(pd) || !isfinite(cd) || pd < 0.0 || cd < 0.0) err |= kErrHessian;
  const double diff = __dadd_rn(pd, -cd);
  const double tol = __dmul_rn(1e-5, fmax(1.0, fmax(fabs(pd), fabs(cd))));
  if (diff < -tol) err |= kErrSubtraction;
  return (unsigned long long)__double_as_longlong(diff < 0.0 ? 0.0 : diff);
}

// stage_feature_hist of a sibling's histogram, formed on the way and written back over the
// parent's words in the same 16-byte chunks.
template <bool FIXED>
__device__ __forceinline__ void stage_sibling_hist(unsigned long long* parent,
                                                   const unsigned long long* built,
                                                   unsigned long long* dst, int lane, uint32_t& err) {
  constexpr int kChunks = int(kScanHistBytes / 16);  // 384
  constexpr int kPerLane = kChunks / 32;              // 12
  constexpr int kBatch = 4;
  ulonglong2* p2 = reinterpret_cast<ulonglong2*>(parent);
  const ulonglong2* c2 = reinterpret_cast<const ulonglong2*>(built);
#pragma unroll 1
  for (int part = 0; part < kPerLane / kBatch; ++part) {
    ulonglong2 pv[kBatch], cv[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      pv[j] = p2[(part * kBatch + j) * 32 + lane];
      cv[j] = c2[(part * kBatch + j) * 32 + lane];
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const uint32_t w0 = uint32_t((part * kBatch + j) * 32 + lane) * 2u;
      unsigned long long out[2];
#pragma unroll
      for (uint32_t q = 0; q < 2; ++q) {
        const unsigned long long pw = q ? pv[j].y : pv[j].x, cw = q ? cv[j].y : cv[j].x;
        const uint32_t w = w0 + q, word = w % 3u;
        const unsigned long long r = sibling_word<FIXED>(pw, cw, word, err);
        out[q] = r;
        const uint32_t slot = w / 3u;
        dst[(word * 8u + (slot & 7u)) * 32u + (slot >> 3)] = r;
      }
      p2[(part * kBatch + j) * 32 + lane] = make_ulonglong2(out[0], out[1]);
    }
  }
  __syncwarp();
}

// A feature with at most 32 bins: its slots 0-31 staged one per lane (slot l's words at
// dst[(w * 8) * 32 + l]) and its missing slot returned in *miss_words (every lane). All
// other slots are empty: every bin is below the feature's bin count. sub: parent minus the
// built child (`built`), written back as stage_sibling_hist does.
template <bool FIXED>
__device__ __forceinline__ void stage_few_slots(unsigned long long* slot_hist,
                                                const unsigned long long* built, bool hm,
                                                unsigned long long* dst, int lane,
                                                unsigned long long* miss_words, uint32_t& err) {
#pragma unroll
  for (uint32_t w = 0; w < 3; ++w) {
    const size_t at = size_t(lane) * 3 + w;
    unsigned long long v = slot_hist[at];
    if (built) {
      v = sibling_word<FIXED>(v, built[at], w, err);
      slot_hist[at] = v;
    }
    dst[(w * 8u) * 32u + uint32_t(lane)] = v;
  }
#pragma unroll
  for (uint32_t w = 0; w < 3; ++w) {
    const size_t at = size_t(kMissingSlot) * 3 + w;
    unsigned long long v = 0;
    if (hm) {
      v = slot_hist[at];
      if (built) {
        v = sibling_word<FIXED>(v, built[at], w, err);
        __syncwarp();
        if (lane == 0) slot_hist[at] = v;
      }
    }
    miss_words[w] = v;
  }
  __syncwarp();
}

// The split scan of a level in one launch, one warp per (node, feature), a CTA per (node,
// chunk of blockDim/32 features): where the two-launch scan below does not apply (no FP32
// screen, or the per-feature entry point, which needs every feature's best split). A
// feature the screen does apply to is screened against its own maximum. Each chunk's best
// split goes to partial[node][chunk].
//
// WIDE (a dataset with more than kSlots slots per feature): each warp walks its feature's
// slots in pages of kSlots, first for the total count and the missing slot (the last
// page's slot kMissingSlot), then per scan pass page by page with the left prefix carried
// from page to page; thresholds are numbered across pages.
template <bool FIXED, bool WIDE>
__global__ void __launch_bounds__(kScanThreadsMax) split_scan_kernel(TrainerDev a, int parity) {
  using V = typename Stat<FIXED>::V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  SplitRec* warp_best = reinterpret_cast<SplitRec*>(smem_raw);
  unsigned long long* s_hist =
      reinterpret_cast<unsigned long long*>(smem_raw + sizeof(SplitRec) * nwarps);
  ScanCand<FIXED>* s_queue = reinterpret_cast<ScanCand<FIXED>*>(
      smem_raw + (sizeof(SplitRec) + kScanHistBytes) * nwarps);
  static_assert(sizeof(SplitRec) % 8 == 0, "staged words and queue entries stay 8-byte aligned");
  const TreeParams& P = a.params;
  const uint32_t n_chunks = a.n_fchunks;
  const uint32_t n_nodes = a.ctl->n_nodes;
  const uint32_t items = n_nodes * n_chunks;
  const bool fuse_sub = !WIDE && a.fused_sub != 0;  // the launch forms the siblings' histograms
  // The work on one (node, chunk) item; every thread of the CTA calls it.
  auto eval_item = [&](uint32_t item) {
    const uint32_t i = item / n_chunks, c = item % n_chunks;
    const NodeRec node = a.nodes[parity][i];
    const uint32_t f = c * uint32_t(nwarps) + uint32_t(warp);
    const double inv_g = a.trees[node.tree].inv_g, inv_h = a.trees[node.tree].inv_h;
    const int st_kh = a.trees[node.tree].kh;
    SplitRec best;
    best.valid = 0;
    best.gain = 0.0;
    best.feature = f;
    best.threshold = 0;
    best.default_left = 1;
    uint32_t err = 0;
    float best32 = -1.0f;  // best certainly admissible FP32 score of the feature
    // A node with fewer than 2 * min_samples_leaf rows has no admissible split.
    bool active = f < a.features && node.count >= 2 * P.min_samples_leaf;
    if (active) {
      const uint32_t allowed = a.node_allowed[parity][i * P.path_words + (f >> 5)];
      active = (allowed >> (f & 31)) & 1u;
    }
    if (active) {  // warp-uniform
      const uint32_t df = dataset_feature(a, node.tree, f);
      const uint32_t nb = a.bin_count[df];
      const bool hm = a.has_missing[df] != 0;
      // At most 32 bins: one slot per lane (slot = lane), the missing slot apart.
      const bool few = !WIDE && nb <= 32u;
      const int kper = few ? 1 : 8;
      unsigned long long* sh = s_hist + size_t(warp) * (kScanHistBytes / 8);
      const uint32_t pages = WIDE ? a.slots / uint32_t(kSlots) : 1u;
      const unsigned long long* fhist =
          a.hist + (size_t(node.slot) * a.features + f) * size_t(WIDE ? a.slots : uint32_t(kSlots)) * 3;
      // Slot lane * 8 + k of the staged page (few bins: slot lane, k = 0): word w at
      // sh[(w * 8 + k) * 32 + lane].
      auto slot_word = [&](int k, int w) -> unsigned long long { return sh[(w * 8 + k) * 32 + lane]; };
      auto slot_of = [&](int k) -> int { return few ? lane : lane * 8 + k; };
      // The lane's total of its 8 slots of the staged page; the missing slot (slot
      // kMissingSlot of the last page) goes to `miss` instead. Raw counts add to `count`.
      auto page_sums = [&](bool last, Stat<FIXED>& sum, Stat<FIXED>& miss,
                           unsigned long long& count) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          if (k >= kper) break;
          const int s = slot_of(k);
          Stat<FIXED> b;
          const unsigned long long raw_count = slot_word(k, 0);
          b.count = uint32_t(raw_count);  // the total below checks the full word
          if constexpr (FIXED) {
            b.g = (long long)slot_word(k, 1);
            b.h = (long long)slot_word(k, 2);
          } else {
            b.g = __longlong_as_double((long long)slot_word(k, 1));
            b.h = __longlong_as_double((long long)slot_word(k, 2));
            if (!isfinite(b.g) || !isfinite(b.h) || b.h < 0.0) err |= kErrNonFinite;
          }
          count += raw_count;
          if (hm && last && s == kMissingSlot) {
            miss = b;
          } else {
            sum = stat_add<FIXED>(sum, b);
          }
        }
      };
      auto inclusive_prefix = [&](Stat<FIXED> incl) -> Stat<FIXED> {
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const Stat<FIXED> y = shfl_up_stat<FIXED>(incl, off);
          if (lane >= off) incl = stat_add<FIXED>(y, incl);
        }
        return incl;
      };
      auto exclusive_of = [&](const Stat<FIXED>& incl) -> Stat<FIXED> {
        Stat<FIXED> cin = shfl_up_stat<FIXED>(incl, 1);
        if (lane == 0) cin = stat_zero<FIXED>();
        return cin;
      };
      Stat<FIXED> miss = stat_zero<FIXED>(), carry_in = stat_zero<FIXED>();
      unsigned long long total_count = 0;
      if constexpr (WIDE) {
        for (uint32_t p = 0; p < pages; ++p) {
          __syncwarp();
          stage_feature_hist(fhist + size_t(p) * kSlots * 3, sh, lane);
          Stat<FIXED> unused = stat_zero<FIXED>();
          page_sums(p + 1 == pages, unused, miss, total_count);
        }
      } else {
        const bool sub = fuse_sub && node.sub_from != 0;
        unsigned long long* own = a.hist + (size_t(node.slot) * a.features + f) * kSlots * 3;
        const unsigned long long* built =
            sub ? a.hist + (size_t(node.sub_from - 1) * a.features + f) * kSlots * 3 : nullptr;
        unsigned long long mw[3] = {0ull, 0ull, 0ull};
        if (few) {
          stage_few_slots<FIXED>(own, built, hm, sh, lane, mw, err);
        } else if (sub) {
          stage_sibling_hist<FIXED>(own, built, sh, lane, err);
        } else {
          stage_feature_hist(fhist, sh, lane);
        }
        Stat<FIXED> sum = stat_zero<FIXED>();
        page_sums(true, sum, miss, total_count);
        carry_in = exclusive_of(inclusive_prefix(sum));
        if (few) {  // the missing slot, in every lane; its rows counted once
          miss.count = uint32_t(mw[0]);
          if constexpr (FIXED) {
            miss.g = (long long)mw[1];
            miss.h = (long long)mw[2];
          } else {
            miss.g = __longlong_as_double((long long)mw[1]);
            miss.h = __longlong_as_double((long long)mw[2]);
            if (!isfinite(miss.g) || !isfinite(miss.h) || miss.h < 0.0) err |= kErrNonFinite;
          }
          if (lane == 0) total_count += mw[0];
        }
      }
      if (!few) miss = shfl_stat<FIXED>(miss, 31);
      for (int off = 16; off > 0; off >>= 1)
        total_count += __shfl_xor_sync(0xffffffffu, total_count, off);
      if (total_count != node.count) err |= kErrCountMismatch;
      Stat<FIXED> parent;
      parent.count = node.count;
      if constexpr (FIXED) {
        parent.g = node.qg;
        parent.h = node.qh;
      } else {
        parent.g = node.g;
        parent.h = node.h;
      }
      if (nb >= 2 && total_count == node.count) {
        bool miss_h_above;
        if constexpr (FIXED) {
          // The images q * 2^-k compare as the quantized sums while those convert exactly.
          const long long lim = 1ll << 53;
          miss_h_above = (miss.h > -lim && miss.h < lim && parent.h > -lim && parent.h < lim)
                             ? miss.h > parent.h
                             : images_above(miss.h, parent.h, inv_h);
        } else {
          miss_h_above = miss.h > parent.h;
        }
        if (miss.count > parent.count || miss_h_above) err |= kErrMissing;
        const Stat<FIXED> nmp = stat_sub<FIXED>(parent, miss);
        const int8_t mono = P.has_monotonic ? a.monotonic[df] : 0;
        const uint32_t rnd =
            P.split_strategy == 1
                ? stable_random_threshold(
                      a.tree_seeds ? a.tree_seeds[node.tree] : P.random_seed,
                      a.feature_rank ? a.feature_rank[size_t(node.tree) * a.features + f] : f,
                      node.node_index, node.depth, nb - 1)
                : 0xffffffffu;
        const ScreenScale scale = screen_scale<FIXED>(P, mono, st_kh);
        const bool screen = scale.on;
        auto classify = [&](const Stat<FIXED>& cl, const Stat<FIXED>& cr, float* s32) -> int {
          return screen_classify<FIXED>(min_leaf_rows(P), scale, cl, cr, s32);
        };
        // Visits every (threshold, missing direction) step of the lane's 8 slots of the
        // staged page (the left prefix before them `cin`, the page's first threshold
        // `base`) with the candidate's left/right statistics; `cand` is false where no
        // candidate exists. Every lane visits every step (the visitor may use warp
        // collectives).
        auto scan_candidates = [&](const Stat<FIXED>& cin, uint32_t base, bool last, auto&& visit) {
          Stat<FIXED> left = cin;
#pragma unroll 1
          for (int k = 0; k < kper; ++k) {
            const int s = slot_of(k);
            bool empty_bin = false;
            if (!(hm && last && s == kMissingSlot)) {  // reload the slot from the staging area
              Stat<FIXED> b;
              b.count = uint32_t(slot_word(k, 0));
              empty_bin = b.count == 0;
              if constexpr (FIXED) {
                b.g = (long long)slot_word(k, 1);
                b.h = (long long)slot_word(k, 2);
              } else {
                b.g = __longlong_as_double((long long)slot_word(k, 1));
                b.h = __longlong_as_double((long long)slot_word(k, 2));
              }
              left = stat_add<FIXED>(left, b);
            }
            const uint32_t t = base + uint32_t(s);
            const Stat<FIXED> right = stat_sub<FIXED>(nmp, left);
            bool cand = t + 1 < nb;
            if (cand && left.count > nmp.count) {
              err |= kErrPrefix;
              cand = false;
            }
            if (left.count == 0 && right.count == 0) cand = false;
            if (P.split_strategy == 1 && t != rnd) cand = false;
            // After an empty bin the candidate repeats threshold t-1's statistics exactly
            // and loses the tie to it (IsBetterSplit prefers the lower threshold).
            if (P.split_strategy == 0 && t > 0 && empty_bin) cand = false;
            for (int d = 0; d < 2; ++d) {
              const uint32_t dl = 1u - uint32_t(d);  // default_left 1, then 0
              if (dl == 0 && miss.count == 0) break;  // warp-uniform
              const Stat<FIXED> cl = dl ? stat_add<FIXED>(left, miss) : left;
              const Stat<FIXED> cr = dl ? right : stat_add<FIXED>(right, miss);
              visit(cand, cl, cr, t, dl);
            }
          }
        };
        // Runs body(left prefix, first threshold, last page) for each page: the one page
        // staged above, or (wide) each page staged in turn with the prefix carried over.
        auto for_pages = [&](auto&& body) {
          if constexpr (!WIDE) {
            body(carry_in, 0u, true);
          } else {
            Stat<FIXED> carry = stat_zero<FIXED>();
            for (uint32_t p = 0; p < pages; ++p) {
              __syncwarp();
              stage_feature_hist(fhist + size_t(p) * kSlots * 3, sh, lane);
              const bool last = p + 1 == pages;
              Stat<FIXED> sum = stat_zero<FIXED>(), unused = stat_zero<FIXED>();
              unsigned long long unused_count = 0;
              page_sums(last, sum, unused, unused_count);
              const Stat<FIXED> incl = inclusive_prefix(sum);
              body(stat_add<FIXED>(carry, exclusive_of(incl)), p * uint32_t(kSlots), last);
              carry = stat_add<FIXED>(carry, shfl_stat<FIXED>(incl, 31));
            }
          }
        };
        // The lane's best certainly admissible FP32 score.
        auto screen_scores = [&]() {
          for_pages([&](const Stat<FIXED>& cin, uint32_t base, bool last) {
            scan_candidates(cin, base, last, [&](bool cand, const Stat<FIXED>& cl,
                                                 const Stat<FIXED>& cr, uint32_t, uint32_t) {
              if (!cand) return;
              float sc = 0.0f;
              const int cls = classify(cl, cr, &sc);
              if (cls == 1) best32 = fmaxf(best32, sc);
            });
          });
          for (int off = 16; off > 0; off >>= 1)
            best32 = fmaxf(best32, __shfl_xor_sync(0xffffffffu, best32, off));
        };
        {
          float cut = -1.0f;
          if (screen) {
            screen_scores();
            cut = best32 >= 1e-30f ? best32 * (1.0f - 0x1p-18f) : -1.0f;
          }
          // Candidates that pass the screen queue up, and the warp evaluates them in FP64
          // one per lane: the narrow FP64 pipe runs one pass per 32 survivors instead of
          // one per (threshold, direction) step that has a survivor in any lane.
          ScanCand<FIXED>* queue = s_queue + size_t(warp) * kScanQueue;
          uint32_t queued = 0;
          auto drain = [&]() {
            __syncwarp();
            if (uint32_t(lane) < queued) {
              const ScanCand<FIXED> e = queue[lane];
              consider<FIXED>(P, e.cl, e.cr, inv_g, inv_h, mono, node.lo, node.hi, f, e.threshold,
                              e.default_left, best, err);
            }
            __syncwarp();
            queued = 0;
          };
          for_pages([&](const Stat<FIXED>& cin, uint32_t base, bool last) {
            scan_candidates(cin, base, last, [&](bool cand, const Stat<FIXED>& cl,
                                                 const Stat<FIXED>& cr, uint32_t t, uint32_t dl) {
              bool want = cand;
              if (want && screen && cut > 0.0f) {
                float sc = 0.0f;
                const int cls = classify(cl, cr, &sc);
                want = cls == 2 || (cls == 1 && sc >= cut);
              }
              const uint32_t ballot = __ballot_sync(0xffffffffu, want);
              if (ballot == 0) return;
              const uint32_t n_new = uint32_t(__popc(ballot));
              if (queued + n_new > kScanQueue) drain();
              if (want) {
                ScanCand<FIXED> e;
                e.cl = cl;
                e.cr = cr;
                e.threshold = t;
                e.default_left = dl;
                queue[queued + uint32_t(__popc(ballot & ((1u << lane) - 1u)))] = e;
              }
              queued += n_new;
            });
          });
          if (queued) drain();
        }
      }
    }
    if (err) raise(a.ctl, err);
    {
      // Warp argmax (all lanes share the feature): every lane ends with the winner's id.
      uint32_t win = uint32_t(lane);
      {
        double g = best.gain;
        uint32_t v = best.valid, thr = best.threshold, dl = best.default_left;
        for (int off = 16; off > 0; off >>= 1) {
          const double og = __shfl_xor_sync(0xffffffffu, g, off);
          const uint32_t ov = __shfl_xor_sync(0xffffffffu, v, off);
          const uint32_t ot = __shfl_xor_sync(0xffffffffu, thr, off);
          const uint32_t od = __shfl_xor_sync(0xffffffffu, dl, off);
          const uint32_t ow = __shfl_xor_sync(0xffffffffu, win, off);
          bool take;
          if (ov != v) take = ov > v;
          else if (!v) take = ow < win;
          else if (og != g) take = og > g;
          else if (ot != thr) take = ot < thr;
          else if (od != dl) take = od > dl;
          else take = ow < win;
          if (take) {
            g = og;
            v = ov;
            thr = ot;
            dl = od;
            win = ow;
          }
        }
      }
      if (uint32_t(lane) == win) warp_best[warp] = best;
      __syncthreads();
      if (threadIdx.x == 0) {
        SplitRec b = warp_best[0];
        for (int w = 1; w < nwarps; ++w)
          if (better_split(warp_best[w], b)) b = warp_best[w];
        a.partial[size_t(i) * n_chunks + c] = b;
      }
      __syncthreads();
    }
  };
  for (uint32_t item = blockIdx.x; item < items; item += gridDim.x) eval_item(item);
  (void)sizeof(V);
}

// ---- Split scan in two launches ---------------------------------------------------------
// Where the FP32 screen applies (best-split strategy, no reg_alpha, reg_lambda > 0):
//  split_screen_kernel forms every (node, feature)'s prefix sums and the FP32 scores of its
//    candidates, raises the node's maximum of certainly admissible scores (node_screen,
//    atomicMax on the float bits) and writes the feature's own (feature_screen).
//  split_exact_kernel, with the node's final maximum M, evaluates in FP64, as the reference
//    does, the features that hold a candidate at or above M(1 - 2^-18) or one to evaluate
//    whatever the maximum, and of those features the candidates at or above that cut and
//    the close calls. A candidate below the cut has a strictly lower exact gain than the
//    admissible candidate that scored M, so it cannot win the node. partial[node] is the
//    node's best split.
// Both give a page of kSlots slots to a CTA, two neighbouring slots per thread (48
// contiguous bytes, three 16-byte loads): a block-wide prefix sum, then each thread
// evaluates its own thresholds' candidates. One slot per thread spends half its
// instructions on the prefix sum, eight (a warp per page) load 192-byte strides and leave a
// shallow level's few features to few warps. Threads past the feature's bins load and
// evaluate nothing, so a feature of few bins costs little.
constexpr int kScanCta = kSlots / 2;
constexpr int kScanCtaWarps = kScanCta / 32;
constexpr uint32_t kScanFeaturesPerItem = 8;  // at most; fewer where that leaves SMs idle

// A feature_screen word: 0 (no candidate), or the best certainly admissible FP32 score's
// bits (at least 1), with kFeatureExact set where the feature is evaluated exactly whatever
// the node's maximum (its screen is off, or a candidate is too close to call in FP32).
constexpr uint32_t kFeatureExact = 0x80000000u;

// The warps' totals of a page, exchanged through shared memory, and the missing slot.
template <bool FIXED>
struct PageTotals {
  typename Stat<FIXED>::V g[kScanCtaWarps], h[kScanCtaWarps];
  typename Stat<FIXED>::V miss_g, miss_h;
  uint32_t count[kScanCtaWarps], miss_count;
};

template <bool FIXED>
__device__ __forceinline__ Stat<FIXED> warp_inclusive(Stat<FIXED> x, int lane) {
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const Stat<FIXED> y = shfl_up_stat<FIXED>(x, off);
    if (lane >= off) x = stat_add<FIXED>(y, x);
  }
  return x;
}

// Block-wide inclusive prefix of one value per thread; *total gets the page's sum and *below
// (floating-point sums only) the prefix without the thread's own value. One barrier; `t` may be
// written again after the CTA's next barrier.
template <bool FIXED>
__device__ __forceinline__ Stat<FIXED> page_prefix(const Stat<FIXED>& own, PageTotals<FIXED>& t,
                                                   Stat<FIXED>* total, Stat<FIXED>* below) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Stat<FIXED> incl = warp_inclusive<FIXED>(own, lane);
  if (lane == 31) {
    t.count[warp] = incl.count;
    t.g[warp] = incl.g;
    t.h[warp] = incl.h;
  }
  __syncthreads();
  Stat<FIXED> before = stat_zero<FIXED>(), all = stat_zero<FIXED>();
#pragma unroll
  for (int q = 0; q < kScanCtaWarps; ++q) {
    if (q == warp) before = all;
    Stat<FIXED> w;
    w.count = t.count[q];
    w.g = t.g[q];
    w.h = t.h[q];
    all = stat_add<FIXED>(all, w);
  }
  *total = all;
  if constexpr (!FIXED) {
    Stat<FIXED> lower = shfl_up_stat<FIXED>(incl, 1);
    if (lane == 0) lower = stat_zero<FIXED>();
    *below = stat_add<FIXED>(before, lower);
  }
  return stat_add<FIXED>(before, incl);
}

// The raw words of a thread's two slots (count, g, h of the even one, then of the odd one),
// and the built sibling's where the histogram is formed on the way.
struct SlotWords {
  unsigned long long own[6], built[6];
};

__device__ __forceinline__ void load_pair(unsigned long long (&w)[6], const unsigned long long* src) {
  const ulonglong2* v = reinterpret_cast<const ulonglong2*>(src);  // 48-byte pairs of a 16-byte aligned slot
  const ulonglong2 x = v[0], y = v[1], z = v[2];
  w[0] = x.x;
  w[1] = x.y;
  w[2] = y.x;
  w[3] = y.y;
  w[4] = z.x;
  w[5] = z.y;
}

template <bool FIXED>
__device__ __forceinline__ Stat<FIXED> slot_stat(unsigned long long c, unsigned long long g,
                                                 unsigned long long h, uint32_t& err) {
  Stat<FIXED> b;
  b.count = uint32_t(c);
  if (c >> 32) err |= kErrCountMismatch;  // a node holds fewer than 2^32 rows
  if constexpr (FIXED) {
    b.g = (long long)g;
    b.h = (long long)h;
  } else {
    b.g = __longlong_as_double((long long)g);
    b.h = __longlong_as_double((long long)h);
    if (!isfinite(b.g) || !isfinite(b.h) || b.h < 0.0) err |= kErrNonFinite;
  }
  return b;
}

// What the scans need of a node, its tree and the launch.
template <bool FIXED>
struct ScanNode {
  uint32_t slot, sub_from;
  Stat<FIXED> parent;
  double inv_h;
};

template <bool FIXED>
__device__ __forceinline__ ScanNode<FIXED> scan_node(const NodeRec& node, double inv_h) {
  ScanNode<FIXED> s;
  s.slot = node.slot;
  s.sub_from = node.sub_from;
  s.parent.count = uint32_t(node.count);
  if constexpr (FIXED) {
    s.parent.g = node.qg;
    s.parent.h = node.qh;
  } else {
    s.parent.g = node.g;
    s.parent.h = node.h;
  }
  s.inv_h = inv_h;
  return s;
}

// The missing rows' statistics never exceed the node's (tree_split.cpp:186-189).
template <bool FIXED>
__device__ __forceinline__ bool missing_above(const Stat<FIXED>& miss, const Stat<FIXED>& parent,
                                              double inv_h) {
  if (miss.count > parent.count) return true;
  if constexpr (FIXED) {
    // The images q * 2^-k compare as the quantized sums while those convert exactly.
    const long long lim = 1ll << 53;
    return (miss.h > -lim && miss.h < lim && parent.h > -lim && parent.h < lim)
               ? miss.h > parent.h
               : images_above(miss.h, parent.h, inv_h);
  } else {
    return miss.h > parent.h;
  }
}

// Whether a page-`p` pair holds anything: every slot from the feature's bin count on is
// empty, but for the missing rows' (the last of all, odd: the second of its pair).
__device__ __forceinline__ bool pair_held(uint32_t s, uint32_t nb, bool hm, uint32_t S) {
  return s < nb || (hm && s + 2 == S);
}

// Words of the pair that starts at slot s (zeros where both slots are empty).
template <bool FIXED>
__device__ __forceinline__ SlotWords load_slots(const TrainerDev& a, const ScanNode<FIXED>& node,
                                                uint32_t f, uint32_t nb, bool hm, uint32_t S, uint32_t s) {
  SlotWords w{};
  if (pair_held(s, nb, hm, S)) {
    load_pair(w.own, a.hist + ((size_t(node.slot) * a.features + f) * S + s) * 3);
    if (node.sub_from != 0)
      load_pair(w.built, a.hist + ((size_t(node.sub_from - 1) * a.features + f) * S + s) * 3);
  }
  return w;
}

// One feature of one node, every thread of the CTA: calls visit(left, right, threshold,
// default_left) for each candidate of the thread's slots. `first` holds page 0's words of
// the thread's pair. A sibling's histogram (node.sub_from) is formed as parent minus built
// child on the way, with subtract_kernel's checks, and written back where a later launch
// reads it.
// ROOT: the node's statistics are the feature's own totals (every feature of a root holds
// all of its rows, so in fixed point they are the same), which it leaves in node.parent.
template <bool FIXED, bool WIDE, bool ROOT, class Visit>
__device__ __forceinline__ void scan_feature(const TrainerDev& a, ScanNode<FIXED>& node, bool write_back,
                                             uint32_t f, uint32_t nb, bool hm, const SlotWords& first,
                                             PageTotals<FIXED>* totals, uint32_t& buf, uint32_t& err,
                                             Visit&& visit) {
  const uint32_t S = WIDE ? a.slots : uint32_t(kSlots);
  const uint32_t pages = WIDE ? S / uint32_t(kSlots) : 1u;
  const bool sub = node.sub_from != 0;
  Stat<FIXED> miss = stat_zero<FIXED>(), carry = stat_zero<FIXED>();
  if (WIDE && hm) {  // the last page's last slot, needed from the first page on
    uint32_t ignored = 0;
    SlotWords w = load_slots<FIXED>(a, node, f, nb, hm, S, S - 2);
#pragma unroll
    for (uint32_t k = 3; k < 6; ++k)
      if (sub) w.own[k] = sibling_word<FIXED>(w.own[k], w.built[k], k - 3, ignored);
    miss = slot_stat<FIXED>(w.own[3], w.own[4], w.own[5], ignored);
  }
  for (uint32_t p = 0; p < pages; ++p) {
    const uint32_t s = p * uint32_t(kSlots) + 2 * threadIdx.x;
    SlotWords w = first;
    if (WIDE && p > 0) w = load_slots<FIXED>(a, node, f, nb, hm, S, s);
    if (sub && pair_held(s, nb, hm, S)) {
#pragma unroll
      for (uint32_t k = 0; k < 6; ++k) w.own[k] = sibling_word<FIXED>(w.own[k], w.built[k], k % 3, err);
      if (write_back) {
        ulonglong2* out = reinterpret_cast<ulonglong2*>(
            a.hist + ((size_t(node.slot) * a.features + f) * S + s) * 3);
        out[0] = make_ulonglong2(w.own[0], w.own[1]);
        out[1] = make_ulonglong2(w.own[2], w.own[3]);
        out[2] = make_ulonglong2(w.own[4], w.own[5]);
      }
    }
    const Stat<FIXED> b0 = slot_stat<FIXED>(w.own[0], w.own[1], w.own[2], err);
    Stat<FIXED> b1 = slot_stat<FIXED>(w.own[3], w.own[4], w.own[5], err);
    PageTotals<FIXED>& t = totals[buf];
    buf ^= 1u;
    if (hm && s + 2 == S) {
      t.miss_count = b1.count;
      t.miss_g = b1.g;
      t.miss_h = b1.h;
      b1 = stat_zero<FIXED>();
    }
    // The left sums of the pair's two thresholds. Integers: the lower one by subtraction. FP64
    // sums are only added: (a + b) - b loses what is small beside b.
    Stat<FIXED> total, left0;
    const Stat<FIXED> left1 =
        stat_add<FIXED>(carry, page_prefix<FIXED>(stat_add<FIXED>(b0, b1), t, &total, &left0));
    if constexpr (FIXED) left0 = stat_sub<FIXED>(left1, b1);
    else left0 = stat_add<FIXED>(stat_add<FIXED>(carry, left0), b0);
    carry = stat_add<FIXED>(carry, total);
    if (!WIDE && hm) {
      miss.count = t.miss_count;
      miss.g = t.miss_g;
      miss.h = t.miss_h;
    }
    if constexpr (ROOT) {  // one page
      const uint32_t rows = node.parent.count;
      node.parent = stat_add<FIXED>(carry, miss);
      if (node.parent.count != rows) {
        err |= kErrCountMismatch;
        return;  // the same in every thread
      }
    }
    if (p + 1 == pages && carry.count + miss.count != node.parent.count) {
      err |= kErrCountMismatch;
      if (!WIDE) return;  // the same in every thread
    }
    if (p == 0 && nb >= 2 && missing_above<FIXED>(miss, node.parent, node.inv_h)) err |= kErrMissing;
    const Stat<FIXED> nmp = stat_sub<FIXED>(node.parent, miss);
    // A threshold's candidates. An empty bin's repeat threshold s-1's statistics exactly and
    // lose the tie to them (IsBetterSplit prefers the lower threshold).
    auto at = [&](uint32_t th, const Stat<FIXED>& left, bool empty_bin) {
      if (th + 1 >= nb || (empty_bin && th > 0)) return;
      if (left.count > nmp.count) {
        err |= kErrPrefix;
        return;
      }
      const Stat<FIXED> right = stat_sub<FIXED>(nmp, left);
      if (left.count == 0 && right.count == 0) return;
      visit(stat_add<FIXED>(left, miss), right, th, 1u);
      if (miss.count != 0) visit(left, stat_add<FIXED>(right, miss), th, 0u);
    };
    at(s, left0, b0.count == 0);
    at(s + 1, left1, b1.count == 0);
  }
}

template <bool FIXED, bool WIDE, bool ROOT>
__global__ void __launch_bounds__(kScanCta, WIDE ? 5 : 6) split_screen_kernel(TrainerDev a, int parity, bool last) {
  static_assert(!ROOT || (FIXED && !WIDE), "the features' totals are the same in fixed point only");
  __shared__ PageTotals<FIXED> s_totals[2];
  __shared__ uint32_t s_word[2][kScanFeaturesPerItem][kScanCtaWarps];
  const TreeParams& P = a.params;
  launch_order();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t F = a.features, S = WIDE ? a.slots : uint32_t(kSlots);
  const uint32_t msl = min_leaf_rows(P);
  const uint32_t n_nodes = a.ctl->n_nodes;
  // An item: up to kScanFeaturesPerItem features of one node, fewer while the level has
  // fewer (node, feature) pairs than that many per CTA.
  const uint64_t pairs = uint64_t(n_nodes) * F;
  const uint32_t per = uint32_t(min(uint64_t(kScanFeaturesPerItem), max(uint64_t(1), pairs / gridDim.x)));
  const uint32_t chunks = ceil_div(F, per);
  const uint32_t items = n_nodes * chunks;
  uint32_t buf = 0, ib = 0, err = 0;
  for (uint32_t item = blockIdx.x; item < items; item += gridDim.x, ib ^= 1u) {
    const uint32_t i = item / chunks, f0 = (item - i * chunks) * per;
    const uint32_t nf = min(per, F - f0);
    NodeRec& rec = a.nodes[parity][i];
    const TreeState& tree = a.trees[rec.tree];
    ScanNode<FIXED> node = scan_node<FIXED>(rec, tree.inv_h);
    if constexpr (ROOT) node.parent.count = rec.seg_cnt;
    const int kh = tree.kh;
    // A node with fewer than 2 * min_samples_leaf rows has no admissible split (a root's
    // statistics are formed all the same).
    const bool usable = ROOT || rec.count >= 2 * P.min_samples_leaf;
    const uint32_t* allowed = a.node_allowed[parity] + size_t(i) * P.path_words;
    auto active = [&](uint32_t k) -> bool {
      return k < nf && usable && ((allowed[(f0 + k) >> 5] >> ((f0 + k) & 31)) & 1u);
    };
    bool act = active(0);
    uint32_t df = act ? dataset_feature(a, rec.tree, f0) : 0u;
    uint32_t nb = act ? a.bin_count[df] : 0u;
    bool hm = act && a.has_missing[df] != 0;
    SlotWords w = !WIDE && act ? load_slots<FIXED>(a, node, f0, nb, hm, S, 2 * threadIdx.x) : SlotWords{};
    for (uint32_t k = 0; k < nf; ++k) {
      // The next feature's words are in flight while this one is scanned (a wide feature's
      // pages are many and its registers fewer: its own words only).
      const uint32_t f = f0 + k;
      const bool act_next = active(k + 1);
      const uint32_t df_next = act_next ? dataset_feature(a, rec.tree, f + 1) : 0u;
      const uint32_t nb_next = act_next ? a.bin_count[df_next] : 0u;
      const bool hm_next = act_next && a.has_missing[df_next] != 0;
      const SlotWords w_next = !WIDE && act_next
                                   ? load_slots<FIXED>(a, node, f + 1, nb_next, hm_next, S, 2 * threadIdx.x)
                                   : SlotWords{};
      if (WIDE && act) w = load_slots<FIXED>(a, node, f, nb, hm, S, 2 * threadIdx.x);
      uint32_t word = 0, exact = 0;
      if (act) {  // the same in every thread
        const ScreenScale scale = screen_scale<FIXED>(P, P.has_monotonic ? a.monotonic[df] : int8_t(0), kh);
        scan_feature<FIXED, WIDE, ROOT>(
            a, node, !last, f, nb, hm, w, s_totals, buf, err,
            [&](const Stat<FIXED>& cl, const Stat<FIXED>& cr, uint32_t, uint32_t) {
              if (!scale.on) {
                exact = kFeatureExact;
                return;
              }
              float score = 0.0f;
              const int cls = screen_classify<FIXED>(msl, scale, cl, cr, &score);
              if (cls == 1) word = max(word, max(__float_as_uint(score), 1u));
              if (cls == 2) exact = kFeatureExact;
            });
        if constexpr (ROOT) {
          if (threadIdx.x == 0) {
            // The tree's first allowed feature writes the root's record and leaf.
            bool lead = (allowed[f >> 5] & ((1u << (f & 31)) - 1u)) == 0;
            for (uint32_t q = 0; q < (f >> 5); ++q) lead = lead && allowed[q] == 0;
            if (lead) {
              rec.count = node.parent.count;
              rec.qg = node.parent.g;
              rec.qh = node.parent.h;
              rec.g = q_image(node.parent.g, tree.inv_g);
              rec.h = q_image(node.parent.h, tree.inv_h);
              write_root_leaf(a, rec.tree, rec.g, rec.h);
            }
          }
          node.parent.count = rec.seg_cnt;
        }
      }
      word = __reduce_max_sync(0xffffffffu, word);
      if (__any_sync(0xffffffffu, exact != 0)) word |= kFeatureExact;
      if (lane == 0) s_word[ib][k][warp] = word;
      act = act_next;
      df = df_next;
      nb = nb_next;
      hm = hm_next;
      w = w_next;
    }
    __syncthreads();
    if (warp == 0) {
      uint32_t best = 0, flag = 0;
      if (uint32_t(lane) < nf) {
#pragma unroll
        for (int q = 0; q < kScanCtaWarps; ++q) {
          const uint32_t v = s_word[ib][lane][q];
          best = max(best, v & ~kFeatureExact);
          flag |= v & kFeatureExact;
        }
        a.feature_screen[size_t(i) * F + f0 + lane] = best | flag;
      }
      best = __reduce_max_sync(0xffffffffu, best);
      if (lane == 0 && __uint_as_float(best) >= 1e-30f) atomicMax(a.node_screen + i, best);
    }
  }
  if (err) raise(a.ctl, err);
}

// One CTA per node, or `parts` for each node of a small level of many features. Mostly a node
// has one to three features to evaluate and its first CTA takes them. With more than
// kExactAlone (features under monotone constraints, hessians at min_child_weight, equal
// columns) every CTA takes its share, 2 to 12 us a feature, and the last one to finish picks
// the best. Ten trees of depth 6, one CTA per node -> shared: 100,000 x 200 all monotone
// 147 -> 30.4 ms, 2,000 x 500 with min_child_weight 20 unweighted 86.9 -> 9.8, 100,000 x 200 of
// eight distinct columns 9.3 -> 5.0, 200 x 5,000 down to single rows (whose splits tie in many
// features) 368 -> 22.7.
// to_active: a leaf-wise step, whose nodes' splits go to their active leaves. last: the
// level's children are leaves, so no later level subtracts from a sibling's histogram: the
// screen leaves it unwritten (a quarter of its bytes) and the few features evaluated here
// form it again.
// The common path is short of instructions on purpose, as each launch fetches it cold: what only
// shared nodes need is out of line, and the features are counted at a barrier (inlined, with a
// sum through shared memory, ordinary levels took 1 us more). A level that could share costs 0.2
// to 0.5 us more than one CTA per node.
constexpr uint32_t kExactAlone = 8;

// Whether the thread's listed feature is one of this part's: every parts-th of the node's.
// `before`: listed features of the blocks before, moved on. Every thread of the CTA.
__device__ __noinline__ bool part_takes(bool listed, uint32_t* before, uint32_t part, uint32_t parts) {
  __shared__ uint32_t s_rank[kScanCtaWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t ballot = __ballot_sync(0xffffffffu, listed);
  if (lane == 0) s_rank[warp] = uint32_t(__popc(ballot));
  __syncthreads();
  uint32_t rank = *before + uint32_t(__popc(ballot & ((1u << lane) - 1u)));
#pragma unroll
  for (int q = 0; q < kScanCtaWarps; ++q) {
    if (q < warp) rank += s_rank[q];
    *before += s_rank[q];
  }
  return listed && rank % parts == part;
}

// The end of a shared node's part, whose record is written: the last part to come here copies
// the best of the node's records to *out. Every thread of the CTA.
__device__ __noinline__ void part_done(const SplitRec* records, uint32_t* done, uint32_t parts, SplitRec* out) {
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    s_last = atomicAdd(done, 1u) == parts - 1;
    if (s_last) *done = 0;
  }
  __syncthreads();
  if (!s_last || threadIdx.x >= 32) return;
  __threadfence();
  uint32_t v = 0, f = 0xffffffffu, at = 0;
  double g = 0.0;
  auto consider_record = [&](uint32_t ov, double og, uint32_t of, uint32_t oat) {
    if (ov && (!v || og > g || (og == g && of < f))) {  // no two records share a feature
      v = ov;
      g = og;
      f = of;
      at = oat;
    }
  };
  for (uint32_t q = threadIdx.x; q < parts; q += 32)
    consider_record(__ldcg(&records[q].valid), __ldcg(&records[q].gain), __ldcg(&records[q].feature), q);
  for (int off = 16; off > 0; off >>= 1) {
    const uint32_t ov = __shfl_xor_sync(0xffffffffu, v, off), of = __shfl_xor_sync(0xffffffffu, f, off);
    const uint32_t oat = __shfl_xor_sync(0xffffffffu, at, off);
    const double og = __shfl_xor_sync(0xffffffffu, g, off);
    consider_record(ov, og, of, oat);
  }
  at = __shfl_sync(0xffffffffu, at, 0);  // without a split: any of the records
  const unsigned long long* src = reinterpret_cast<const unsigned long long*>(records + at);
  unsigned long long* dst = reinterpret_cast<unsigned long long*>(out);
  if (threadIdx.x < sizeof(SplitRec) / 8) dst[threadIdx.x] = __ldcg(src + threadIdx.x);
}

template <bool FIXED, bool WIDE, bool PARTS>
__global__ void __launch_bounds__(kScanCta, 4) split_exact_kernel(TrainerDev a, int parity, bool to_active, bool last) {
  __shared__ PageTotals<FIXED> s_totals[2];
  __shared__ uint32_t s_list[kScanCta], s_listed;
  __shared__ double s_gain[kScanCtaWarps];
  __shared__ uint32_t s_key[kScanCtaWarps][5];  // valid, feature, threshold, default_left, thread
  const TreeParams& P = a.params;
  launch_order();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t F = a.features, S = WIDE ? a.slots : uint32_t(kSlots);
  const uint32_t msl = min_leaf_rows(P);
  const uint32_t n_nodes = a.ctl->n_nodes;
  uint32_t buf = 0, err = 0;
  // PARTS: the grid is (the level's bound, parts).
  const uint32_t part = PARTS ? blockIdx.y : 0u, parts = PARTS ? gridDim.y : 1u;
  if (PARTS && n_nodes > gridDim.x) {
    if (threadIdx.x == 0) raise(a.ctl, kErrCapacity);
    return;
  }
  for (uint32_t i = blockIdx.x; i < n_nodes; i += gridDim.x) {
    const NodeRec& rec = a.nodes[parity][i];
    const TreeState& tree = a.trees[rec.tree];
    const double inv_g = tree.inv_g, inv_h = tree.inv_h;
    ScanNode<FIXED> node = scan_node<FIXED>(rec, inv_h);
    if (!last) node.sub_from = 0;
    const double lo = rec.lo, hi = rec.hi;
    const float m = __uint_as_float(a.node_screen[i]);
    const float cut = m >= 1e-30f ? m * (1.0f - 0x1p-18f) : -1.0f;
    auto listed_feature = [&](uint32_t f) -> bool {
      const uint32_t word = f < F ? a.feature_screen[size_t(i) * F + f] : 0u;
      return word != 0 && ((word & kFeatureExact) || !(__uint_as_float(word) < cut));
    };
    bool shared = false;  // the node's CTAs share its features; the same in all of them
    uint32_t mine_listed = 0;  // of the thread's first 32 features, one bit each
    if (PARTS) {
      uint32_t all = 0;
      if (threadIdx.x == 0) s_listed = 0;
#pragma unroll 1
      for (uint32_t k = 0; k * kScanCta < F; ++k) {
        const bool l = listed_feature(k * kScanCta + threadIdx.x);
        if (k < 32) mine_listed |= uint32_t(l) << k;
        all += uint32_t(__syncthreads_count(l));
      }
      shared = all > kExactAlone;
      if (!shared && part != 0) continue;
    }
    uint32_t before = 0;  // listed features of the blocks before
    // The thread's best candidate.
    uint32_t valid = 0, feature = 0, threshold = 0, default_left = 0;
    double gain = 0.0;
    Stat<FIXED> cl = stat_zero<FIXED>(), cr = stat_zero<FIXED>();
    for (uint32_t base = 0; base < F; base += kScanCta) {
      if (!PARTS || base) {  // PARTS: cleared with the counting above
        if (threadIdx.x == 0) s_listed = 0;
        __syncthreads();
      }
      const uint32_t mine = base + threadIdx.x;
      bool take = PARTS && base < 32 * kScanCta ? (mine_listed >> (base / kScanCta)) & 1u : listed_feature(mine);
      if (PARTS && shared) take = part_takes(take, &before, part, parts);
      if (take) s_list[atomicAdd(&s_listed, 1u)] = mine;  // any order: the best split is unique
      __syncthreads();
      const uint32_t listed = s_listed;
      for (uint32_t k = 0; k < listed; ++k) {
        const uint32_t f = s_list[k];
        const uint32_t df = dataset_feature(a, rec.tree, f);
        const uint32_t nb = a.bin_count[df];
        const bool hm = a.has_missing[df] != 0;
        const int8_t mono = P.has_monotonic ? a.monotonic[df] : int8_t(0);
        const ScreenScale scale = screen_scale<FIXED>(P, mono, tree.kh);
        const SlotWords w = load_slots<FIXED>(a, node, f, nb, hm, S, 2 * threadIdx.x);
        scan_feature<FIXED, WIDE, false>(
            a, node, false, f, nb, hm, w, s_totals, buf, err,
            [&](const Stat<FIXED>& l, const Stat<FIXED>& r, uint32_t t, uint32_t dl) {
              if (scale.on && cut > 0.0f) {
                float score = 0.0f;
                const int cls = screen_classify<FIXED>(msl, scale, l, r, &score);
                if (!(cls == 2 || (cls == 1 && score >= cut))) return;
              }
              double g;
              if (!exact_gain<FIXED>(P, l, r, inv_g, inv_h, mono, lo, hi, &g, err)) return;
              bool take = !valid;
              if (!take) {
                if (g != gain) take = g > gain;
                else if (f != feature) take = f < feature;
                else if (t != threshold) take = t < threshold;
                else take = dl > default_left;
              }
              if (take) {
                valid = 1;
                gain = g;
                feature = f;
                threshold = t;
                default_left = dl;
                cl = l;
                cr = r;
              }
            });
      }
      __syncthreads();  // the list is rewritten
    }
    // The CTA's best: a warp argmax, then over the warps.
    uint32_t win = threadIdx.x;
    {
      double g = gain;
      uint32_t v = valid, f = feature, t = threshold, dl = default_left;
      if (__any_sync(0xffffffffu, v != 0)) {
        for (int off = 16; off > 0; off >>= 1) {
          const double og = __shfl_xor_sync(0xffffffffu, g, off);
          const uint32_t ov = __shfl_xor_sync(0xffffffffu, v, off);
          const uint32_t of = __shfl_xor_sync(0xffffffffu, f, off);
          const uint32_t ot = __shfl_xor_sync(0xffffffffu, t, off);
          const uint32_t od = __shfl_xor_sync(0xffffffffu, dl, off);
          const uint32_t ow = __shfl_xor_sync(0xffffffffu, win, off);
          bool take;
          if (ov != v) take = ov > v;
          else if (!v) take = ow < win;
          else if (og != g) take = og > g;
          else if (of != f) take = of < f;
          else if (ot != t) take = ot < t;
          else if (od != dl) take = od > dl;
          else take = ow < win;
          if (take) {
            g = og;
            v = ov;
            f = of;
            t = ot;
            dl = od;
            win = ow;
          }
        }
      }
      if (lane == 0) {
        s_gain[warp] = g;
        s_key[warp][0] = v;
        s_key[warp][1] = f;
        s_key[warp][2] = t;
        s_key[warp][3] = dl;
        s_key[warp][4] = win;
      }
    }
    __syncthreads();
    int bw = -1;
#pragma unroll
    for (int q = 0; q < kScanCtaWarps; ++q) {
      if (!s_key[q][0]) continue;
      bool take = bw < 0;
      if (!take) {
        if (s_gain[q] != s_gain[bw]) take = s_gain[q] > s_gain[bw];
        else if (s_key[q][1] != s_key[bw][1]) take = s_key[q][1] < s_key[bw][1];
        else if (s_key[q][2] != s_key[bw][2]) take = s_key[q][2] < s_key[bw][2];
        else take = s_key[q][3] > s_key[bw][3];
      }
      if (take) bw = q;
    }
    SplitRec* node_best = a.partial + i;
    if (to_active) {
      const uint32_t at = a.lw_scan_map[i];
      LeafActive& leaf = a.lw_active[size_t(at >> 16) * a.lw_cap + (at & 0xFFFFu)];
      node_best = &leaf.best;
      if (threadIdx.x == 0 && part == 0) leaf.scanned = 1;
    }
    SplitRec* out = PARTS && shared ? a.exact_part + size_t(i) * parts + part : node_best;
    if (bw < 0) {
      if (threadIdx.x == 0) *out = no_split();
    } else if (threadIdx.x == s_key[bw][4]) {
      const int8_t mono =
          P.has_monotonic ? a.monotonic[dataset_feature(a, rec.tree, feature)] : int8_t(0);
      *out = split_record<FIXED>(P, cl, cr, inv_g, inv_h, mono, lo, hi, gain, feature, threshold,
                                 default_left);
    }
    if (PARTS && shared) part_done(a.exact_part + size_t(i) * parts, a.exact_done + i, parts, node_best);
    __syncthreads();  // the argmax arrays and the list are rewritten by the next node
  }
  if (err) raise(a.ctl, err);
}

// ------------------------------------------------------------------------------------
// Level finalize (one CTA)
// ------------------------------------------------------------------------------------
__device__ void write_leaf(TreeNodeOut* dst, double value) {
  TreeNodeOut n;
  n.feature_index = 0;
  n.threshold_bin = 0;
  n.left_child = 0xffffffffu;
  n.right_child = 0xffffffffu;
  n.leaf_value = value;
  n.gain = 0.0;
  n.default_left = 1;
  n.flags = 1;
  for (int k = 0; k < 6; ++k) n.reserved[k] = 0;
  *dst = n;
}

__device__ bool bounded_leaf(const TreeParams& p, double g, double h, double lo, double hi,
                             double* out) {
  if (lo > hi) return false;
  double w;
  if (!leaf_weight(g, h, p, &w)) return false;
  *out = clamp_bounds(w, lo, hi);
  return true;
}

// InteractionAllowsFeature (tree_interactions.cpp:32-45) of a child: word w of its allowed
// features from its path words.
__device__ __forceinline__ uint32_t allowed_word(const TrainerDev& a, const uint32_t* path,
                                                 uint32_t tree, uint32_t w) {
  const TreeParams& P = a.params;
  uint32_t allowed = 0xffffffffu;
  if (P.n_groups > 0) {
    allowed = 0;
    for (uint32_t g = 0; g < P.n_groups; ++g) {
      bool subset = true;
      for (uint32_t u = 0; u < P.path_words && subset; ++u)
        subset = (path[u] & ~a.group_masks[g * P.path_words + u]) == 0;
      if (subset) allowed |= a.group_masks[g * P.path_words + w];
    }
  }
  if (a.tree_feature_masks != nullptr) allowed &= a.tree_feature_masks[tree * P.path_words + w];
  return allowed;
}

__global__ void __launch_bounds__(1024) finalize_kernel(TrainerDev a, int parity, uint32_t depth) {
  __shared__ uint32_t sh[33 * 6];
  Control* ctl = a.ctl;
  launch_order();
  const TreeParams& P = a.params;
  const uint32_t n = ctl->n_nodes;
  const uint32_t W = P.path_words;
  const bool last = depth + 1 >= P.max_depth;  // children are leaves
  const uint32_t* tree_base = a.tree_scratch;                 // [T] valid prefix at first node
  uint32_t* tree_acc_base = a.tree_scratch + a.n_trees;       // [T] accepted prefix at first node
  uint32_t* tree_acc = a.tree_scratch + 2 * a.n_trees;        // [T] accepted count
  uint32_t* tree_vbase = a.tree_scratch;
  for (uint32_t t = threadIdx.x; t < a.n_trees; t += blockDim.x) tree_acc[t] = 0;
  __syncthreads();

  // Phase A0 (a scan that left one record per feature chunk): one warp per node merges them
  // into the first record (lanes read chunks in parallel; the features of different chunks
  // differ, so the total order of better_split has a unique winner among valid records).
  const uint32_t nfc = a.partial_stride;
  if (depth < P.max_depth && nfc > 1) {  // nodes at max_depth never split (tree.cpp:152-154)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (uint32_t i = warp; i < n; i += nw) {
      SplitRec* rec = a.partial + size_t(i) * nfc;
      uint32_t mine = lane < int(nfc) ? uint32_t(lane) : 0u;
      for (uint32_t c = lane + 32; c < nfc; c += 32)
        if (better_split(rec[c], rec[mine])) mine = c;
      uint32_t v = rec[mine].valid, f = rec[mine].feature, thr = rec[mine].threshold;
      uint32_t dl = rec[mine].default_left;
      double g = rec[mine].gain;
      for (int off = 16; off > 0; off >>= 1) {
        const uint32_t ov = __shfl_xor_sync(0xffffffffu, v, off);
        const double og = __shfl_xor_sync(0xffffffffu, g, off);
        const uint32_t of = __shfl_xor_sync(0xffffffffu, f, off);
        const uint32_t ot = __shfl_xor_sync(0xffffffffu, thr, off);
        const uint32_t od = __shfl_xor_sync(0xffffffffu, dl, off);
        const uint32_t om = __shfl_xor_sync(0xffffffffu, mine, off);
        bool take;
        if (ov != v) take = ov > v;
        else if (!v) take = om < mine;  // all invalid: keep chunk 0's record
        else if (og != g) take = og > g;
        else if (of != f) take = of < f;
        else if (ot != thr) take = ot < thr;
        else if (od != dl) take = od > dl;
        else take = om < mine;
        if (take) {
          v = ov;
          g = og;
          f = of;
          thr = ot;
          dl = od;
          mine = om;
        }
      }
      if (mine != 0) {  // copy the winner's record into chunk 0, word by word
        const unsigned long long* src = reinterpret_cast<const unsigned long long*>(rec + mine);
        unsigned long long* dst = reinterpret_cast<unsigned long long*>(rec);
        const unsigned long long w = lane < int(sizeof(SplitRec) / 8) ? src[lane] : 0ull;
        __syncwarp();
        if (lane < int(sizeof(SplitRec) / 8)) dst[lane] = w;
      }
    }
  }
  __syncthreads();

  // Phase A: valid flags, valid prefix; rows the next level builds.
  uint32_t carry = 0, built_units = 0;
  for (uint32_t base = 0; base < n; base += blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    uint32_t v[2] = {0, 0};
    uint32_t tree = 0;
    bool first = false;
    if (i < n) {
      if (depth < P.max_depth) {
        const SplitRec& b = a.partial[size_t(i) * a.partial_stride];
        v[0] = b.valid;
        if (b.valid) v[1] = uint32_t(((b.lcount <= b.rcount ? b.lcount : b.rcount) + 255) / 256);
      }
      tree = a.nodes[parity][i].tree;
      first = i == 0 || a.nodes[parity][i - 1].tree != tree;
    }
    uint32_t tot[2];
    const uint32_t own = v[0];
    block_scan<2>(v, tot, sh);
    if (i < n) {
      a.scratch_flags[i] = own;
      a.scratch_prefix[i] = carry + v[0];
      if (first) tree_vbase[tree] = carry + v[0];
    }
    carry += tot[0];
    built_units += tot[1];
    __syncthreads();
  }
  __syncthreads();
  // The next level's item size: it builds a node per valid split.
  const uint32_t level_per_sm = level_items_per_sm(a, n);
  const uint32_t item_rows =
      a.item_rows ? a.item_rows : adaptive_item_rows(uint64_t(built_units) * 256, a, level_per_sm, carry);

  // Phase B1: acceptance under max_leaves, accepted prefix, chunk prefixes.
  // Scanned values: 0 accepted, 1 build chunks, 2 partition chunks, 3 leaf segments,
  // 4 leaf chunks, 5 freed slots.
  uint32_t carry6[6] = {0, 0, 0, 0, 0, 0};
  const uint32_t leafseg_base = ctl->n_leafseg;
  const uint32_t leafchunk_base = ctl->leaf_chunks;
  for (uint32_t base = 0; base < n; base += blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    uint32_t v[6] = {0, 0, 0, 0, 0, 0};
    uint32_t tree = 0;
    bool first = false;
    if (i < n) {
      const NodeRec node = a.nodes[parity][i];
      tree = node.tree;
      first = i == 0 || a.nodes[parity][i - 1].tree != tree;
      const uint32_t within = a.scratch_prefix[i] - tree_base[tree];
      const bool acc = a.scratch_flags[i] && (a.trees[tree].leaf_count + within < P.max_leaves);
      v[0] = acc;
      if (acc) {
        const SplitRec& b = a.partial[size_t(i) * a.partial_stride];
        uint64_t left = b.lcount, right = b.rcount;
        fit_children(node.seg_cnt, left, right);
        const uint32_t built = uint32_t(left <= right ? left : right);
        if (!last) {
          v[1] = ceil_div(built, item_rows);
          v[2] = ceil_div(node.seg_cnt, kPartChunk);
        }
      }
      const bool leafseg = !acc || last;
      v[3] = leafseg;
      v[4] = leafseg ? ceil_div(node.seg_cnt, a.apply_chunk) : 0;
      v[5] = (!acc && !last) ? 1u : 0u;
    }
    const uint32_t own0 = v[0];
    uint32_t tot[6];
    block_scan<6>(v, tot, sh);
    if (i < n) {
      a.scratch_flags[i] = own0;
      a.scratch_prefix[i] = carry6[0] + v[0];
      a.scratch_aux[i] = carry6[5] + v[5];
      if (first) tree_acc_base[tree] = carry6[0] + v[0];
      if (own0) {
        const uint32_t k = carry6[0] + v[0];
        if (!last) {
          a.build_prefix[k] = carry6[1] + v[1];
          a.part_prefix[k] = carry6[2] + v[2];
        }
      }
      if (!own0 || last) a.leaf_prefix[leafseg_base + carry6[3] + v[3]] = leafchunk_base + carry6[4] + v[4];
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) carry6[k] += tot[k];
    __syncthreads();
  }
  const uint32_t n_acc = carry6[0];
  const uint32_t free_top = ctl->free_top;
  __syncthreads();

  // Phase B2: apply splits, next-level nodes, build / subtract / partition / leaf lists.
  uint32_t err = 0;
  NodeRec* next = a.nodes[parity ^ 1];
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
    const NodeRec node = a.nodes[parity][i];
    const uint32_t t = node.tree;
    TreeNodeOut* tn = a.tree_nodes + size_t(t) * a.max_tree_nodes;
    const bool acc = a.scratch_flags[i] != 0;
    if (acc) {
      SplitRec b = a.partial[size_t(i) * a.partial_stride];
      if (!fit_children(node.seg_cnt, b.lcount, b.rcount)) err |= kErrPartition;
      const uint32_t k = a.scratch_prefix[i];
      const uint32_t kt = k - tree_acc_base[t];
      atomicAdd(&tree_acc[t], 1u);
      const uint32_t li = a.trees[t].n_tree_nodes + 2 * kt, ri = li + 1;
      if (ri >= a.max_tree_nodes) {
        err |= kErrCapacity;
        continue;
      }
      double lv = 0.0, rv = 0.0;
      if (!bounded_leaf(P, b.lg, b.lh, b.ll, b.lu, &lv)) err |= kErrNonFinite;
      if (!bounded_leaf(P, b.rg, b.rh, b.rl, b.ru, &rv)) err |= kErrNonFinite;
      write_leaf(&tn[li], lv);
      write_leaf(&tn[ri], rv);
      TreeNodeOut& pn = tn[node.node_index];
      pn.feature_index = dataset_feature(a, t, b.feature);
      pn.threshold_bin = b.threshold;
      pn.left_child = li;
      pn.right_child = ri;
      pn.leaf_value = 0.0;
      pn.gain = b.gain;
      pn.default_left = uint8_t(b.default_left);
      pn.flags = 0;
      if (!last) {
        const bool build_left = b.lcount <= b.rcount;
        const uint32_t new_slot = a.free_stack[free_top - 1 - k];
        NodeRec L, R;
        L.seg_off = node.seg_off;
        L.seg_cnt = uint32_t(b.lcount);
        R.seg_off = node.seg_off + uint32_t(b.lcount);
        R.seg_cnt = uint32_t(b.rcount);
        L.node_index = li;
        R.node_index = ri;
        L.slot = build_left ? new_slot : node.slot;
        R.slot = build_left ? node.slot : new_slot;
        L.count = b.lcount;
        R.count = b.rcount;
        L.qg = b.lqg;
        L.qh = b.lqh;
        R.qg = b.rqg;
        R.qh = b.rqh;
        L.g = b.lg;
        L.h = b.lh;
        R.g = b.rg;
        R.h = b.rh;
        L.lo = b.ll;
        L.hi = b.lu;
        R.lo = b.rl;
        R.hi = b.ru;
        L.tree = R.tree = t;
        L.depth = R.depth = node.depth + 1;
        // The sibling of the built child keeps the parent's slot, from which the next
        // level's split scan (fused_sub) or subtract_kernel subtracts the built child's.
        L.sub_from = (a.fused_sub && !build_left) ? new_slot + 1 : 0;
        R.sub_from = (a.fused_sub && build_left) ? new_slot + 1 : 0;
        next[2 * k] = L;
        next[2 * k + 1] = R;
        for (uint32_t w = 0; w < W; ++w) {
          uint32_t path = a.node_path[parity][i * W + w];
          if ((b.feature >> 5) == w) path |= 1u << (b.feature & 31);
          a.node_path[parity ^ 1][(2 * k) * W + w] = path;
          a.node_path[parity ^ 1][(2 * k + 1) * W + w] = path;
        }
        for (uint32_t w = 0; w < W; ++w) {
          const uint32_t allowed = allowed_word(a, a.node_path[parity ^ 1] + size_t(2 * k) * W, t, w);
          a.node_allowed[parity ^ 1][(2 * k) * W + w] = allowed;
          a.node_allowed[parity ^ 1][(2 * k + 1) * W + w] = allowed;
        }
        BuildEntry be;
        be.tree = t;
        be.parity = uint32_t(parity ^ 1);
        be.seg_off = build_left ? L.seg_off : R.seg_off;
        be.seg_cnt = build_left ? L.seg_cnt : R.seg_cnt;
        be.slot = new_slot;
        be.pad = 0;
        a.build[k] = be;
        SubEntry se;
        se.parent_slot = node.slot;
        se.built_slot = new_slot;
        a.sub[k] = se;
        PartEntry pe;
        pe.tree = t;
        pe.parity = uint32_t(parity);
        pe.seg_off = node.seg_off;
        pe.seg_cnt = node.seg_cnt;
        pe.feature = dataset_feature(a, t, b.feature);
        pe.threshold = b.threshold;
        pe.default_left = b.default_left;
        pe.lcount = uint32_t(b.lcount);
        a.part[k] = pe;
      }
      if (last) {
        // leaf segment index: number of leaf segments before node i in this level
        // equals i (every node of the last level produces one).
        LeafSeg ls;
        ls.tree = t;
        ls.parity = uint32_t(parity);
        ls.seg_off = node.seg_off;
        ls.seg_cnt = node.seg_cnt;
        ls.split = 1;
        ls.feature = dataset_feature(a, t, b.feature);
        ls.threshold = b.threshold;
        ls.default_left = b.default_left;
        ls.value = 0.0;
        ls.left_value = lv;
        ls.right_value = rv;
        if (leafseg_base + i < a.max_leafsegs) a.leafseg[leafseg_base + i] = ls;
        else err |= kErrCapacity;
      }
    } else {
      // Node stays a leaf: its rows keep the current leaf value.
      const uint32_t before_acc = a.scratch_prefix[i];
      const uint32_t idx = last ? i : (i - before_acc);  // leaf segments before i
      LeafSeg ls;
      ls.tree = t;
      ls.parity = uint32_t(parity);
      ls.seg_off = node.seg_off;
      ls.seg_cnt = node.seg_cnt;
      ls.split = 0;
      ls.feature = ls.threshold = ls.default_left = 0;
      ls.value = tn[node.node_index].leaf_value;
      ls.left_value = ls.right_value = 0.0;
      if (leafseg_base + idx < a.max_leafsegs) a.leafseg[leafseg_base + idx] = ls;
      else err |= kErrCapacity;
    }
  }
  __syncthreads();
  // Phase C: free slots of nodes that stopped (non-last levels), counters.
  if (!last) {
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
      if (!a.scratch_flags[i]) {
        const uint32_t j = a.scratch_aux[i];
        a.free_stack[free_top - n_acc + j] = a.nodes[parity][i].slot;
      }
    }
  }
  __syncthreads();
  for (uint32_t t = threadIdx.x; t < a.n_trees; t += blockDim.x) {
    a.trees[t].n_tree_nodes += 2 * tree_acc[t];
    a.trees[t].leaf_count += tree_acc[t];
  }
  if (err) raise(ctl, err);
  if (threadIdx.x == 0) {
    const uint32_t n_leafseg_level = carry6[3];
    ctl->n_leafseg = leafseg_base + n_leafseg_level;
    ctl->leaf_chunks = leafchunk_base + carry6[4];
    if (leafseg_base + n_leafseg_level <= a.max_leafsegs)
      a.leaf_prefix[leafseg_base + n_leafseg_level] = leafchunk_base + carry6[4];
    if (last) {
      ctl->n_nodes = 0;
      ctl->n_build = 0;
      ctl->n_sub = 0;
      ctl->n_part = 0;
      ctl->hist_items = 0;
      ctl->part_chunks = 0;
    } else {
      ctl->free_top = free_top - n_acc + (n - n_acc);
      ctl->n_nodes = 2 * n_acc;
      ctl->n_build = n_acc;
      ctl->n_sub = n_acc;
      ctl->n_part = n_acc;
      a.build_prefix[n_acc] = carry6[1];
      a.part_prefix[n_acc] = carry6[2];
      ctl->hist_items = carry6[1] * a.nfb;
      ctl->part_chunks = carry6[2];
      ctl->item_rows = item_rows;
    }
    ctl->hist_counter = 0;
  }
}

// The finalize of a level with at most one node per thread (up to kNodeFinalizeMax): a
// node's record, split and prefixes stay in its thread's registers, where the general
// kernel walks the nodes in five passes that each read back from global memory what the
// pass before wrote. Latency-bound: a chain of three loads (counts, records, tree state),
// two block scans and the stores.
constexpr uint32_t kNodeFinalizeMax = 512;

__global__ void __launch_bounds__(kNodeFinalizeMax) finalize_nodes_kernel(TrainerDev a, int parity,
                                                                          uint32_t depth) {
  __shared__ uint32_t sh[33 * 6];
  __shared__ uint32_t s_valid_base[kNodeFinalizeMax], s_acc_base[kNodeFinalizeMax + 1];
  __shared__ uint32_t s_node_of[kNodeFinalizeMax];  // accepted split k: its node
  Control* ctl = a.ctl;
  launch_order();
  const TreeParams& P = a.params;
  const uint32_t n = ctl->n_nodes;
  const uint32_t free_top = ctl->free_top;
  const uint32_t leafseg_base = ctl->n_leafseg, leafchunk_base = ctl->leaf_chunks;
  const uint32_t W = P.path_words;
  const bool last = depth + 1 >= P.max_depth;  // children are leaves
  const uint32_t i = threadIdx.x;
  uint32_t err = 0;
  if (n > blockDim.x) {  // the launch covers the level's bound
    if (i == 0) raise(ctl, kErrCapacity);
    return;
  }
  NodeRec node;
  SplitRec b;
  node.tree = 0;
  node.seg_cnt = 0;
  b.valid = 0;
  uint32_t leaf_count = 0, tree_nodes = 0;
  bool first = false;
  double lv = 0.0, rv = 0.0;
  if (i < n) {
    node = a.nodes[parity][i];
    if (depth < P.max_depth) b = a.partial[size_t(i) * a.partial_stride];  // else: tree.cpp:152-154
    first = i == 0 || a.nodes[parity][i - 1].tree != node.tree;
    leaf_count = a.trees[node.tree].leaf_count;
    tree_nodes = a.trees[node.tree].n_tree_nodes;
  }
  const bool fits = !b.valid || fit_children(node.seg_cnt, b.lcount, b.rcount);
  const uint32_t built = b.valid ? uint32_t(b.lcount <= b.rcount ? b.lcount : b.rcount) : 0u;
  // Valid splits before the node and, through its tree's ordinal in the level, before its
  // tree's first node; rows the next level builds.
  uint32_t v3[3] = {b.valid ? 1u : 0u, (built + 255) / 256, first ? 1u : 0u}, tot3[3];
  block_scan<3>(v3, tot3, sh);
  const uint32_t ord = first ? v3[2] : (i < n ? v3[2] - 1 : 0u);
  if (first) s_valid_base[ord] = v3[0];
  __syncthreads();
  const uint32_t level_per_sm = level_items_per_sm(a, n);
  const uint32_t item_rows =
      a.item_rows ? a.item_rows : adaptive_item_rows(uint64_t(tot3[1]) * 256, a, level_per_sm, tot3[0]);
  const bool acc = i < n && b.valid && (leaf_count + (v3[0] - s_valid_base[ord]) < P.max_leaves);
  const bool leafseg = i < n && (!acc || last);
  // 0 accepted, 1 build chunks, 2 partition chunks, 3 leaf segments, 4 leaf chunks, 5 freed.
  uint32_t v[6] = {acc ? 1u : 0u,
                   acc && !last ? ceil_div(built, item_rows) : 0u,
                   acc && !last ? ceil_div(node.seg_cnt, kPartChunk) : 0u,
                   leafseg ? 1u : 0u,
                   leafseg ? ceil_div(node.seg_cnt, a.apply_chunk) : 0u,
                   i < n && !acc && !last ? 1u : 0u};
  uint32_t tot[6];
  block_scan<6>(v, tot, sh);
  const uint32_t n_acc = tot[0], k = v[0];
  if (first) s_acc_base[ord] = k;
  if (i == 0) s_acc_base[tot3[2]] = n_acc;
  if (acc) s_node_of[k] = i;
  const uint32_t new_slot = acc && !last ? a.free_stack[free_top - 1 - k] : 0u;
  if (acc) {
    if (!bounded_leaf(P, b.lg, b.lh, b.ll, b.lu, &lv)) err |= kErrNonFinite;
    if (!bounded_leaf(P, b.rg, b.rh, b.rl, b.ru, &rv)) err |= kErrNonFinite;
  }
  __syncthreads();  // also: the new slots are read before stopped nodes return theirs
  if (i < n) {
    const uint32_t t = node.tree;
    TreeNodeOut* tn = a.tree_nodes + size_t(t) * a.max_tree_nodes;
    LeafSeg ls;
    ls.tree = t;
    ls.parity = uint32_t(parity);
    ls.seg_off = node.seg_off;
    ls.seg_cnt = node.seg_cnt;
    ls.split = 0;
    ls.feature = ls.threshold = ls.default_left = 0;
    ls.value = ls.left_value = ls.right_value = 0.0;
    const uint32_t li = tree_nodes + 2 * (k - s_acc_base[ord]), ri = li + 1;
    const bool room = !acc || ri < a.max_tree_nodes;
    if (!room) err |= kErrCapacity;
    if (acc && room) {
      write_leaf(&tn[li], lv);
      write_leaf(&tn[ri], rv);
      TreeNodeOut& pn = tn[node.node_index];
      pn.feature_index = dataset_feature(a, t, b.feature);
      pn.threshold_bin = b.threshold;
      pn.left_child = li;
      pn.right_child = ri;
      pn.leaf_value = 0.0;
      pn.gain = b.gain;
      pn.default_left = uint8_t(b.default_left);
      pn.flags = 0;
      if (!fits) err |= kErrPartition;
      if (!last) {
        const bool build_left = b.lcount <= b.rcount;
        NodeRec c;  // the left child, then the right one
        c.tree = t;
        c.depth = node.depth + 1;
        c.seg_off = node.seg_off;
        c.seg_cnt = uint32_t(b.lcount);
        c.node_index = li;
        c.slot = build_left ? new_slot : node.slot;
        c.count = b.lcount;
        c.qg = b.lqg;
        c.qh = b.lqh;
        c.g = b.lg;
        c.h = b.lh;
        c.lo = b.ll;
        c.hi = b.lu;
        // The sibling of the built child keeps the parent's slot, from which the next
        // level's split scan (fused_sub) or subtract_kernel subtracts the built child's.
        c.sub_from = (a.fused_sub && !build_left) ? new_slot + 1 : 0;
        a.nodes[parity ^ 1][2 * k] = c;
        BuildEntry be;
        be.tree = t;
        be.parity = uint32_t(parity ^ 1);
        be.seg_off = node.seg_off;
        be.seg_cnt = uint32_t(b.lcount);
        be.slot = new_slot;
        be.pad = 0;
        c.seg_off = node.seg_off + uint32_t(b.lcount);
        c.seg_cnt = uint32_t(b.rcount);
        c.node_index = ri;
        c.slot = build_left ? node.slot : new_slot;
        c.count = b.rcount;
        c.qg = b.rqg;
        c.qh = b.rqh;
        c.g = b.rg;
        c.h = b.rh;
        c.lo = b.rl;
        c.hi = b.ru;
        c.sub_from = (a.fused_sub && build_left) ? new_slot + 1 : 0;
        a.nodes[parity ^ 1][2 * k + 1] = c;
        if (!build_left) {
          be.seg_off = c.seg_off;
          be.seg_cnt = c.seg_cnt;
        }
        a.build[k] = be;
        a.build_prefix[k] = v[1];
        a.sub[k] = SubEntry{node.slot, new_slot};
        PartEntry pe;
        pe.tree = t;
        pe.parity = uint32_t(parity);
        pe.seg_off = node.seg_off;
        pe.seg_cnt = node.seg_cnt;
        pe.feature = dataset_feature(a, t, b.feature);
        pe.threshold = b.threshold;
        pe.default_left = b.default_left;
        pe.lcount = uint32_t(b.lcount);
        a.part[k] = pe;
        a.part_prefix[k] = v[2];
        if (P.n_groups > 0) {
          uint32_t* path = a.node_path[parity ^ 1] + size_t(2 * k) * W;
          for (uint32_t w = 0; w < W; ++w) {
            uint32_t word = a.node_path[parity][size_t(i) * W + w];
            if ((b.feature >> 5) == w) word |= 1u << (b.feature & 31);
            path[w] = path[W + w] = word;
          }
          for (uint32_t w = 0; w < W; ++w) {
            const uint32_t word = allowed_word(a, path, t, w);
            a.node_allowed[parity ^ 1][size_t(2 * k) * W + w] = word;
            a.node_allowed[parity ^ 1][size_t(2 * k + 1) * W + w] = word;
          }
        }
      } else {
        ls.split = 1;
        ls.feature = dataset_feature(a, t, b.feature);
        ls.threshold = b.threshold;
        ls.default_left = b.default_left;
        ls.left_value = lv;
        ls.right_value = rv;
      }
    } else if (!acc) {
      ls.value = tn[node.node_index].leaf_value;  // the node's rows keep the current leaf value
      if (!last) a.free_stack[free_top - n_acc + v[5]] = node.slot;
    }
    if (leafseg) {
      const uint32_t at = leafseg_base + v[3];
      if (at < a.max_leafsegs) {
        a.leafseg[at] = ls;
        a.leaf_prefix[at] = leafchunk_base + v[4];
      } else {
        err |= kErrCapacity;
      }
    }
    if (first) {
      const uint32_t mine = s_acc_base[ord + 1] - s_acc_base[ord];
      a.trees[t].n_tree_nodes = tree_nodes + 2 * mine;
      a.trees[t].leaf_count = leaf_count + mine;
    }
  }
  // Without interaction groups a child's allowed features are its tree's (all, or a
  // forest tree's subset); its path is not needed.
  if (!last && P.n_groups == 0)
    for (uint32_t idx = i; idx < 2 * n_acc * W; idx += blockDim.x) {
      uint32_t word = 0xffffffffu;
      if (a.tree_feature_masks != nullptr) {
        const uint32_t t = a.nodes[parity][s_node_of[idx / (2 * W)]].tree;
        word = a.tree_feature_masks[size_t(t) * W + idx % W];
      }
      a.node_allowed[parity ^ 1][idx] = word;
    }
  if (err) raise(ctl, err);
  if (i == 0) {
    ctl->n_leafseg = leafseg_base + tot[3];
    ctl->leaf_chunks = leafchunk_base + tot[4];
    if (leafseg_base + tot[3] <= a.max_leafsegs) a.leaf_prefix[leafseg_base + tot[3]] = leafchunk_base + tot[4];
    const uint32_t acc_next = last ? 0u : n_acc;
    ctl->n_nodes = 2 * acc_next;
    ctl->n_build = acc_next;
    ctl->n_sub = acc_next;
    ctl->n_part = acc_next;
    ctl->hist_items = last ? 0u : tot[1] * a.nfb;
    ctl->part_chunks = last ? 0u : tot[2];
    if (!last) {
      ctl->free_top = free_top - n_acc + (n - n_acc);
      a.build_prefix[n_acc] = tot[1];
      a.part_prefix[n_acc] = tot[2];
      ctl->item_rows = item_rows;
    }
    ctl->hist_counter = 0;
  }
}

// ------------------------------------------------------------------------------------
// Partition
// ------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t find_entry(const uint32_t* prefix, uint32_t n, uint32_t c) {
  uint32_t lo = 0, hi = n;  // last entry with prefix <= c
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (prefix[mid] <= c) lo = mid; else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ bool row_goes_left(const TrainerDev& a, uint32_t row, uint32_t f,
                                              uint32_t thr, uint32_t dl) {
  // Feature-major copy: a node's rows are sorted, so neighbouring rows share sectors.
  uint32_t b, missing_slot;
  if (a.bins16_fm) {  // wide dataset (launch-uniform)
    b = a.bins16_fm[size_t(f) * a.n_rows + row];
    missing_slot = a.slots - 1;
  } else {
    b = a.bins_fm[size_t(f) * a.n_rows + row];
    missing_slot = kMissingSlot;
  }
  if (a.has_missing[f] && b == missing_slot) return dl != 0;
  return b <= thr;
}

constexpr int kPartThreads = 512;
constexpr int kPartPerThread = kPartChunk / kPartThreads;  // 8

__global__ void __launch_bounds__(kPartThreads) partition_count_kernel(TrainerDev a) {
  __shared__ uint32_t warp_counts[kPartThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  launch_order();
  for (uint32_t c = blockIdx.x; c < a.ctl->part_chunks; c += gridDim.x) {
    const uint32_t e = find_entry(a.part_prefix, a.ctl->n_part, c);
    const PartEntry pe = a.part[e];
    const uint32_t lc = c - a.part_prefix[e];
    const uint32_t start = lc * kPartChunk;
    const uint32_t count = min(kPartChunk, pe.seg_cnt - start);
    const uint32_t* rows = a.rows + (size_t(pe.tree) * 2 + pe.parity) * a.seg_stride + pe.seg_off + start;
    uint32_t mine = 0;
    // All row ids, then all bin gathers, then the stores: nothing in flight waits on a
    // store that might alias it.
    uint32_t r[kPartPerThread];
#pragma unroll
    for (int k = 0; k < kPartPerThread; ++k) {
      const uint32_t p = uint32_t(k * kPartThreads) + threadIdx.x;
      r[k] = p < count ? __ldg(rows + p) : 0xffffffffu;
    }
    bool left[kPartPerThread];
#pragma unroll
    for (int k = 0; k < kPartPerThread; ++k)
      left[k] = r[k] < a.n_rows && row_goes_left(a, r[k], pe.feature, pe.threshold, pe.default_left);
#pragma unroll
    for (int k = 0; k < kPartPerThread; ++k) {
      const uint32_t word = __ballot_sync(0xffffffffu, left[k]);
      if (lane == 0) a.part_flags[size_t(c) * (kPartChunk / 32) + k * (kPartThreads / 32) + warp] = word;
      mine += left[k];
    }
    for (int off = 16; off > 0; off >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, off);
    if (lane == 0) warp_counts[warp] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t s = 0;
      for (int w = 0; w < kPartThreads / 32; ++w) s += warp_counts[w];
      a.part_counts[c] = s;
    }
    __syncthreads();
  }
}

// Exclusive prefix of the chunk counts of each partitioned node.
__global__ void __launch_bounds__(1024) partition_scan_kernel(TrainerDev a) {
  __shared__ uint32_t sh[33];
  launch_order();
  uint32_t err = 0;
  for (uint32_t e = blockIdx.x; e < a.ctl->n_part; e += gridDim.x) {
    const uint32_t c0 = a.part_prefix[e], c1 = a.part_prefix[e + 1];
    uint32_t carry = 0;
    for (uint32_t base = c0; base < c1; base += blockDim.x) {
      const uint32_t c = base + threadIdx.x;
      uint32_t v[1] = {c < c1 ? a.part_counts[c] : 0u};
      uint32_t tot[1];
      block_scan<1>(v, tot, sh);
      if (c < c1) a.part_offsets[c] = carry + v[0];
      carry += tot[0];
    }
    if (carry != a.part[e].lcount) err |= kErrPartition;
    if (threadIdx.x == 0) atomicAdd(&a.ctl->rows_partitioned, (unsigned long long)a.part[e].seg_cnt);
    __syncthreads();
  }
  if (err && threadIdx.x == 0) raise(a.ctl, err);
}

__global__ void __launch_bounds__(kPartThreads) partition_scatter_kernel(TrainerDev a) {
  constexpr int kWords = kPartChunk / 32;  // 128
  __shared__ uint32_t word_prefix[kWords];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  launch_order();
  uint32_t err = 0;
  for (uint32_t c = blockIdx.x; c < a.ctl->part_chunks; c += gridDim.x) {
    const uint32_t e = find_entry(a.part_prefix, a.ctl->n_part, c);
    const PartEntry pe = a.part[e];
    const uint32_t lc = c - a.part_prefix[e];
    const uint32_t start = lc * kPartChunk;
    const uint32_t count = min(kPartChunk, pe.seg_cnt - start);
    const uint32_t* flags = a.part_flags + size_t(c) * kWords;
    // Exclusive prefix of the word popcounts, in position order.
    if (warp == 0) {
      uint32_t cnt[4], s = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        cnt[q] = __popc(flags[lane * 4 + q]);
        s += cnt[q];
      }
      uint32_t x = s;
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
      }
      uint32_t run = x - s;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        word_prefix[lane * 4 + q] = run;
        run += cnt[q];
      }
    }
    __syncthreads();
    const size_t src_off = (size_t(pe.tree) * 2 + pe.parity) * a.seg_stride + pe.seg_off + start;
    const size_t dst_off = (size_t(pe.tree) * 2 + (pe.parity ^ 1)) * a.seg_stride + pe.seg_off;
    const uint32_t* src = a.rows + src_off;
    uint32_t* dst = a.rows + dst_off;
    const float2* gh_src = a.gh_ordered ? a.gh + src_off : nullptr;
    float2* gh_dst = a.gh_ordered ? a.gh + dst_off : nullptr;
    const uint32_t left_before_chunk = a.part_offsets[c];
    const uint32_t right_before_chunk = start - left_before_chunk;
    // Loads first (flag words, row ids, g/h), then the stores.
    uint32_t word[kPartPerThread], r[kPartPerThread];
    float2 g[kPartPerThread];
#pragma unroll
    for (int k = 0; k < kPartPerThread; ++k) {
      const uint32_t p = uint32_t(k * kPartThreads) + threadIdx.x;
      word[k] = __ldg(flags + k * (kPartThreads / 32) + warp);
      r[k] = p < count ? __ldg(src + p) : 0u;
      g[k] = (p < count && a.gh_ordered) ? __ldg(gh_src + p) : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < kPartPerThread; ++k) {
      const uint32_t p = uint32_t(k * kPartThreads) + threadIdx.x;
      const int wi = k * (kPartThreads / 32) + warp;
      if (p < count) {
        const uint32_t below = __popc(word[k] & ((1u << lane) - 1u));
        const uint32_t lpos = word_prefix[wi] + below;  // left rows before p in the chunk
        const bool left = (word[k] >> lane) & 1u;
        const uint32_t rel = left ? left_before_chunk + lpos : pe.lcount + right_before_chunk + (p - lpos);
        if (rel < pe.seg_cnt) {  // always true when the counts agree
          dst[rel] = r[k];
          if (a.gh_ordered) gh_dst[rel] = g[k];
        } else {
          err = kErrPartition;
        }
      }
    }
    __syncthreads();
  }
  if (err) raise(a.ctl, err);
}

// One launch for levels of few rows: a thread-block cluster per split node. Each CTA routes
// a contiguous part of the node's rows (flags in shared memory), the CTAs read each other's
// left counts through distributed shared memory, and each writes its part. Bound by the
// latency of its two passes over the part; the three launches above, which spread a node's
// rows over the whole GPU, cost 20 us on a 100,000-row node where this takes one launch.
constexpr int kClusterThreads = 1024;
constexpr uint32_t kClusterPartRows = 65536;  // rows per CTA (flag words in shared memory)

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_ctas() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// The u32 at shared address `addr` of the cluster's CTA `rank`.
__device__ __forceinline__ uint32_t ld_cluster_u32(uint32_t addr, uint32_t rank) {
  uint32_t remote, v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.u32 %0, [%1];\n" : "=r"(v) : "r"(remote) : "memory");
  return v;
}

__global__ void __launch_bounds__(kClusterThreads) partition_cluster_kernel(TrainerDev a) {
  constexpr uint32_t kWords = kClusterPartRows / 32;
  constexpr int kUnroll = 4;
  __shared__ uint32_t s_flags[kWords], s_prefix[kWords];
  __shared__ uint32_t s_scan[33], s_left;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  launch_order();
  const uint32_t rank = cluster_rank(), ctas = cluster_ctas();
  const uint32_t n_part = a.ctl->n_part;
  uint32_t err = 0;
  for (uint32_t e = blockIdx.x / ctas; e < n_part; e += gridDim.x / ctas) {  // the cluster's nodes
    const PartEntry pe = a.part[e];
    // The CTA's rows: [start, start + count), whole 32-row words.
    const uint32_t per = ceil_div(ceil_div(pe.seg_cnt, ctas), 32u) * 32u;
    const uint32_t start = min(rank * per, pe.seg_cnt);
    uint32_t count = min(per, pe.seg_cnt - start);
    if (count > kClusterPartRows) {  // the launch is chosen for nodes that fit
      err |= kErrCapacity;
      count = 0;
    }
    const size_t src_off = (size_t(pe.tree) * 2 + pe.parity) * a.seg_stride + pe.seg_off + start;
    const size_t dst_off = (size_t(pe.tree) * 2 + (pe.parity ^ 1)) * a.seg_stride + pe.seg_off;
    const uint32_t* src = a.rows + src_off;
    uint32_t* dst = a.rows + dst_off;
    const uint32_t words = ceil_div(count, 32u);
    for (uint32_t p0 = 0; p0 < words * 32u; p0 += kUnroll * kClusterThreads) {
      uint32_t r[kUnroll];
#pragma unroll
      for (int k = 0; k < kUnroll; ++k) {
        const uint32_t p = p0 + uint32_t(k * kClusterThreads) + threadIdx.x;
        r[k] = p < count ? __ldg(src + p) : 0xffffffffu;
      }
      bool left[kUnroll];
#pragma unroll
      for (int k = 0; k < kUnroll; ++k)
        left[k] = r[k] < a.n_rows && row_goes_left(a, r[k], pe.feature, pe.threshold, pe.default_left);
#pragma unroll
      for (int k = 0; k < kUnroll; ++k) {
        const uint32_t word = __ballot_sync(0xffffffffu, left[k]);
        const uint32_t w = (p0 + uint32_t(k * kClusterThreads)) / 32u + uint32_t(warp);
        if (lane == 0 && w < words) s_flags[w] = word;
      }
    }
    __syncthreads();
    // Exclusive prefix of the words' left rows, a run of neighbouring words per thread.
    {
      constexpr uint32_t kRun = kWords / kClusterThreads;
      uint32_t c[kRun], v[1] = {0}, tot[1];
#pragma unroll
      for (uint32_t q = 0; q < kRun; ++q) {
        const uint32_t w = threadIdx.x * kRun + q;
        c[q] = w < words ? uint32_t(__popc(s_flags[w])) : 0u;
        v[0] += c[q];
      }
      block_scan<1>(v, tot, s_scan);
      uint32_t run = v[0];
#pragma unroll
      for (uint32_t q = 0; q < kRun; ++q) {
        const uint32_t w = threadIdx.x * kRun + q;
        if (w < words) s_prefix[w] = run;
        run += c[q];
      }
      if (threadIdx.x == 0) s_left = tot[0];
    }
    cluster_barrier();  // every CTA's left count (and this CTA's prefix) is written
    uint32_t left_before = 0, left_all = 0;
    {
      const uint32_t mine = uint32_t(lane) < ctas
                                ? ld_cluster_u32(static_cast<uint32_t>(__cvta_generic_to_shared(&s_left)), uint32_t(lane))
                                : 0u;
      left_all = __reduce_add_sync(0xffffffffu, mine);
      left_before = __reduce_add_sync(0xffffffffu, uint32_t(lane) < rank ? mine : 0u);
    }
    if (left_all != pe.lcount) err |= kErrPartition;
    if (rank == 0 && threadIdx.x == 0) atomicAdd(&a.ctl->rows_partitioned, (unsigned long long)pe.seg_cnt);
    const uint32_t right_before = start - left_before;
    const float2* gh_src = a.gh_ordered ? a.gh + src_off : nullptr;
    float2* gh_dst = a.gh_ordered ? a.gh + dst_off : nullptr;
    for (uint32_t p0 = 0; p0 < count; p0 += kUnroll * kClusterThreads) {
      uint32_t r[kUnroll];
      float2 g[kUnroll];
#pragma unroll
      for (int k = 0; k < kUnroll; ++k) {
        const uint32_t p = p0 + uint32_t(k * kClusterThreads) + threadIdx.x;
        r[k] = p < count ? __ldg(src + p) : 0u;
        g[k] = (p < count && a.gh_ordered) ? __ldg(gh_src + p) : make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int k = 0; k < kUnroll; ++k) {
        const uint32_t p = p0 + uint32_t(k * kClusterThreads) + threadIdx.x;
        if (p >= count) continue;
        const uint32_t word = s_flags[p >> 5];
        const uint32_t lpos = s_prefix[p >> 5] + uint32_t(__popc(word & ((1u << lane) - 1u)));
        const bool left = (word >> lane) & 1u;
        const uint32_t rel = left ? left_before + lpos : pe.lcount + right_before + (p - lpos);
        if (rel < pe.seg_cnt) {  // always true when the counts agree
          dst[rel] = r[k];
          if (a.gh_ordered) gh_dst[rel] = g[k];
        } else {
          err |= kErrPartition;
        }
      }
    }
    // No CTA exits or rewrites its count and flags while another reads the count.
    cluster_barrier();
  }
  if (err) raise(a.ctl, err);
}

// ------------------------------------------------------------------------------------
// Leaf-wise growth (TrainLeafWiseRegressionTree, tree_leafwise.cpp:56-142)
//
// Each step splits, in every tree, the active leaf with the largest gain (the smaller
// node index on equal gains); leaves at max_depth stay active but never split. A leaf's
// best split depends only on its rows, so it is scanned once, when the leaf is created
// (in fixed point the reference's re-evaluation reproduces the same split exactly). A
// step is: select (this kernel: choose, ApplySplit, children, work lists), partition of
// the chosen leaves, histogram of each smaller child, subtraction for its sibling, split
// scan of the children, merge (the children's best splits into the active lists).
// ------------------------------------------------------------------------------------
__device__ SplitRec merged_split(const TrainerDev& a, uint32_t i) {
  SplitRec b = a.partial[size_t(i) * a.partial_stride];
  for (uint32_t c = 1; c < a.partial_stride; ++c) {
    const SplitRec x = a.partial[size_t(i) * a.partial_stride + c];
    if (better_split(x, b)) b = x;
  }
  return b;
}

// Root of every tree becomes its first active leaf (after the level-0 split scan).
__global__ void leafwise_init_kernel(TrainerDev a) {
  launch_order();
  const TreeParams& P = a.params;
  const uint32_t W = P.path_words, T = a.n_trees, S = a.lw_slot_cap;
  for (uint32_t t = threadIdx.x; t < T; t += blockDim.x) {
    // Slot t holds the root (round_setup); the tree's other slots form its stack.
    for (uint32_t j = 0; j < S; ++j) a.lw_slots[size_t(t) * S + j] = T + t * S + j;
    a.lw_slot_top[t] = S;
    LeafActive r;
    r.node = a.nodes[0][t];
    r.best = P.max_depth > 0 ? merged_split(a, t) : no_split();
    r.parity = 0;
    r.scanned = 1;
    a.lw_active[size_t(t) * a.lw_cap] = r;
    for (uint32_t w = 0; w < W; ++w) {
      a.lw_path[size_t(t) * a.lw_cap * W + w] = 0;
      a.lw_allowed[size_t(t) * a.lw_cap * W + w] = a.node_allowed[0][t * W + w];
    }
    a.lw_count[t] = 1;
    a.lw_done[t] = 0;
  }
}

// A warp per tree, kSelectTrees at a time: the lanes compare the active leaves and copy the
// records, where one thread walked them before (29 us a step at 31 leaves).
constexpr uint32_t kSelectTrees = 8;

__global__ void __launch_bounds__(32 * kSelectTrees) leafwise_select_kernel(TrainerDev a) {
  __shared__ uint32_t sh[33 * 3];
  __shared__ unsigned long long built_rows;
  launch_order();
  const TreeParams& P = a.params;
  const uint32_t W = P.path_words, cap = a.lw_cap, S = a.lw_slot_cap;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) built_rows = 0;
  __syncthreads();
  uint32_t err = 0;
  uint32_t n_part = 0, n_build = 0, n_scan = 0;  // entries of the rounds before
  for (uint32_t base = 0; base < a.n_trees; base += blockDim.x / 32) {
    const uint32_t t = base + warp;
    bool split = false, build = false;
    uint32_t last = 0;
    PartEntry pe{};
    BuildEntry be{};
    SubEntry se{};
    LeafActive kid[2];
    const bool open = t < a.n_trees && !a.lw_done[t];  // the same in the whole warp
    __syncwarp();  // every lane has read lw_done, which lane 0 may set
    if (open) {
      LeafActive* act = a.lw_active + size_t(t) * cap;
      uint32_t* path = a.lw_path + size_t(t) * cap * W;
      uint32_t* allowed = a.lw_allowed + size_t(t) * cap * W;
      TreeState& ts = a.trees[t];
      const uint32_t cnt = a.lw_count[t], leaf_count = ts.leaf_count, tree_nodes = ts.n_tree_nodes;
      const uint32_t slot_top = a.lw_slot_top[t];
      uint32_t best = 0xffffffffu, best_node = 0xffffffffu;
      double best_gain = 0.0;
      if (cnt > a.lw_max_active) {
        err |= kErrLeafQueue;
      } else if (leaf_count < a.lw_max_leaves) {
        // IsBetterLeafWiseCandidate (tree_leafwise.cpp:16-27): the larger gain, then the
        // smaller node index.
        for (uint32_t j = lane; j < cnt; j += 32) {
          const LeafActive& l = act[j];
          const uint32_t d = l.node.depth, sc = l.scanned, va = l.best.valid, ni = l.node.node_index;
          const double g = l.best.gain;
          if (d >= P.max_depth || !sc || !va) continue;
          if (best == 0xffffffffu || g > best_gain || (g == best_gain && ni < best_node)) {
            best = j;
            best_gain = g;
            best_node = ni;
          }
        }
        for (int off = 16; off > 0; off >>= 1) {
          const uint32_t ob = __shfl_xor_sync(0xffffffffu, best, off);
          const uint32_t on = __shfl_xor_sync(0xffffffffu, best_node, off);
          const double og = __shfl_xor_sync(0xffffffffu, best_gain, off);
          if (ob != 0xffffffffu &&
              (best == 0xffffffffu || og > best_gain || (og == best_gain && on < best_node))) {
            best = ob;
            best_gain = og;
            best_node = on;
          }
        }
      }
      if (best == 0xffffffffu) {
        if (lane == 0) a.lw_done[t] = 1;
      } else {
        LeafActive c = act[best];  // every lane (the loads broadcast)
        const bool fits = fit_children(c.node.seg_cnt, c.best.lcount, c.best.rcount);
        const SplitRec& b = c.best;
        TreeNodeOut* tn = a.tree_nodes + size_t(t) * a.max_tree_nodes;
        const uint32_t li = tree_nodes, ri = li + 1;
        const uint32_t depth = c.node.depth + 1;
        const bool grow = depth < P.max_depth;
        const uint32_t new_slot = grow && slot_top ? a.lw_slots[size_t(t) * S + slot_top - 1] : 0xffffffffu;
        // Every lane holds the chosen leaf and the tree's counters: lane 0 and the copy below
        // overwrite them.
        __syncwarp();
        if (ri >= a.max_tree_nodes || cnt + 2 > cap || (grow && slot_top == 0)) {
          err |= kErrCapacity;
          if (lane == 0) a.lw_done[t] = 1;
        } else {
          // ApplySplit (tree_structure.cpp:118-148).
          double lv = 0.0, rv = 0.0;
          if (!bounded_leaf(P, b.lg, b.lh, b.ll, b.lu, &lv)) err |= kErrNonFinite;
          if (!bounded_leaf(P, b.rg, b.rh, b.rl, b.ru, &rv)) err |= kErrNonFinite;
          if (!fits) err |= kErrPartition;
          // Children in the other row buffer: left rows, then right rows (the partition).
          const uint32_t np = c.parity ^ 1u;
          const bool build_left = b.lcount <= b.rcount;
          if (lane == 0) {
            write_leaf(&tn[li], lv);
            write_leaf(&tn[ri], rv);
            TreeNodeOut& pn = tn[c.node.node_index];
            pn.feature_index = b.feature;
            pn.threshold_bin = b.threshold;
            pn.left_child = li;
            pn.right_child = ri;
            pn.leaf_value = 0.0;
            pn.gain = b.gain;
            pn.default_left = uint8_t(b.default_left);
            pn.flags = 0;
            ts.n_tree_nodes = tree_nodes + 2;
            ts.leaf_count = leaf_count + 1;
            // A leaf at max_depth has no child histograms: its slot is free again.
            if (!grow) a.lw_slots[size_t(t) * S + slot_top] = c.node.slot;
            a.lw_slot_top[t] = grow ? slot_top - 1 : slot_top + 1;
          }
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            NodeRec& n = kid[k].node;
            const bool left = k == 0;
            n.seg_off = left ? c.node.seg_off : c.node.seg_off + uint32_t(b.lcount);
            n.seg_cnt = uint32_t(left ? b.lcount : b.rcount);
            n.node_index = left ? li : ri;
            n.slot = !grow ? 0xffffffffu : ((left == build_left) ? new_slot : c.node.slot);
            n.count = left ? b.lcount : b.rcount;
            n.qg = left ? b.lqg : b.rqg;
            n.qh = left ? b.lqh : b.rqh;
            n.g = left ? b.lg : b.rg;
            n.h = left ? b.lh : b.rh;
            n.lo = left ? b.ll : b.rl;
            n.hi = left ? b.lu : b.ru;
            n.tree = t;
            n.depth = depth;
            // As in finalize: the sibling of the built child keeps the parent's slot.
            n.sub_from = (a.fused_sub && grow && left != build_left) ? new_slot + 1 : 0;
            kid[k].best = no_split();
            kid[k].parity = np;
            kid[k].scanned = grow ? 0u : 1u;
          }
          last = cnt - 1;
          if (P.n_groups > 0) {
            // Children's path and allowed words go to positions cnt, cnt + 1 (free), the
            // chosen leaf's place takes the last leaf, then the children move down by one.
            if (lane == 0) {
              for (uint32_t k = 0; k < 2; ++k)
                for (uint32_t w = 0; w < W; ++w) {
                  uint32_t pw = path[size_t(best) * W + w];
                  if ((b.feature >> 5) == w) pw |= 1u << (b.feature & 31);
                  path[size_t(cnt + k) * W + w] = pw;
                }
              for (uint32_t w = 0; w < W; ++w) {
                const uint32_t al = allowed_word(a, path + size_t(cnt) * W, t, w);
                allowed[size_t(cnt) * W + w] = al;
                allowed[size_t(cnt + 1) * W + w] = al;
              }
              for (uint32_t w = 0; w < W && best != last; ++w) {
                path[size_t(best) * W + w] = path[size_t(last) * W + w];
                allowed[size_t(best) * W + w] = allowed[size_t(last) * W + w];
              }
              for (uint32_t k = 0; k < 2; ++k)
                for (uint32_t w = 0; w < W; ++w) {
                  path[size_t(last + k) * W + w] = path[size_t(cnt + k) * W + w];
                  allowed[size_t(last + k) * W + w] = allowed[size_t(cnt + k) * W + w];
                }
            }
          }
          if (best != last) {  // the chosen leaf's place takes the last leaf, word by word
            static_assert(sizeof(LeafActive) % 8 == 0, "a warp copies 8-byte words");
            const unsigned long long* src = reinterpret_cast<const unsigned long long*>(act + last);
            unsigned long long* dst = reinterpret_cast<unsigned long long*>(act + best);
            for (uint32_t q = lane; q < sizeof(LeafActive) / 8; q += 32) dst[q] = src[q];
          }
          __syncwarp();
          if (lane < 2) act[last + lane] = lane == 0 ? kid[0] : kid[1];
          // Room for both children (tree_leafwise.cpp:130-134).
          const bool full = !(cnt - 1 + 2 <= a.lw_max_active || leaf_count + 1 >= a.lw_max_leaves);
          if (full) err |= kErrLeafQueue;
          if (lane == 0) {
            a.lw_count[t] = cnt + 1;
            if (full) a.lw_done[t] = 1;
          }
          split = true;
          pe.tree = t;
          pe.parity = c.parity;
          pe.seg_off = c.node.seg_off;
          pe.seg_cnt = c.node.seg_cnt;
          pe.feature = b.feature;
          pe.threshold = b.threshold;
          pe.default_left = b.default_left;
          pe.lcount = uint32_t(b.lcount);
          if (grow) {
            build = true;
            be.tree = t;
            be.parity = np;
            be.seg_off = build_left ? kid[0].node.seg_off : kid[1].node.seg_off;
            be.seg_cnt = build_left ? kid[0].node.seg_cnt : kid[1].node.seg_cnt;
            be.slot = new_slot;
            be.pad = 0;
            se.parent_slot = c.node.slot;
            se.built_slot = new_slot;
            if (lane == 0) atomicAdd(&built_rows, (unsigned long long)be.seg_cnt);
          }
        }
      }
    }
    const bool lead = lane == 0;  // the warp's entries
    uint32_t v[2] = {lead && split ? 1u : 0u, lead && build ? 1u : 0u}, tot[2];
    block_scan<2>(v, tot, sh);
    const uint32_t at_part = n_part + __shfl_sync(0xffffffffu, v[0], 0);
    const uint32_t at_build = n_build + __shfl_sync(0xffffffffu, v[1], 0);
    if (lead && split) a.part[at_part] = pe;
    if (build) {
      // Both children of a grown leaf are scanned: two scan entries per build entry.
      if (lead) {
        a.build[at_build] = be;
        a.sub[at_build] = se;
      }
      if (lane < 2) {
        a.nodes[1][2 * at_build + lane] = lane == 0 ? kid[0].node : kid[1].node;
        a.lw_scan_map[2 * at_build + lane] = (t << 16) | (last + lane);
      }
      for (uint32_t w = lane; w < 2 * W; w += 32) {
        const uint32_t word = w < W ? w : w - W;
        uint32_t al = 0xffffffffu;
        if (P.n_groups > 0) al = a.lw_allowed[(size_t(t) * cap + last) * W + word];
        else if (a.tree_feature_masks != nullptr) al = a.tree_feature_masks[t * W + word];
        a.node_allowed[1][size_t(2 * at_build) * W + w] = al;
      }
    }
    n_part += tot[0];
    n_build += tot[1];
    n_scan += 2 * tot[1];
  }
  if (err) raise(a.ctl, err);
  __syncthreads();
  if (warp == 0) {  // work lists of the step, 32 entries at a time
    Control* ctl = a.ctl;
    const uint32_t item_rows =
        a.item_rows ? a.item_rows : adaptive_item_rows(built_rows, a, a.items_per_sm ? a.items_per_sm : default_items_per_sm(a.slots), a.n_trees);
    auto prefix = [&](uint32_t n, uint32_t* out, auto&& chunks_of) -> uint32_t {
      uint32_t acc = 0;
      for (uint32_t e0 = 0; e0 < n; e0 += 32) {
        const uint32_t e = e0 + lane;
        const uint32_t own = e < n ? chunks_of(e) : 0u;
        uint32_t x = own;
        for (int off = 1; off < 32; off <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
          if (lane >= uint32_t(off)) x += y;
        }
        if (e < n) out[e] = acc + x - own;
        acc += __shfl_sync(0xffffffffu, x, 31);
      }
      if (lane == 0) out[n] = acc;
      return acc;
    };
    const uint32_t part_chunks =
        prefix(n_part, a.part_prefix, [&](uint32_t e) { return ceil_div(a.part[e].seg_cnt, kPartChunk); });
    const uint32_t build_chunks =
        prefix(n_build, a.build_prefix, [&](uint32_t e) { return ceil_div(a.build[e].seg_cnt, item_rows); });
    if (lane == 0) {
      ctl->n_part = n_part;
      ctl->part_chunks = part_chunks;
      ctl->n_build = n_build;
      ctl->n_sub = n_build;
      ctl->hist_items = build_chunks * a.nfb;
      ctl->hist_counter = 0;
      ctl->item_rows = item_rows;
      ctl->n_nodes = n_scan;
    }
  }
}

// The children's best splits into their active entries (after a one-launch scan).
__global__ void leafwise_merge_kernel(TrainerDev a) {
  for (uint32_t s = threadIdx.x; s < a.ctl->n_nodes; s += blockDim.x) {
    const uint32_t m = a.lw_scan_map[s];
    LeafActive& l = a.lw_active[size_t(m >> 16) * a.lw_cap + (m & 0xFFFFu)];
    l.best = merged_split(a, s);
    l.scanned = 1;
  }
}

// Every active leaf becomes a leaf segment of the prediction update: one warp, a leaf per
// lane.
__global__ void leafwise_finish_kernel(TrainerDev a) {
  launch_order();
  const uint32_t lane = threadIdx.x;
  Control* ctl = a.ctl;
  uint32_t n = 0, chunks = 0, err = 0;
  for (uint32_t t = 0; t < a.n_trees; ++t) {
    const LeafActive* act = a.lw_active + size_t(t) * a.lw_cap;
    const TreeNodeOut* tn = a.tree_nodes + size_t(t) * a.max_tree_nodes;
    const uint32_t count = a.lw_count[t];
    for (uint32_t j0 = 0; j0 < count; j0 += 32) {
      const uint32_t j = j0 + lane;
      LeafSeg ls{};
      if (j < count) {
        ls.tree = t;
        ls.parity = act[j].parity;
        ls.seg_off = act[j].node.seg_off;
        ls.seg_cnt = act[j].node.seg_cnt;
        ls.value = tn[act[j].node.node_index].leaf_value;
      }
      const uint32_t own = j < count ? ceil_div(ls.seg_cnt, a.apply_chunk) : 0u;
      uint32_t x = own;
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= uint32_t(off)) x += y;
      }
      if (j < count) {
        if (n + lane < a.max_leafsegs) {
          a.leafseg[n + lane] = ls;
          a.leaf_prefix[n + lane] = chunks + x - own;
        } else {
          err |= kErrCapacity;
        }
      }
      n += min(32u, count - j0);
      chunks += __shfl_sync(0xffffffffu, x, 31);
    }
  }
  if (__any_sync(0xffffffffu, err != 0)) {
    if (lane == 0) raise(ctl, kErrCapacity);
    n = min(n, a.max_leafsegs);
  }
  if (lane == 0) {
    a.leaf_prefix[n] = chunks;
    ctl->n_leafseg = n;
    ctl->leaf_chunks = chunks;
    ctl->n_nodes = ctl->n_build = ctl->n_sub = ctl->n_part = 0;
    ctl->hist_items = ctl->part_chunks = 0;
  }
}

// ------------------------------------------------------------------------------------
// Leaf application and round end
// ------------------------------------------------------------------------------------
// The prediction update runs in two passes. The first walks the leaf segments (a
// segment's rows ascend but are spread over the whole row range), routes the rows of
// last-level splits, and records per row which of its segment's steps applies (a 4-byte
// scattered write into an array that stays in L2); the second walks the rows in order and
// adds that step to the row's prediction, so the FP64 predictions are read and written as
// streams instead of one 32-byte sector each way per row.
constexpr uint32_t kNoLeaf = 0xffffffffu;

// The launch also ends the round: each tree's nodes go to the model, and the round counter
// moves on (the launches after it read the round from ctl).
__global__ void __launch_bounds__(256, 4) apply_leaves_kernel(TrainerDev a) {
  launch_order();
  const uint32_t round = a.ctl->round;
  if (round < a.max_rounds) {
    static_assert(sizeof(TreeNodeOut) % 8 == 0, "nodes are copied as 8-byte words");
    for (uint32_t t = blockIdx.x; t < a.n_trees; t += gridDim.x) {
      const uint32_t cnt = a.trees[t].n_tree_nodes;
      const unsigned long long* src =
          reinterpret_cast<const unsigned long long*>(a.tree_nodes + size_t(t) * a.max_tree_nodes);
      unsigned long long* dst = reinterpret_cast<unsigned long long*>(
          a.model_nodes + (size_t(round) * a.n_trees + t) * a.max_tree_nodes);
      for (uint32_t i = threadIdx.x; i < cnt * uint32_t(sizeof(TreeNodeOut) / 8); i += blockDim.x) dst[i] = src[i];
      if (threadIdx.x == 0) a.model_counts[size_t(round) * a.n_trees + t] = cnt;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.round_counter = round + 1;
  } else if (blockIdx.x == 0 && threadIdx.x == 0) {
    raise(a.ctl, kErrCapacity);
  }
  if (a.skip_apply) return;  // forest trees: no training predictions
  const double lr = a.params.learning_rate;
  uint32_t err = 0;
  const uint32_t n_seg = a.ctl->n_leafseg;
  const uint32_t chunks = a.ctl->leaf_chunks;
  for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x) {
    const uint32_t s = find_entry(a.leaf_prefix, n_seg, c);
    const LeafSeg ls = a.leafseg[s];
    const uint32_t start = (c - a.leaf_prefix[s]) * a.apply_chunk;
    const uint32_t count = min(a.apply_chunk, ls.seg_cnt - start);
    const uint32_t* rows = a.rows + (size_t(ls.tree) * 2 + ls.parity) * a.seg_stride + ls.seg_off + start;
    uint32_t* leaf_of = a.leaf_of + size_t(ls.tree) * a.n_rows;
    if (start == 0 && threadIdx.x == 0) {
      // lr * leaf is the same product for every row of a leaf.
      const double step = __dmul_rn(lr, ls.value);
      a.leaf_steps[2 * s] = ls.split ? __dmul_rn(lr, ls.left_value) : step;
      a.leaf_steps[2 * s + 1] = ls.split ? __dmul_rn(lr, ls.right_value) : step;
    }
    // Eight rows per thread at a time: row ids, then the routing gathers, then the stores.
    constexpr int B = 8;
    for (uint32_t p0 = 0; p0 < count; p0 += B * blockDim.x) {
      uint32_t r[B];
#pragma unroll
      for (int k = 0; k < B; ++k) {
        const uint32_t p = p0 + k * blockDim.x + threadIdx.x;
        r[k] = p < count ? __ldg(rows + p) : kNoLeaf;
      }
      uint32_t side[B];
#pragma unroll
      for (int k = 0; k < B; ++k)
        side[k] = (ls.split && r[k] < a.n_rows &&
                   !row_goes_left(a, r[k], ls.feature, ls.threshold, ls.default_left)) ? 1u : 0u;
#pragma unroll
      for (int k = 0; k < B; ++k) {
        const uint32_t p = p0 + k * blockDim.x + threadIdx.x;
        if (p >= count) continue;
        if (r[k] >= a.n_rows) {
          err = kErrCapacity;
          continue;
        }
        leaf_of[r[k]] = 2 * s + side[k];
      }
    }
  }
  if (err) raise(a.ctl, err);
}

// Row order: prediction += the step recorded for the row, then the record is cleared, so
// a row that no leaf segment covered in a round is caught in the next.
__global__ void __launch_bounds__(256) apply_steps_kernel(TrainerDev a) {
  launch_order();
  if (a.skip_apply) return;
  uint32_t err = 0;
  const uint32_t steps = 2 * a.ctl->n_leafseg;
  // Softmax trees update the margins of the current round's class.
  const uint32_t klass = a.n_classes ? a.ctl->round % a.n_classes : 0u;
  const size_t total = size_t(a.n_trees) * a.n_rows;
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += size_t(gridDim.x) * blockDim.x) {
    const uint32_t t = uint32_t(i / a.n_rows);
    const uint32_t r = uint32_t(i - size_t(t) * a.n_rows);
    const uint32_t idx = a.leaf_of[i];
    if (idx >= steps) {
      err = kErrPartition;
      continue;
    }
    a.leaf_of[i] = kNoLeaf;
    double* pred = a.preds + size_t(a.n_classes ? klass : t) * a.n_rows;
    const double out = __dadd_rn(pred[r], a.leaf_steps[idx]);
    if (!f64_finite(out)) err = kErrNonFinite;
    pred[r] = out;
  }
  if (err) raise(a.ctl, err);
}

// ---- Forest trees ----------------------------------------------------------------------
// A tree's sample is given as row multiplicities (u8 per row); its root segment is the
// rows in ascending order, each as often as it was drawn. Rows in chunks of kExpandChunk:
// chunk sums, a prefix per tree, then each chunk writes its part. HBM-bound: one byte read
// twice and four written per row. Grid (chunks, trees).
constexpr uint32_t kExpandThreads = 256, kExpandPer = 16;
static_assert(kExpandChunk == kExpandThreads * kExpandPer, "a thread expands kExpandPer rows");

__device__ __forceinline__ uint32_t expand_counts(const uint8_t* counts, uint32_t n, uint32_t row0,
                                                  uint32_t (&c)[kExpandPer]) {
  uint32_t sum = 0;
#pragma unroll
  for (uint32_t k = 0; k < kExpandPer; ++k) {
    c[k] = row0 + k < n ? counts[row0 + k] : 0u;
    sum += c[k];
  }
  return sum;
}

__global__ void __launch_bounds__(kExpandThreads) expand_sum_kernel(const uint8_t* counts, uint32_t n,
                                                                    uint32_t* chunk_sum) {
  __shared__ uint32_t sh[33];
  uint32_t c[kExpandPer], v[1], tot[1];
  const uint32_t row0 = blockIdx.x * kExpandChunk + threadIdx.x * kExpandPer;
  v[0] = expand_counts(counts + size_t(blockIdx.y) * n, n, row0, c);
  block_scan<1>(v, tot, sh);
  if (threadIdx.x == 0) chunk_sum[size_t(blockIdx.y) * gridDim.x + blockIdx.x] = tot[0];
}

__global__ void __launch_bounds__(1024) expand_scan_kernel(uint32_t* chunk_sum, uint32_t chunks) {
  __shared__ uint32_t sh[33];
  uint32_t* c = chunk_sum + size_t(blockIdx.x) * chunks;
  uint32_t carry = 0;
  for (uint32_t base = 0; base < chunks; base += blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    uint32_t v[1] = {i < chunks ? c[i] : 0u}, tot[1];
    block_scan<1>(v, tot, sh);
    if (i < chunks) c[i] = carry + v[0];
    carry += tot[0];
  }
}

__global__ void __launch_bounds__(kExpandThreads) expand_write_kernel(const uint8_t* counts, uint32_t n,
                                                                      const uint32_t* chunk_begin, uint32_t cap,
                                                                      uint32_t* sample) {
  __shared__ uint32_t sh[33];
  uint32_t c[kExpandPer], v[1], tot[1];
  const uint32_t row0 = blockIdx.x * kExpandChunk + threadIdx.x * kExpandPer;
  v[0] = expand_counts(counts + size_t(blockIdx.y) * n, n, row0, c);
  block_scan<1>(v, tot, sh);
  uint32_t at = chunk_begin[size_t(blockIdx.y) * gridDim.x + blockIdx.x] + v[0];
  uint32_t* out = sample + size_t(blockIdx.y) * cap;
  for (uint32_t k = 0; k < kExpandPer; ++k)
    for (uint32_t r = 0; r < c[k]; ++r, ++at)
      if (at < cap) out[at] = row0 + k;  // always: cap is the largest sample
}

// Compact forests: each tree's own features, [trees][n][nfb * 32] u8 rows, from the
// feature-major bins (a tree of 10 of 100 features then builds one feature block and 10
// features' histograms instead of four and 100). A thread takes four rows: a 4-byte load
// per feature, 4 x 4 byte transposes in registers, one 32-byte store per row. Grid (row
// tiles of 512, feature blocks, trees); feature_of 0xffffffff: no feature.
__global__ void __launch_bounds__(128) pack_tree_bins_kernel(const uint8_t* bins_fm, uint32_t n,
                                                             const uint32_t* feature_of, uint32_t features,
                                                             uint32_t nfb, uint8_t* out) {
  const uint32_t tree = blockIdx.z, fb = blockIdx.y;
  const uint32_t row = blockIdx.x * 512 + threadIdx.x * 4;
  if (row >= n) return;
  const bool words = n % 4 == 0;  // every feature's rows start on a word
  uint32_t w[32];
#pragma unroll
  for (uint32_t c = 0; c < 32; ++c) {
    const uint32_t f = fb * 32 + c;
    const uint32_t df = f < features ? __ldg(feature_of + size_t(tree) * features + f) : 0xffffffffu;
    w[c] = 0;
    if (df != 0xffffffffu) {
      const uint8_t* src = bins_fm + size_t(df) * n + row;
      if (words) {
        w[c] = __ldg(reinterpret_cast<const uint32_t*>(src));
      } else {
        for (uint32_t q = 0; q < 4 && row + q < n; ++q) w[c] |= uint32_t(__ldg(src + q)) << (8 * q);
      }
    }
  }
#pragma unroll
  for (uint32_t r = 0; r < 4; ++r) {
    uint32_t v[8];
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q) {
      const uint32_t lo = __byte_perm(w[4 * q], w[4 * q + 1], r | ((4 + r) << 4));
      const uint32_t hi = __byte_perm(w[4 * q + 2], w[4 * q + 3], r | ((4 + r) << 4));
      v[q] = __byte_perm(lo, hi, 0x5410);
    }
    if (row + r < n)
      asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(
                       out + ((size_t(tree) * n + row + r) * nfb + fb) * 32),
                   "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                   : "memory");
  }
}

// Rows of each class id 0..classes-1 (counts[classes]: rows whose label is none of them).
// The class priors and the logistic base score of an unweighted fit are these whole
// numbers, in any order of addition. HBM-bound (8 B per row); shared-memory counters per
// CTA.
__global__ void __launch_bounds__(256) label_counts_kernel(const double* labels, uint64_t n, uint32_t classes,
                                                           unsigned long long* counts) {
  extern __shared__ uint32_t s_counts[];  // [classes + 1]
  for (uint32_t k = threadIdx.x; k <= classes; k += blockDim.x) s_counts[k] = 0;
  __syncthreads();
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) {
    const double y = labels[i];
    const bool id = y >= 0.0 && y < double(classes) && floor(y) == y;
    atomicAdd(s_counts + (id ? uint32_t(y) : classes), 1u);
  }
  __syncthreads();
  for (uint32_t k = threadIdx.x; k <= classes; k += blockDim.x)
    if (s_counts[k]) atomicAdd(counts + k, (unsigned long long)s_counts[k]);
}

// ------------------------------------------------------------------------------------
// Standalone entries
// ------------------------------------------------------------------------------------
__global__ void squared_error_kernel(const double* labels, const double* preds, uint64_t n,
                                     double* out, uint32_t* error) {
  uint32_t bad = 0;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n;
       i += uint64_t(gridDim.x) * blockDim.x) {
    const double y = labels[i], p = preds[i];
    const double g = __dadd_rn(p, -y);
    if (!isfinite(y) || !isfinite(p) || !isfinite(g)) bad = 1;
    out[2 * i] = g;
    out[2 * i + 1] = 1.0;
  }
  if (bad) atomicOr(error, kErrGradient);
}

// RegressionModel::Predict (trainer.cpp:268-282): per row, trees in order,
// result += lr * leaf; traversal of RegressionTree::Predict (tree.cpp:179-214).
// BinT: u8 bins (missing rows at 255) or u16 bins of a wide dataset (at missing_slot).
template <typename BinT>
__global__ void predict_kernel(const BinT* bins_fm, uint32_t missing_slot, uint32_t n_rows,
                               const uint8_t* has_missing, const TreeNodeOut* nodes,
                               const uint32_t* tree_offsets, uint32_t n_trees, double base,
                               double lr, double* out, uint32_t* error) {
  uint32_t bad = 0;
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += gridDim.x * blockDim.x) {
    double acc = base;
    for (uint32_t t = 0; t < n_trees; ++t) {
      const TreeNodeOut* tn = nodes + tree_offsets[t];
      const uint32_t size = tree_offsets[t + 1] - tree_offsets[t];
      uint32_t node = 0, visited = 0;
      for (;;) {
        if (node >= size || ++visited > size) {
          bad = 1;
          break;
        }
        const TreeNodeOut nd = tn[node];
        if (nd.flags & 1u) {
          acc = __dadd_rn(acc, __dmul_rn(lr, nd.leaf_value));
          break;
        }
        const uint32_t f = nd.feature_index;
        const uint32_t b = bins_fm[size_t(f) * n_rows + r];
        const bool left = (has_missing[f] && b == missing_slot) ? nd.default_left != 0
                                                                : b <= nd.threshold_bin;
        node = left ? nd.left_child : nd.right_child;
      }
    }
    out[r] = acc;
  }
  if (bad) atomicOr(error, kErrCapacity);
}

// The same traversal from shared memory, for trees that fit its node format (PackedForest).
// A CTA stages the bins of its rows ([feature][row], one row per thread) and walks the
// trees in groups whose nodes and leaf steps it stages too, so a node visit is two
// shared-memory loads where the general kernel above loads a 40-byte node and gathers a
// byte from a 32-byte sector of the feature-major matrix. Bound by shared-memory load
// latency and bank conflicts between lanes at different nodes.
template <typename BinT>
__global__ void __launch_bounds__(1024) predict_packed_kernel(const BinT* bins_fm, uint32_t missing_slot,
                                                              uint32_t n_rows, uint32_t features,
                                                              PackedForest f, double base, double* out) {
  extern __shared__ __align__(16) unsigned char predict_smem[];
  const uint32_t rows = blockDim.x;
  const uint32_t pitch = predict_pitch<BinT>(rows);
  double* s_steps = reinterpret_cast<double*>(predict_smem);                       // [kPredictLeaves]
  uint2* s_nodes = reinterpret_cast<uint2*>(s_steps + kPredictLeaves);             // [kPredictNodes]
  BinT* s_bins = reinterpret_cast<BinT*>(s_nodes + kPredictNodes);                 // [features][pitch]
  const uint32_t row0 = blockIdx.x * rows, row = row0 + threadIdx.x;
  if (size_t(n_rows) * sizeof(BinT) % 4 == 0 && row0 + rows <= n_rows) {  // whole words (rows is a multiple of 128)
    const uint32_t words = rows * uint32_t(sizeof(BinT)) / 4, pitch4 = pitch * uint32_t(sizeof(BinT)) / 4;
    const uint32_t per = rows / words;  // features per pass
    const uint32_t w = threadIdx.x % words;
    for (uint32_t c = threadIdx.x / words; c < features; c += per)
      reinterpret_cast<uint32_t*>(s_bins)[size_t(c) * pitch4 + w] =
          __ldg(reinterpret_cast<const uint32_t*>(bins_fm + size_t(c) * n_rows + row0) + w);
  } else {
    for (uint32_t c = 0; c < features; ++c)
      s_bins[size_t(c) * pitch + threadIdx.x] = row < n_rows ? bins_fm[size_t(c) * n_rows + row] : BinT(0);
  }
  const BinT* mine = s_bins + threadIdx.x;
  double acc = base;
  for (uint32_t g = 0; g < f.n_groups; ++g) {
    const uint32_t t0 = f.group_first[g], t1 = f.group_first[g + 1];
    const uint4 first = f.trees[t0], end = f.trees[t1];  // {first node, first leaf, root, 0}
    __syncthreads();  // the group before is done (and the bins are staged)
    for (uint32_t i = threadIdx.x; i < end.x - first.x; i += rows) s_nodes[i] = f.nodes[first.x + i];
    for (uint32_t i = threadIdx.x; i < end.y - first.y; i += rows) s_steps[i] = f.steps[first.y + i];
    __syncthreads();
    for (uint32_t t = t0; t < t1; ++t) {
      const uint4 tree = f.trees[t];
      const uint2* nodes = s_nodes + (tree.x - first.x);
      uint32_t ref = tree.z;
      while (!(ref & kPackedLeaf)) {  // children follow their parents
        const uint2 nd = nodes[ref];
        const uint32_t b = mine[size_t(nd.x >> 17) * pitch];
        const bool left = b <= (nd.x & 0xFFFFu) || ((nd.x & 0x10000u) && b == missing_slot);
        ref = left ? nd.y & 0xFFFFu : nd.y >> 16;
      }
      acc = __dadd_rn(acc, s_steps[tree.y - first.y + (ref & ~kPackedLeaf)]);
    }
  }
  if (row < n_rows) out[row] = acc;
}

// Feature-major [features][rows] bins (u8 or u16) + optional missing mask -> three u8
// layouts with missing rows at 255: rows padded to nfb * 32 bytes and column blocks
// [nfb][rows][32] (histograms of sparse and dense levels), and a feature-major copy (row
// routing). Out-of-range bins set bit 0 of `error`.
// Feature block fb0 + blockIdx.y of the dataset. `src` and `missing` hold the features from
// src_f0 on (the whole matrix: src_f0 = 0; one staged feature block: src_f0 = 32 * fb0).
__global__ void pack_bins_kernel(const void* src, uint32_t width, const uint8_t* missing,
                                 const uint32_t* bin_count, uint32_t n_rows, uint32_t features,
                                 uint32_t nfb, uint8_t* out, uint8_t* out_blocked,
                                 uint8_t* out_fm, uint32_t* error, uint32_t fb0, uint32_t src_f0) {
  __shared__ uint8_t tile[32][129];
  const uint32_t fb = fb0 + blockIdx.y;
  uint32_t bad = 0;
  for (uint32_t r0 = blockIdx.x * 128; r0 < n_rows; r0 += gridDim.x * 128) {
    // load 32 features x 128 rows (coalesced along rows)
    if (width == 1 && n_rows % 16 == 0 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0 &&
        (reinterpret_cast<uintptr_t>(missing) & 15u) == 0) {
      // Sixteen rows per thread: 8 threads read one feature's 128 rows, a warp four
      // features (four 128-byte requests per instruction).
      for (uint32_t k = threadIdx.x; k < 32 * 8; k += blockDim.x) {
        const uint32_t c = k / 8, r = (k % 8) * 16;
        const uint32_t f = fb * 32 + c, row = r0 + r;
        uint4 out4 = make_uint4(0, 0, 0, 0);
        if (f < features && row < n_rows) {  // n_rows % 16 == 0: all sixteen rows exist
          const size_t idx = size_t(f) * n_rows + row, sidx = size_t(f - src_f0) * n_rows + row;
          const uint4 b16 = *reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(src) + sidx);
          const uint4 m16 = missing ? *reinterpret_cast<const uint4*>(missing + sidx) : make_uint4(0, 0, 0, 0);
          const uint32_t nb = bin_count[f];
          const uint32_t bw[4] = {b16.x, b16.y, b16.z, b16.w}, mw[4] = {m16.x, m16.y, m16.z, m16.w};
          uint32_t ow[4];
#pragma unroll
          for (uint32_t j = 0; j < 4; ++j) {
            uint32_t word = 0;
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
              const uint32_t b = (bw[j] >> (8 * q)) & 0xFFu;
              uint32_t v;
              if ((mw[j] >> (8 * q)) & 0xFFu) {
                if (nb > 255) bad = 1;
                v = kMissingSlot;
              } else {
                if (b >= nb) bad = 1;
                v = b;
              }
              tile[c][r + 4 * j + q] = uint8_t(v);
              word |= v << (8 * q);
            }
            ow[j] = word;
          }
          out4 = make_uint4(ow[0], ow[1], ow[2], ow[3]);
          *reinterpret_cast<uint4*>(out_fm + idx) = out4;
        } else {
#pragma unroll
          for (uint32_t q = 0; q < 16; ++q) tile[c][r + q] = 0;
        }
      }
    } else if (width == 1 && n_rows % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & 3u) == 0 &&
               (reinterpret_cast<uintptr_t>(missing) & 3u) == 0) {
      // Four rows per thread: a warp reads one feature's 128 rows as one 128-byte request
      // (the source may be page-locked host memory read over the host link).
      for (uint32_t k = threadIdx.x; k < 32 * 32; k += blockDim.x) {
        const uint32_t c = k / 32, r = (k % 32) * 4;
        const uint32_t f = fb * 32 + c, row = r0 + r;
        uint32_t word = 0;
        if (f < features && row < n_rows) {  // n_rows % 4 == 0: all four rows exist
          const size_t idx = size_t(f) * n_rows + row, sidx = size_t(f - src_f0) * n_rows + row;
          const uint32_t b4 = *reinterpret_cast<const uint32_t*>(static_cast<const uint8_t*>(src) + sidx);
          const uint32_t m4 = missing ? *reinterpret_cast<const uint32_t*>(missing + sidx) : 0u;
          const uint32_t nb = bin_count[f];
#pragma unroll
          for (uint32_t q = 0; q < 4; ++q) {
            const uint32_t b = (b4 >> (8 * q)) & 0xFFu;
            uint32_t v;
            if ((m4 >> (8 * q)) & 0xFFu) {
              if (nb > 255) bad = 1;
              v = kMissingSlot;
            } else {
              if (b >= nb) bad = 1;
              v = b;
            }
            tile[c][r + q] = uint8_t(v);
            word |= v << (8 * q);
          }
          *reinterpret_cast<uint32_t*>(out_fm + idx) = word;
        } else {
#pragma unroll
          for (uint32_t q = 0; q < 4; ++q) tile[c][r + q] = 0;
        }
      }
    } else {
      for (uint32_t k = threadIdx.x; k < 32 * 128; k += blockDim.x) {
        const uint32_t c = k / 128, r = k % 128;
        const uint32_t f = fb * 32 + c, row = r0 + r;
        uint8_t v = 0;
        if (f < features && row < n_rows) {
          const size_t sidx = size_t(f - src_f0) * n_rows + row;
          const uint32_t b = width == 1 ? static_cast<const uint8_t*>(src)[sidx]
                                        : static_cast<const uint16_t*>(src)[sidx];
          const bool miss = missing != nullptr && missing[sidx] != 0;
          if (miss) {
            if (bin_count[f] > 255) bad = 1;
            v = uint8_t(kMissingSlot);
          } else {
            if (b >= bin_count[f]) bad = 1;
            v = uint8_t(b);
          }
        }
        tile[c][r] = v;
        if (f < features && row < n_rows) out_fm[size_t(f) * n_rows + row] = v;
      }
    }
    __syncthreads();
    // store 128 rows x 32 bytes: row-major rows padded to nfb * 32 bytes
    for (uint32_t k = threadIdx.x; k < 32 * 128; k += blockDim.x) {
      const uint32_t r = k / 32, c = k % 32;
      const uint32_t row = r0 + r;
      if (row < n_rows) {
        out[size_t(row) * nfb * kBlockFeatures + fb * kBlockFeatures + c] = tile[c][r];
        out_blocked[(size_t(fb) * n_rows + row) * kBlockFeatures + c] = tile[c][r];
      }
    }
    __syncthreads();
  }
  if (bad) atomicOr(error, 1u);
}

// Wide datasets: one feature block fb (features 32 fb .. 32 fb + 31, staged from src, u8 or
// u16, with the optional missing mask) -> the u16 column blocks [nfb][n_rows][32] (histogram
// gathers: a row's block is 64 contiguous bytes) and the feature-major u16 copy (row
// routing), missing rows at slots - 1. Out-of-range bins set bit 0 of `error`.
__global__ void pack_bins16_kernel(const void* src, uint32_t width, const uint8_t* missing,
                                   const uint32_t* bin_count, uint32_t n_rows, uint32_t features,
                                   uint32_t fb, uint32_t slots, uint16_t* out_blocked,
                                   uint16_t* out_fm, uint32_t* error) {
  __shared__ uint16_t tile[32][130];
  uint32_t bad = 0;
  for (uint32_t r0 = blockIdx.x * 128; r0 < n_rows; r0 += gridDim.x * 128) {
    // 32 features x 128 rows, read along rows.
    for (uint32_t k = threadIdx.x; k < 32 * 128; k += blockDim.x) {
      const uint32_t c = k / 128, r = k % 128;
      const uint32_t f = fb * 32 + c, row = r0 + r;
      uint32_t v = 0;
      if (f < features && row < n_rows) {
        const size_t sidx = size_t(c) * n_rows + row;
        const uint32_t b = width == 1 ? static_cast<const uint8_t*>(src)[sidx]
                                      : static_cast<const uint16_t*>(src)[sidx];
        if (missing != nullptr && missing[sidx] != 0) {
          if (bin_count[f] > slots - 1) bad = 1;
          v = slots - 1;
        } else {
          if (b >= bin_count[f]) bad = 1;
          v = b;
        }
        out_fm[size_t(f) * n_rows + row] = uint16_t(v);
      }
      tile[c][r] = uint16_t(v);
    }
    __syncthreads();
    // 128 rows x 32 features: a warp writes one row's 64-byte block.
    for (uint32_t k = threadIdx.x; k < 32 * 128; k += blockDim.x) {
      const uint32_t r = k / 32, c = k % 32;
      const uint32_t row = r0 + r;
      if (row < n_rows) out_blocked[(size_t(fb) * n_rows + row) * 32 + c] = tile[c][r];
    }
    __syncthreads();
  }
  if (bad) atomicOr(error, 1u);
}

}  // namespace

// A launch in a round's chain: with a.early_launch its CTAs may become resident while the
// kernel before it still runs, and wait there (launch_order) for all of its writes. A level's
// four or five short kernels each spend 1-2 us on their start otherwise: 100,000 x 32, 50 trees
// 14.8 -> 14.1 ms, 2,000 x 12 softmax 5.36 -> 5.19, ten leaf-wise trees of 300,000 rows
// 14.2 -> 13.6, logistic 1,000,000 x 256 of depth 10 24.2 -> 23.5; unchanged where the kernels
// are long. Not the histogram builds: their CTAs take a whole SM's registers while they wait
// (logistic 24.2 -> 26.2 ms).
template <class... Params, class... Args>
cudaError_t launch_chained(void (*kernel)(Params...), const TrainerDev& a, dim3 grid, uint32_t block,
                           cudaStream_t s, uint32_t cluster, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.stream = s;
  cudaLaunchAttribute attr[2] = {};
  if (a.early_launch) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = cluster;
    attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  cfg.attrs = attr;
  return cudaLaunchKernelEx(&cfg, kernel, a, args...);
}

cudaError_t launch_gradients(const TrainerDev& a, bool g_only, int grid, cudaStream_t s) {
  if (a.objective == 0 && !a.n_classes)  // twice the CTAs: twice as many fit on an SM
    gradients_kernel<true><<<dim3(2 * grid, a.n_trees), 256, 0, s>>>(a, g_only);
  else
    gradients_kernel<false><<<dim3(grid, a.n_trees), 256, 0, s>>>(a, g_only);
  return cudaGetLastError();
}
cudaError_t launch_zero_build_slots(const TrainerDev& a, int grid, cudaStream_t s) {
  zero_slots_kernel<<<grid, 256, 0, s>>>(a, int(kZeroBuilt));
  return cudaGetLastError();
}
cudaError_t launch_zero_root_slots(const TrainerDev& a, bool g_only, int grid, cudaStream_t s) {
  zero_slots_kernel<<<grid, 256, 0, s>>>(a, int(g_only ? kRestoreRoots : kZeroRoots));
  return cudaGetLastError();
}
cudaError_t launch_root_stats(const TrainerDev& a, cudaStream_t s) {
  root_stats_kernel<<<1, 1024, 0, s>>>(a);
  return cudaGetLastError();
}
cudaError_t launch_root_cache(const TrainerDev& a, int grid, cudaStream_t s) {
  root_cache_kernel<<<grid, 256, 0, s>>>(a);
  return cudaGetLastError();
}
cudaError_t launch_subtract(const TrainerDev& a, int grid, cudaStream_t s) {
  subtract_kernel<<<grid, 256, 0, s>>>(a);
  return cudaGetLastError();
}
uint32_t split_scan_kernels(const TrainerDev& a) {
  return a.node_screen && a.scan_two_phase ? 2u : 1u;
}
bool scan_forms_root(const TrainerDev& a) {
  return split_scan_kernels(a) == 2 && a.mode == kModeFixed && a.slots == uint32_t(kSlots);
}
template <bool FIXED, bool WIDE>
cudaError_t launch_scan_one(const TrainerDev& a, int parity, int grid, int threads, cudaStream_t s) {
  const size_t smem = scan_smem_per_warp<FIXED>() * size_t(threads / 32);
  static std::atomic<unsigned long long> configured{0};  // one bit per device
  const cudaError_t err = opt_in_dynamic_smem(configured, split_scan_kernel<FIXED, WIDE>,
                                              scan_smem_per_warp<FIXED>() * (kScanThreadsMax / 32));
  if (err != cudaSuccess) return err;
  split_scan_kernel<FIXED, WIDE><<<grid, threads, smem, s>>>(a, parity);
  return cudaGetLastError();
}
template <bool FIXED, bool WIDE>
cudaError_t launch_scan_two(const TrainerDev& a, int parity, uint32_t max_nodes, ScanKind kind, bool last,
                            cudaStream_t s) {
  const uint64_t resident = uint64_t(a.sm_count ? a.sm_count : 152) * kScanCtasPerSm;
  const uint32_t screen = uint32_t(std::min<uint64_t>(resident, uint64_t(max_nodes) * a.features));
  auto kernel = split_screen_kernel<FIXED, WIDE, false>;
  if constexpr (FIXED && !WIDE)
    if (kind == ScanKind::kRoot && scan_forms_root(a)) kernel = split_screen_kernel<true, false, true>;
  const cudaError_t err = launch_chained(kernel, a, screen, kScanCta, s, 0, parity, last);
  if (err != cudaSuccess) return err;
  // CTAs that may share a node's features: one per kExactFeatures of them, while the level's
  // nodes leave room on the SMs.
  const uint32_t parts = uint32_t(std::max<uint64_t>(
      1, std::min<uint64_t>((a.features + kExactFeatures - 1) / kExactFeatures, a.exact_cap / max_nodes)));
  const uint32_t nodes = uint32_t(std::min<uint64_t>(resident, max_nodes));
  if (parts > 1)
    return launch_chained(split_exact_kernel<FIXED, WIDE, true>, a, dim3(nodes, parts), kScanCta, s, 0, parity,
                          kind == ScanKind::kActive, last);
  return launch_chained(split_exact_kernel<FIXED, WIDE, false>, a, nodes, kScanCta, s, 0, parity,
                        kind == ScanKind::kActive, last);
}

cudaError_t launch_split_scan(const TrainerDev& a, int parity, uint32_t max_nodes, ScanKind kind,
                              bool last, int grid, cudaStream_t s) {
  const bool fixed = a.mode == kModeFixed, wide = a.slots != uint32_t(kSlots);
  if (a.slots < uint32_t(kSlots) || a.slots % uint32_t(kSlots) || max_nodes == 0) return cudaErrorInvalidValue;
  if (split_scan_kernels(a) == 2) {
    // node_screen was cleared by the level's zero_slots_kernel.
    if (fixed) return wide ? launch_scan_two<true, true>(a, parity, max_nodes, kind, last, s)
                           : launch_scan_two<true, false>(a, parity, max_nodes, kind, last, s);
    return wide ? launch_scan_two<false, true>(a, parity, max_nodes, kind, last, s)
                : launch_scan_two<false, false>(a, parity, max_nodes, kind, last, s);
  }
  const int threads = int(a.scan_threads);
  if (threads < 32 || threads > kScanThreadsMax || threads % 32) return cudaErrorInvalidValue;
  // The readers of partial find a node's records where the scan writes them.
  if (a.partial_stride != a.n_fchunks) return cudaErrorInvalidValue;
  if (fixed) return wide ? launch_scan_one<true, true>(a, parity, grid, threads, s)
                         : launch_scan_one<true, false>(a, parity, grid, threads, s);
  return wide ? launch_scan_one<false, true>(a, parity, grid, threads, s)
              : launch_scan_one<false, false>(a, parity, grid, threads, s);
}
cudaError_t launch_leafwise_init(const TrainerDev& a, cudaStream_t s) {
  return launch_chained(leafwise_init_kernel, a, 1, 256, s, 0);
}
cudaError_t launch_leafwise_select(const TrainerDev& a, cudaStream_t s) {
  return launch_chained(leafwise_select_kernel, a, 1, 32 * std::min(a.n_trees, kSelectTrees), s, 0);
}
cudaError_t launch_leafwise_merge(const TrainerDev& a, cudaStream_t s) {
  leafwise_merge_kernel<<<1, 256, 0, s>>>(a);
  return cudaGetLastError();
}
cudaError_t launch_leafwise_finish(const TrainerDev& a, cudaStream_t s) {
  return launch_chained(leafwise_finish_kernel, a, 1, 32, s, 0);
}
cudaError_t launch_finalize(const TrainerDev& a, int parity, uint32_t depth, uint32_t max_nodes,
                            cudaStream_t s) {
  if (max_nodes <= kNodeFinalizeMax && a.partial_stride == 1)
    return launch_chained(finalize_nodes_kernel, a, 1, (max_nodes + 31) / 32 * 32, s, 0, parity, depth);
  return launch_chained(finalize_kernel, a, 1, 1024, s, 0, parity, depth);
}
// CTAs per node of the cluster launch for a level of at most max_nodes split nodes (0: the
// three launches). As many as fit the GPU at once (one of these CTAs per SM), up to the 16
// of a non-portable cluster; not where a node that held every row (half of them from four
// nodes on, a quarter in a leaf-wise step, whose nodes soon are small) would leave a thread
// more than 16: at 1,000,000 rows the cluster launch takes 31-42 us a level, the three
// launches 19; at 100,000 10 and 15; ten leaf-wise trees of 300,000 rows 15.1 and 15.9 ms.
static uint32_t partition_cluster_ctas(const TrainerDev& a, uint32_t max_nodes) {
  const uint32_t sms = a.sm_count ? a.sm_count : 152;
  uint32_t ctas = 16;
  while (ctas > 1 && uint64_t(max_nodes) * ctas > sms) ctas >>= 1;
  if (max_nodes > 2 * sms) return 0;  // each cluster would take several nodes in turn
  if (uint64_t(a.seg_stride) > uint64_t(ctas) * kClusterPartRows) return 0;  // the largest node possible
  const uint32_t largest =
      a.lw_active ? a.seg_stride / 4 : (max_nodes / a.n_trees >= 4 ? a.seg_stride / 2 : a.seg_stride);
  return largest <= 16u * ctas * kClusterThreads ? ctas : 0;
}

uint32_t partition_kernels(const TrainerDev& a, uint32_t max_nodes) {
  return partition_cluster_ctas(a, max_nodes) ? 1u : 3u;
}

cudaError_t launch_partition(const TrainerDev& a, uint32_t max_nodes, int grid, cudaStream_t s) {
  if (const uint32_t ctas = partition_cluster_ctas(a, max_nodes)) {
    static std::atomic<unsigned long long> configured{0};  // one bit per device
    cudaError_t err = allow_large_clusters(configured, partition_cluster_kernel);
    if (err != cudaSuccess) return err;
    const uint32_t sms = a.sm_count ? a.sm_count : 152;
    const uint32_t clusters = std::min(max_nodes, std::max(1u, sms / ctas));
    return launch_chained(partition_cluster_kernel, a, clusters * ctas, kClusterThreads, s, ctas);
  }
  cudaError_t err = launch_chained(partition_count_kernel, a, uint32_t(grid), kPartThreads, s, 0);
  if (err == cudaSuccess) err = launch_chained(partition_scan_kernel, a, uint32_t(grid), 1024, s, 0);
  if (err == cudaSuccess) err = launch_chained(partition_scatter_kernel, a, uint32_t(grid), kPartThreads, s, 0);
  return err;
}
cudaError_t launch_partition_count(const TrainerDev& a, int grid, cudaStream_t s) {
  partition_count_kernel<<<grid, kPartThreads, 0, s>>>(a);
  return cudaGetLastError();
}
cudaError_t launch_partition_finish(const TrainerDev& a, int grid, cudaStream_t s) {
  partition_scan_kernel<<<grid, 1024, 0, s>>>(a);
  partition_scatter_kernel<<<grid, kPartThreads, 0, s>>>(a);
  return cudaGetLastError();
}
__global__ void fill_f64_kernel(double* dst, uint64_t n, double value) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x)
    dst[i] = value;
}
cudaError_t launch_fill_f64(double* dst, uint64_t n, double value, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const uint64_t blocks = std::min<uint64_t>((n + 255) / 256, 4096);
  fill_f64_kernel<<<unsigned(blocks), 256, 0, s>>>(dst, n, value);
  return cudaGetLastError();
}
cudaError_t launch_apply_leaves(const TrainerDev& a, int grid, cudaStream_t s) {
  const cudaError_t err = launch_chained(apply_leaves_kernel, a, uint32_t(grid), 256, s, 0);
  return err == cudaSuccess ? launch_chained(apply_steps_kernel, a, uint32_t(grid), 256, s, 0) : err;
}
cudaError_t launch_expand_samples(const uint8_t* counts, uint32_t n, uint32_t trees, uint32_t* chunk_sum,
                                  uint32_t cap, uint32_t* sample, cudaStream_t s) {
  const uint32_t chunks = (n + kExpandChunk - 1) / kExpandChunk;
  for (uint32_t t0 = 0; t0 < trees; t0 += 65535) {  // the grid's y limit
    const uint32_t nt = std::min(65535u, trees - t0);
    const uint8_t* c = counts + size_t(t0) * n;
    uint32_t* sums = chunk_sum + size_t(t0) * chunks;
    expand_sum_kernel<<<dim3(chunks, nt), kExpandThreads, 0, s>>>(c, n, sums);
    expand_scan_kernel<<<nt, 1024, 0, s>>>(sums, chunks);
    expand_write_kernel<<<dim3(chunks, nt), kExpandThreads, 0, s>>>(c, n, sums, cap, sample + size_t(t0) * cap);
  }
  return cudaGetLastError();
}
cudaError_t launch_pack_tree_bins(const uint8_t* bins_fm, uint32_t n, const uint32_t* feature_of,
                                  uint32_t features, uint32_t nfb, uint32_t trees, uint8_t* out, cudaStream_t s) {
  if (nfb > 65535) return cudaErrorInvalidValue;
  for (uint32_t t0 = 0; t0 < trees; t0 += 65535) {
    const uint32_t nt = std::min(65535u, trees - t0);
    pack_tree_bins_kernel<<<dim3((n + 511) / 512, nfb, nt), 128, 0, s>>>(
        bins_fm, n, feature_of + size_t(t0) * features, features, nfb, out + size_t(t0) * n * nfb * 32);
  }
  return cudaGetLastError();
}
cudaError_t launch_label_counts(const double* labels, uint64_t n, uint32_t classes, unsigned long long* counts,
                                cudaStream_t s) {
  if (n == 0 || classes > kLabelCountMax) return cudaErrorInvalidValue;
  const unsigned grid = unsigned(std::min<uint64_t>((n + 1023) / 1024, 152ull * 8));
  label_counts_kernel<<<grid, 256, (classes + 1) * sizeof(uint32_t), s>>>(labels, n, classes, counts);
  return cudaGetLastError();
}
cudaError_t launch_squared_error(const double* labels, const double* preds, uint64_t n,
                                 double* out, uint32_t* error, cudaStream_t s) {
  const int grid = int(std::min<uint64_t>((n + 255) / 256, 152ull * 16));
  squared_error_kernel<<<grid > 0 ? grid : 1, 256, 0, s>>>(labels, preds, n, out, error);
  return cudaGetLastError();
}
cudaError_t launch_pack_bins(const void* src, uint32_t width, const uint8_t* missing,
                             const uint32_t* bin_count, uint32_t n_rows, uint32_t features,
                             uint32_t nfb, uint8_t* out_rows, uint8_t* out_blocked,
                             uint8_t* out_fm, uint32_t* error, cudaStream_t s) {
  const uint32_t gx = std::min<uint32_t>((n_rows + 127) / 128, 4096u);
  pack_bins_kernel<<<dim3(gx > 0 ? gx : 1, nfb), 256, 0, s>>>(src, width, missing, bin_count,
                                                              n_rows, features, nfb, out_rows,
                                                              out_blocked, out_fm, error, 0u, 0u);
  return cudaGetLastError();
}
cudaError_t launch_pack_bins_block(const void* src_block, uint32_t width, const uint8_t* missing_block,
                                   const uint32_t* bin_count, uint32_t n_rows, uint32_t features,
                                   uint32_t nfb, uint32_t fb, uint8_t* out_rows, uint8_t* out_blocked,
                                   uint8_t* out_fm, uint32_t* error, cudaStream_t s) {
  const uint32_t gx = std::min<uint32_t>((n_rows + 127) / 128, 4096u);
  pack_bins_kernel<<<dim3(gx > 0 ? gx : 1, 1), 256, 0, s>>>(src_block, width, missing_block, bin_count,
                                                            n_rows, features, nfb, out_rows, out_blocked,
                                                            out_fm, error, fb, fb * kBlockFeatures);
  return cudaGetLastError();
}
cudaError_t launch_pack_bins16_block(const void* src_block, uint32_t width,
                                     const uint8_t* missing_block, const uint32_t* bin_count,
                                     uint32_t n_rows, uint32_t features, uint32_t fb,
                                     uint32_t slots, uint16_t* out_blocked, uint16_t* out_fm,
                                     uint32_t* error, cudaStream_t s) {
  if (slots < 2 || slots > 65536) return cudaErrorInvalidValue;
  const uint32_t gx = std::min<uint32_t>((n_rows + 127) / 128, 4096u);
  pack_bins16_kernel<<<gx > 0 ? gx : 1, 256, 0, s>>>(src_block, width, missing_block, bin_count, n_rows,
                                                     features, fb, slots, out_blocked, out_fm, error);
  return cudaGetLastError();
}
template <typename BinT>
static cudaError_t launch_predict_tile(const BinT* bins_fm, uint32_t missing_slot, uint32_t n_rows,
                                       uint32_t features, const PackedForest& f, double base, double* out,
                                       cudaStream_t s) {
  const uint32_t rows = predict_rows(n_rows, features, sizeof(BinT));
  if (rows == 0) return cudaErrorInvalidValue;
  static std::atomic<unsigned long long> configured{0};  // one bit per device
  const cudaError_t err = opt_in_dynamic_smem(configured, predict_packed_kernel<BinT>, kPredictSmemMax);
  if (err != cudaSuccess) return err;
  const size_t smem = kPredictTreeBytes + size_t(features) * predict_pitch<BinT>(rows) * sizeof(BinT);
  predict_packed_kernel<BinT><<<(n_rows + rows - 1) / rows, rows, smem, s>>>(bins_fm, missing_slot, n_rows, features,
                                                                            f, base, out);
  return cudaGetLastError();
}
cudaError_t launch_predict_packed(const uint8_t* bins_fm, const uint16_t* bins16_fm, uint32_t slots,
                                  uint32_t n_rows, uint32_t features, const PackedForest& f, double base,
                                  double* out, cudaStream_t s) {
  if (bins16_fm) return launch_predict_tile<uint16_t>(bins16_fm, slots - 1, n_rows, features, f, base, out, s);
  return launch_predict_tile<uint8_t>(bins_fm, uint32_t(kMissingSlot), n_rows, features, f, base, out, s);
}
cudaError_t launch_predict(const uint8_t* bins_fm, const uint16_t* bins16_fm, uint32_t slots,
                           uint32_t n_rows, uint32_t nfb, const uint8_t* has_missing,
                           const TreeNodeOut* nodes, const uint32_t* tree_offsets,
                           uint32_t n_trees, double base, double lr, double* out,
                           uint32_t* error, cudaStream_t s) {
  (void)nfb;
  const int grid = int(std::min<uint64_t>((n_rows + 255) / 256, 152ull * 16));
  if (bins16_fm) {
    if (slots < 2 || slots > 65536) return cudaErrorInvalidValue;
    predict_kernel<uint16_t><<<grid > 0 ? grid : 1, 256, 0, s>>>(
        bins16_fm, slots - 1, n_rows, has_missing, nodes, tree_offsets, n_trees, base, lr, out, error);
  } else {
    predict_kernel<uint8_t><<<grid > 0 ? grid : 1, 256, 0, s>>>(
        bins_fm, uint32_t(kMissingSlot), n_rows, has_missing, nodes, tree_offsets, n_trees, base,
        lr, out, error);
  }
  return cudaGetLastError();
}

}  // namespace mpsb
