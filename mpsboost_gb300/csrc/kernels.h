// Launch interface of the sm_103a kernels (host and device code include this).
#pragma once

#include <atomic>
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

#include "device.cuh"

namespace mpsb {

// Histogram work items per SM where the trainer sets none.
__host__ __device__ constexpr uint32_t default_items_per_sm(uint32_t slots) {
  return slots == uint32_t(kSlots) ? 3u : 1u;
}

constexpr uint32_t kScanCtasPerSm = 6;  // resident CTAs of the two-launch split scan
constexpr uint32_t kExactFeatures = 32;  // more features than this: a node's CTAs may share them

constexpr uint32_t kWideVotePasses = 4;  // passes of a wide block of 32 features, at most

// Device pointers and sizes of one training session, passed by value to every kernel.
struct TrainerDev {
  // dataset
  const uint8_t* bins;          // u8 bins for histograms: row r, feature f at
                                //   r * bins_row_stride + (f/32) * bins_block_stride + f%32
  uint64_t bins_row_stride, bins_block_stride;
  uint64_t bins_tree_stride;    // bytes between the trees' bins (0: all trees read the same)
  const uint8_t* bins_fm;       // [features][n_rows] feature-major u8 bins (routing rows)
  const uint32_t* bin_count;    // [features]
  const uint8_t* has_missing;   // [features]
  // Histogram slots per feature: 256 (u8 bins, missing rows at slot 255), or for wide
  // datasets (a feature with more than 256 bins, or 256 bins and missing values) a larger
  // multiple of 256 with missing rows at slot slots - 1; wide datasets keep u16 copies of
  // the bins in place of the u8 ones.
  uint32_t slots = kSlots;
  const uint16_t* bins16;       // wide: [nfb][n_rows][32] column blocks (else null)
  const uint16_t* bins16_fm;    // wide: [features][n_rows] (else null)
  uint32_t n_rows, features, nfb, n_trees;
  // per-tree arrays
  const double* labels;         // [n_rows]
  const double* weights;        // [n_rows], [n_trees][n_rows] or null (unit weights)
  uint32_t weights_per_tree;
  uint32_t objective;
  double* preds;                // [n_trees][n_rows]; null: every row's is tree_base[tree]
  const double* tree_base;      // [n_trees] (single-round forest trees)
  float2* gh;                   // gh_ordered: [n_trees][2][seg_stride] in row-segment order
                                // (moved along by the partition); else [n_trees][n_rows]
  uint32_t gh_ordered;
  uint32_t* rows;               // [n_trees][2][seg_stride] row ids of the level's segments
  uint32_t seg_stride;          // positions per (tree, parity) of rows / gh: n_rows, or the
                                // largest sample of a forest (a row appears once per draw)
  // Forest samples (null for boosting): per tree the multiset of rows it trains on,
  // [n_trees][seg_stride] in ascending row order, and its size; the feature rank of each
  // feature in the tree's subset (random thresholds hash the rank) and per-tree seeds.
  const uint32_t* sample_rows;
  const uint32_t* sample_count;   // [n_trees]
  const uint32_t* feature_rank;   // [n_trees][features] or null (rank = feature)
  // Compact forests: a tree's features are numbered within its own ascending subset
  // (`features` is the largest subset; bins, histograms, masks and splits count that way)
  // and feature_of [n_trees][features] names the dataset's. Null: the dataset's numbers.
  const uint32_t* feature_of;
  const uint32_t* tree_seeds;     // [n_trees] or null (params.random_seed)
  uint32_t skip_apply;            // 1: no prediction update (forest trees are single-round)
  uint32_t unit_hess;             // every row's hessian is 1 (no weights; squared error or
                                  // quantile): fixed-point builds take kModeFixedCG
  TreeState* trees;             // [n_trees]
  TreeParams params;
  const int8_t* monotonic;      // [features] or null
  const uint32_t* group_masks;  // [n_groups][path_words]
  const uint32_t* tree_feature_masks;  // [n_trees][path_words] or null
  // histogram slots: [n_slots][features][slots] x {count, g, h} 64-bit words
  unsigned long long* hist;
  uint32_t* free_stack;         // [n_slots]
  uint32_t n_slots;
  // level buffers (index = level parity)
  NodeRec* nodes[2];            // [max_level_nodes]
  uint32_t* node_path[2];       // [max_level_nodes][path_words]
  uint32_t* node_allowed[2];    // [max_level_nodes][path_words]
  uint32_t max_level_nodes;
  SplitRec* partial;            // [max_level_nodes][partial_stride]
  uint32_t partial_stride;      // records per node: 1 (two-launch scan) or n_fchunks
  // Two-launch split scan (scan_two_phase: the FP32 screen applies): [max_level_nodes]
  // maximum FP32 screen score of each node's certainly admissible candidates (float
  // bits; zeroed by each level's zero_slots_kernel, which every scan of the trainer
  // follows) and [max_level_nodes][features] each feature's maximum and exact flag. Null
  // node_screen: one launch, each feature screened on its own (the per-feature entry point
  // needs every feature's best split).
  uint32_t* node_screen;
  uint32_t* feature_screen;
  uint32_t scan_two_phase;
  // Nodes whose exact evaluation several CTAs share: each CTA's best split, [node][CTA] within
  // exact_cap records (0: a CTA per node), and how many of a node's CTAs are done (zero between
  // launches).
  SplitRec* exact_part;
  uint32_t* exact_done;
  uint32_t exact_cap;
  uint32_t n_fchunks;           // feature chunks of the one-launch split scan (a warp each feature)
  BuildEntry* build;            // [max_level_nodes]
  uint32_t* build_prefix;       // [max_level_nodes + 1] chunk prefix
  SubEntry* sub;                // [max_level_nodes]
  PartEntry* part;              // [max_level_nodes]
  uint32_t* part_prefix;        // [max_level_nodes + 1] chunk prefix
  uint32_t* part_counts;        // [max_part_chunks] left rows per chunk
  uint32_t* part_offsets;       // [max_part_chunks] left rows before the chunk in its node
  uint32_t* part_flags;         // [max_part_chunks][kPartChunk / 32]
  uint32_t max_part_chunks;
  LeafSeg* leafseg;             // [max_leafsegs]
  uint32_t* leaf_of;            // [n_trees][n_rows]: 2 x leaf segment + side, per row of the
                                // round (kNoLeaf between rounds)
  double* leaf_steps;           // [2 * max_leafsegs]: lr x leaf value per (segment, side)
  uint32_t* leaf_prefix;        // [max_leafsegs + 1]
  uint32_t apply_chunk;         // rows per leaf-application chunk
  uint32_t max_leafsegs;
  TreeNodeOut* tree_nodes;      // [n_trees][max_tree_nodes]
  uint32_t max_tree_nodes;
  Control* ctl;
  uint32_t* limb_votes;         // [nfb][2], wide [nfb][kWideVotePasses][2], of the launch's depth
                                // level: work items (a wide block's passes) that passed and
                                // failed the packed-limb check (null: split limbs only)
  uint32_t item_rows_max;       // the adaptive item size's upper end (0: kItemRowsMax)
  uint32_t early_launch;        // a round's kernels wait for one another on the device (launch_chained)
  uint32_t store_single;        // below the roots: a node of one row chunk is stored by its work
                                // items, so its slot is not cleared (register-direct kernel)
  uint32_t item_rows;           // rows per histogram work item (<= kItemRowsMax); 0: the
                                // level's adaptive value ctl->item_rows
  uint32_t sm_count;
  uint32_t items_per_sm;        // histogram work items per SM of the adaptive item size (0:
                                // default_items_per_sm)
  uint32_t mode;                // kModeFixed / kModeFloat
  uint32_t ovr;                 // labels are class ids; tree t fits class t (logistic)
  uint32_t n_classes;           // native softmax: K classes, one tree per class in turn;
                                // preds holds the margins [K][n_rows] and the round
                                // counter modulo K is the class of the current tree
  uint32_t scan_threads;        // block size of the one-launch split scan (multiple of 32)
  uint32_t fused_sub;           // level-wise siblings are subtracted by the split scan
                                // (NodeRec::sub_from), not by subtract_kernel
  // finalize scratch
  uint32_t* scratch_flags;      // [max_level_nodes]
  uint32_t* scratch_prefix;     // [max_level_nodes] valid-prefix, then accepted-prefix
  uint32_t* scratch_aux;        // [max_level_nodes] free-slot prefix
  uint32_t* tree_scratch;       // [n_trees][4]
  // model output: per round, per tree, max_tree_nodes nodes + node counts
  TreeNodeOut* model_nodes;     // [max_rounds][n_trees][max_tree_nodes]
  uint32_t* model_counts;       // [max_rounds][n_trees]
  uint32_t* round_counter;      // rounds completed (device)
  uint32_t max_rounds;
  // Histogram item range of one launch: [item_begin, item_end); item_end 0 = the whole
  // level (ctl->hist_items). Per-node launches of the plain path set a node's range.
  uint32_t item_begin, item_end;
  // Leaf-wise growth (growth_strategy 1; null for level-wise): per tree the active leaves
  // with their interaction path and allowed-feature words, the active count, a done flag,
  // and a private stack of histogram slots; the scanned children of a step map to
  // (tree << 16 | active index).
  LeafActive* lw_active;        // [n_trees][lw_cap]
  uint32_t* lw_path;            // [n_trees][lw_cap][path_words]
  uint32_t* lw_allowed;         // [n_trees][lw_cap][path_words]
  uint32_t* lw_count;           // [n_trees]
  uint32_t* lw_done;            // [n_trees]
  uint32_t* lw_slots;           // [n_trees][lw_slot_cap] free slots
  uint32_t* lw_slot_top;        // [n_trees]
  uint32_t* lw_scan_map;        // [2 * n_trees]
  uint32_t lw_cap, lw_slot_cap, lw_max_active, lw_max_leaves;
  // Root count/hessian histograms of the fit's first round: [n_trees][features][slots]
  // {count, qh} and the hessian scale they were built with (null: not reused).
  unsigned long long* root_cache;
  int* root_cache_kh;
};

struct HistConfig {
  int threads = 768;        // fixed and float builds
  int stages = 2;
  int root_threads = 1024;  // gradient-only root builds (64 KB histogram)
  // Register-direct fixed-point builds (hist_build_direct_kernel: each lane loads a whole
  // row's 32-byte feature block, no shared-memory staging; flush by TMA bulk reductions);
  // threads 512 or 768. The opt-in TMA staging (bins_tmap) takes precedence. The trainer
  // turns it on; the node-level entries keep the staged kernel.
  bool direct = false;
  // Wide datasets (more than 256 slots per feature): threads of hist_build_wide_kernel,
  // 1024 (32 warps hide the gathers' latency: 1.3x faster than 512 at 512 and 1024 bins
  // on 4M x 128) or 512.
  int wide_threads = 1024;
  // Tensor map of the row-major bins ({row stride, n_rows} u8, box 32 x 1): row-major
  // fixed-point builds stage gathered rows with TMA gather4 copies (opt-in). Null: cp.async.
  const CUtensorMap* bins_tmap = nullptr;
};

// Encodes the tensor map of a row-major bins matrix (rows x row_stride bytes). Returns
// false where the CUDA driver offers no tensor maps.
bool encode_bins_tmap(CUtensorMap* map, const uint8_t* bins, uint64_t row_stride, uint32_t n_rows);

cudaError_t launch_hist_build(const TrainerDev& a, const HistConfig& cfg, int grid,
                              cudaStream_t stream);
cudaError_t launch_fill_f64(double* dst, uint64_t n, double value, cudaStream_t stream);
// Gradients, then the round's setup. g_only: the roots' count and hessian histograms come
// from the fit's first round.
cudaError_t launch_gradients(const TrainerDev& a, bool g_only, int grid, cudaStream_t stream);
cudaError_t launch_zero_build_slots(const TrainerDev& a, int grid, cudaStream_t stream);
// The roots' slots: cleared, or (g_only) started from the kept count and hessian words.
cudaError_t launch_zero_root_slots(const TrainerDev& a, bool g_only, int grid, cudaStream_t stream);
cudaError_t launch_root_stats(const TrainerDev& a, cudaStream_t stream);
// Leaf-wise growth: after the root's split scan (init), per step (select before the
// partition / histogram / subtraction / split scan of the chosen leaves' children, merge
// after), and the leaf segments at the end (finish).
cudaError_t launch_leafwise_init(const TrainerDev& a, cudaStream_t stream);
cudaError_t launch_leafwise_select(const TrainerDev& a, cudaStream_t stream);
cudaError_t launch_leafwise_merge(const TrainerDev& a, cudaStream_t stream);
cudaError_t launch_leafwise_finish(const TrainerDev& a, cudaStream_t stream);
// Copies the roots' count and hessian words into root_cache.
cudaError_t launch_root_cache(const TrainerDev& a, int grid, cudaStream_t stream);
cudaError_t launch_subtract(const TrainerDev& a, int grid, cudaStream_t stream);
// max_nodes: a bound on the nodes the launch scans (ctl->n_nodes), from the level.
// kRoot: level 0, whose statistics the scan forms where scan_forms_root (else
// launch_root_stats has). kActive: a leaf-wise step; a two-launch scan writes its nodes'
// splits to their active leaves (after a one-launch scan launch_leafwise_merge does).
// last: the children of the scanned nodes are leaves.
enum class ScanKind { kRoot, kLevel, kActive };
bool scan_forms_root(const TrainerDev& a);
cudaError_t launch_split_scan(const TrainerDev& a, int parity, uint32_t max_nodes, ScanKind kind,
                              bool last, int grid, cudaStream_t stream);
uint32_t split_scan_kernels(const TrainerDev& a);  // launches per launch_split_scan
// max_nodes: a bound on the level's nodes (ctl->n_nodes).
cudaError_t launch_finalize(const TrainerDev& a, int parity, uint32_t depth, uint32_t max_nodes,
                            cudaStream_t stream);
// max_nodes: a bound on the nodes the launch partitions (ctl->n_part).
cudaError_t launch_partition(const TrainerDev& a, uint32_t max_nodes, int grid, cudaStream_t stream);
uint32_t partition_kernels(const TrainerDev& a, uint32_t max_nodes);  // launches per launch_partition
cudaError_t launch_partition_count(const TrainerDev& a, int grid, cudaStream_t stream);
cudaError_t launch_partition_finish(const TrainerDev& a, int grid, cudaStream_t stream);
cudaError_t launch_apply_leaves(const TrainerDev& a, int grid, cudaStream_t stream);
// Row samples of forest trees from their row multiplicities (counts [trees][n]) into sample
// [trees][cap]; chunk_sum: scratch, [trees][ceil(n / kExpandChunk)].
constexpr uint32_t kExpandChunk = 4096;
cudaError_t launch_expand_samples(const uint8_t* counts, uint32_t n, uint32_t trees, uint32_t* chunk_sum,
                                  uint32_t cap, uint32_t* sample, cudaStream_t stream);
// Each tree's own features as rows [trees][n][nfb * 32] (feature_of: TrainerDev).
cudaError_t launch_pack_tree_bins(const uint8_t* bins_fm, uint32_t n, const uint32_t* feature_of,
                                  uint32_t features, uint32_t nfb, uint32_t trees, uint8_t* out,
                                  cudaStream_t stream);
// counts [classes + 1], zeroed by the caller: rows per class id, then rows of no class.
constexpr uint32_t kLabelCountMax = 8192;  // classes (32 KB of shared counters)
cudaError_t launch_label_counts(const double* labels, uint64_t n, uint32_t classes, unsigned long long* counts,
                                cudaStream_t stream);
cudaError_t launch_squared_error(const double* labels, const double* preds, uint64_t n,
                                 double* out_pairs, uint32_t* error, cudaStream_t stream);
// Bins from the u8 feature-major copy (missing rows at 255), or with bins16_fm set from
// the u16 one (missing rows at slots - 1).
cudaError_t launch_predict(const uint8_t* bins_fm, const uint16_t* bins16_fm, uint32_t slots,
                           uint32_t n_rows, uint32_t nfb, const uint8_t* has_missing,
                           const TreeNodeOut* nodes, const uint32_t* tree_offsets,
                           uint32_t n_trees, double base, double learning_rate, double* out,
                           uint32_t* error, cudaStream_t stream);
// Trees in the packed node format: 8 bytes per inner node, {feature << 17 | missing goes left
// << 16 | threshold, left | right << 16}, a child reference being a node number in its tree
// or kPackedLeaf | leaf number (16 bits: at most 32,768 of either, features below 32,768);
// leaf steps lr x value; trees[t] = {first node, first leaf, root reference, 0} with one
// more entry after the last; groups of trees whose nodes and leaves fit the staging.
struct PackedForest {
  const uint2* nodes;
  const double* steps;
  const uint4* trees;
  const uint32_t* group_first;  // [n_groups + 1]
  uint32_t n_groups;
};
constexpr uint32_t kPackedLeaf = 0x8000u;
constexpr uint32_t kPredictNodes = 4096, kPredictLeaves = 4096;  // staged at a time: 64 KB
constexpr size_t kPredictTreeBytes = size_t(kPredictNodes) * 8 + size_t(kPredictLeaves) * 8;
constexpr size_t kPredictSmemMax = 227 * 1024;
// Elements between two features' staged rows: a word more than the rows, so that lanes at
// different features of neighbouring rows spread over the banks.
template <typename BinT>
constexpr __host__ __device__ uint32_t predict_pitch(uint32_t rows) { return rows + uint32_t(4 / sizeof(BinT)); }
// Rows (threads) per CTA: as many as the staging takes, fewer where that leaves SMs idle
// (128 at least; 0: the features' bins do not fit).
inline uint32_t predict_rows(uint32_t n_rows, uint32_t features, size_t bin_bytes) {
  uint32_t rows = 1024;
  while (rows > 128 && (uint64_t(n_rows) < uint64_t(rows) * 152 ||
                        kPredictTreeBytes + uint64_t(features) * (rows * bin_bytes + 4) > kPredictSmemMax))
    rows >>= 1;
  return kPredictTreeBytes + uint64_t(features) * (rows * bin_bytes + 4) <= kPredictSmemMax ? rows : 0u;
}
// Whether the packed kernel is the faster one. `entries`: inner nodes and leaves of all trees;
// `visits`: nodes a row passes in all of them, were they balanced. Three things it spends that
// the general kernel does not, each against what it saves, the visits' gathers (whole calls on
// resident datasets of 255 bins, complete trees on random features, general -> packed, ms):
//  * a CTA stages every tree: 16 of depth 10 on 30,000 rows (128 rows a CTA: 1.6 entries per row
//    and visit) 0.43 -> 0.50, 64 of depth 8 (0.5) 0.91 -> 0.79, 8 of depth 11 on 1,000,000 x 64
//    (1,024 rows: 0.36) 0.71 -> 0.56;
//  * it stages every feature of its rows, used or not: 1,000,000 x 128, 4 trees of depth 6 (five
//    bytes a visit) 0.18 -> 0.24, 16 (1.3) 0.48 -> 0.40; 30,000 x 512, 16 (5.3) 0.21 and 0.21.
//    Up to 32 KB a CTA do not show: 1,000 x 256, one tree, 0.05 -> 0.04;
//  * the features' bins cut the rows that an SM walks at once: 300,000 x 1,000 (an eighth) 0.05
//    -> 1.88 with one tree, 3.5 -> 7.0 with 256; 300,000 x 512 (a quarter) 3.2 -> 3.8; 1,000,000
//    x 256 (half) 0.10 -> 0.50 with one tree, 1.74 -> 1.55 with 64 of depth 6.
inline bool predict_packed_pays(uint32_t n_rows, uint32_t features, size_t bin_bytes, uint64_t entries,
                                uint64_t visits) {
  const uint64_t rows = predict_rows(n_rows, features, bin_bytes), free_rows = predict_rows(n_rows, 0, bin_bytes);
  const uint64_t row_bytes = features * bin_bytes;
  if (rows == 0 || 5 * entries > 3 * rows * visits + 5120) return false;
  if (rows == free_rows) return row_bytes * rows <= 32768 || row_bytes <= 4 * visits;
  return 2 * rows == free_rows && 3 * row_bytes <= 2 * visits;
}
cudaError_t launch_predict_packed(const uint8_t* bins_fm, const uint16_t* bins16_fm, uint32_t slots,
                                  uint32_t n_rows, uint32_t features, const PackedForest& f, double base,
                                  double* out, cudaStream_t stream);
// Wide datasets: one feature block fb of the u16 copies ([nfb][n_rows][32] column blocks
// and [features][n_rows]) from a staged copy of its source features, missing rows at
// slots - 1.
cudaError_t launch_pack_bins16_block(const void* src_block, uint32_t width,
                                     const uint8_t* missing_block, const uint32_t* bin_count,
                                     uint32_t n_rows, uint32_t features, uint32_t fb,
                                     uint32_t slots, uint16_t* out_blocked, uint16_t* out_fm,
                                     uint32_t* error, cudaStream_t stream);
// One feature block fb of the dataset from a staged copy of its source features
// (src_block / missing_block start at feature 32 * fb).
cudaError_t launch_pack_bins_block(const void* src_block, uint32_t width, const uint8_t* missing_block,
                                   const uint32_t* bin_count, uint32_t n_rows, uint32_t features,
                                   uint32_t nfb, uint32_t fb, uint8_t* out_rows, uint8_t* out_blocked,
                                   uint8_t* out_fm, uint32_t* error, cudaStream_t stream);
cudaError_t launch_pack_bins(const void* src, uint32_t width, const uint8_t* missing,
                             const uint32_t* bin_count, uint32_t n_rows, uint32_t features,
                             uint32_t nfb, uint8_t* out_rows, uint8_t* out_blocked,
                             uint8_t* out_fm, uint32_t* error, cudaStream_t stream);
// Raises `kernel`'s dynamic shared memory limit to `bytes` on the current device before
// its first launch there. The limit is an attribute of the function in that device's
// context, so it is set once per device: bit d of `devices` records device d (devices
// past 63 set it before every launch). Two host threads that race past the check both set
// the same value, which is harmless.
template <typename Kernel>
inline cudaError_t opt_in_dynamic_smem(std::atomic<unsigned long long>& devices, Kernel kernel,
                                       size_t bytes) {
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return err;
  const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0ull;
  if (bit && (devices.load(std::memory_order_acquire) & bit)) return cudaSuccess;
  err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
  if (err == cudaSuccess && bit) devices.fetch_or(bit, std::memory_order_acq_rel);
  return err;
}

// Allows `kernel` clusters of more than the portable 8 CTAs, once per device as above.
template <typename Kernel>
inline cudaError_t allow_large_clusters(std::atomic<unsigned long long>& devices, Kernel kernel) {
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return err;
  const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0ull;
  if (bit && (devices.load(std::memory_order_acquire) & bit)) return cudaSuccess;
  err = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (err == cudaSuccess && bit) devices.fetch_or(bit, std::memory_order_acq_rel);
  return err;
}

}  // namespace mpsb
