// Host side of the CUDA backend: the C ABI of include/mpsb_cuda.h, the device-resident
// dataset, the node-level entries of the reference backend contract
// (include/mpsboost/backend.hpp:52-135) and the device-resident training session.
//
// One backend owns one CUDA stream. A training session keeps every input on the device
// and runs each boosting round as a fixed sequence of kernels (gradients, then per depth
// level: zero slots, histogram build, root stats or sibling subtraction, split scan,
// finalize, partition; then leaf application), captured once as a CUDA graph and
// replayed per round. No row ever returns to the host inside a round; the host reads
// back only the finished trees.
#include <cuda_runtime.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <limits>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "host_types.h"

using namespace mpsb;

namespace mpsb {

thread_local std::string g_error;

// MPSB_TRACE=1: host-side phase times of session setup and export on stderr.
struct PhaseTrace {
  bool on = false;
  std::chrono::steady_clock::time_point t0, last;
  const char* what;
  explicit PhaseTrace(const char* w) : what(w) {
    const char* v = std::getenv("MPSB_TRACE");
    on = v && std::atoi(v) != 0;
    t0 = last = std::chrono::steady_clock::now();
  }
  void mark(const char* phase) {
    if (!on) return;
    const auto now = std::chrono::steady_clock::now();
    std::fprintf(stderr, "[mpsb %s] %-28s %8.3f ms (total %8.3f)\n", what, phase,
                 std::chrono::duration<double, std::milli>(now - last).count(),
                 std::chrono::duration<double, std::milli>(now - t0).count());
    last = now;
  }
};

std::string describe_device_error(uint32_t bits) {
  std::string m = "device reported:";
  if (bits & kErrCountMismatch) m += " Histogram sample count does not match node statistics;";
  if (bits & kErrNonFinite) m += " non-finite histogram, gain or leaf value;";
  if (bits & kErrHessian) m += " Histogram G/H must be finite and Hessian non-negative;";
  if (bits & kErrSubtraction) m += " Histogram subtraction child exceeded parent;";
  if (bits & kErrPartition) m += " Sample partition counts do not match histogram statistics;";
  if (bits & kErrMissing) m += " missing statistics exceed parent statistics;";
  if (bits & kErrCapacity) m += " internal capacity exceeded;";
  if (bits & kErrGradient) m += " invalid label, prediction, weight or gradient;";
  if (bits & kErrPrefix) m += " non-missing histogram prefix exceeded parent;";
  if (bits & kErrRootCache) m += " hessian scale of the reused root histogram changed;";
  if (bits & kErrLeafQueue) m += " leaf-wise active queue reached max_active_leaves;";
  if (bits & kErrCopy) m += " a tensor copy of the histogram build did not complete;";
  return m;
}

// MPSB_HIST_TMA=1: row-major histogram levels stage their gathered rows with TMA gather4
// copies through this map instead of cp.async. Off by default: on GB300 the gather4 path
// builds the depth-8 levels about 8 % slower than cp.async (the copies complete later and
// the warps wait on them), although it takes the row loads off the L1 tag stage.
void attach_bins_tmap(mpsb_cuda_dataset* d) {
  d->has_bins_tmap = false;
  const char* v = std::getenv("MPSB_HIST_TMA");
  if (!v || std::atoi(v) == 0 || d->slots != uint32_t(kSlots)) return;
  d->has_bins_tmap = encode_bins_tmap(&d->bins_tmap, d->bins.as<uint8_t>(),
                                      uint64_t(d->nfb) * kBlockFeatures, d->n_rows);
}

uint32_t dataset_slots(const uint32_t* bin_count, const uint8_t* has_missing, uint32_t features) {
  uint64_t need = 0;
  for (uint32_t f = 0; f < features; ++f) {
    if (bin_count[f] == 0) throw DataError("every feature needs at least one bin");
    if (bin_count[f] > 65536) throw DataError("a feature may have at most 65536 bins");
    const uint64_t n = uint64_t(bin_count[f]) + (has_missing && has_missing[f] ? 1 : 0);
    if (n > 65536)
      throw UnsupportedError("a feature with missing values may have at most 65535 bins on the CUDA backend");
    need = std::max(need, n);
  }
  if (need <= uint64_t(kSlots)) return uint32_t(kSlots);
  return uint32_t((need + kSlots - 1) / kSlots * kSlots);
}

// ---- device memory kept between calls -------------------------------------------------
namespace {
std::mutex g_pools_mutex;
std::vector<DevicePool*> g_pools;
}  // namespace

DevicePool::DevicePool(int dev, cudaStream_t backend_stream) : device(dev), stream_(backend_stream) {
  std::lock_guard<std::mutex> lock(g_pools_mutex);
  g_pools.push_back(this);
}

DevicePool::~DevicePool() {
  {
    std::lock_guard<std::mutex> lock(g_pools_mutex);
    g_pools.erase(std::find(g_pools.begin(), g_pools.end(), this));
  }
  trim();
}

// A kept block of at most an eighth more than the size wanted, or a new one.
void* DevicePool::take(size_t* bytes) {
  const size_t want = (*bytes + kBlock - 1) / kBlock * kBlock;
  {
    std::lock_guard<std::mutex> lock(mutex_);
    auto best = free_.end();
    for (auto it = free_.begin(); it != free_.end(); ++it)
      if (it->second >= want && it->second <= want + want / 8 && (best == free_.end() || it->second < best->second))
        best = it;
    if (best != free_.end()) {
      void* p = best->first;
      *bytes = best->second;
      kept_ -= best->second;
      free_.erase(best);
      return p;
    }
  }
  DevBuf fresh;
  fresh.alloc(want);
  *bytes = want;
  return std::exchange(fresh.p, nullptr);
}

void DevicePool::give(void* p, size_t bytes) {
  std::lock_guard<std::mutex> lock(mutex_);
  if (!stream_ || bytes > kMost) {
    cudaFree(p);
    return;
  }
  try {
    free_.emplace_back(p, bytes);
  } catch (const std::bad_alloc&) {
    cudaFree(p);
    return;
  }
  kept_ += bytes;
  while (kept_ > kMost) {
    cudaFree(free_.front().first);
    kept_ -= free_.front().second;
    free_.pop_front();
  }
}

size_t DevicePool::trim() {
  std::lock_guard<std::mutex> lock(mutex_);
  for (auto& f : free_) cudaFree(f.first);
  free_.clear();
  return std::exchange(kept_, size_t(0));
}

void DevicePool::close() {
  {
    std::lock_guard<std::mutex> lock(mutex_);
    stream_ = nullptr;
  }
  trim();
}

bool DevicePool::idle() {
  std::unique_lock<std::mutex> no_capture(capturing, std::try_to_lock);
  if (!no_capture) return false;
  cudaStream_t s;
  {
    std::lock_guard<std::mutex> lock(mutex_);
    s = stream_;
  }
  return s && cudaStreamSynchronize(s) == cudaSuccess;
}

size_t DevicePool::kept() const {
  std::lock_guard<std::mutex> lock(mutex_);
  return kept_;
}

void DevicePool::trim_all() {
  std::lock_guard<std::mutex> lock(g_pools_mutex);
  for (DevicePool* p : g_pools) p->trim();
}

void* DevArena::alloc(size_t bytes) {
  bytes = (std::max<size_t>(bytes, 16) + 255) / 256 * 256;  // cudaMalloc's alignment
  if (bytes <= left_) {
    void* p = slab_;
    slab_ += bytes;
    left_ -= bytes;
    return p;
  }
  size_t block = bytes;
  void* p = pool->take(&block);
  blocks_.emplace_back(p, block);
  if (block - bytes > left_) {  // the rest serves the next small ones
    slab_ = static_cast<char*>(p) + bytes;
    left_ = block - bytes;
  }
  return p;
}

DevArena::~DevArena() {
  if (blocks_.empty()) return;
  // After an error of the device nothing is kept; cudaFree then waits by itself.
  const bool idle = pool->idle();
  for (auto& b : blocks_) {
    if (idle) pool->give(b.first, b.second);
    else cudaFree(b.first);
  }
}

// ---- reference semantics evaluated on the host --------------------------------------
void validate_tree_params(const mpsb_train_params& p, uint32_t features) {  // tree_structure.cpp:17-52
  if (p.min_samples_leaf == 0) throw TrainingError("min_samples_leaf must be at least 1");
  if (p.max_leaves == 1) throw TrainingError("max_leaves must be zero or at least 2");
  if (p.max_active_leaves == 1) throw TrainingError("max_active_leaves must be zero or at least 2");
  if (p.max_active_leaves != 0 && p.max_leaves != 0 && p.max_active_leaves > p.max_leaves)
    throw TrainingError("max_active_leaves must not exceed max_leaves");
  auto nonneg = [](double v, const char* what) {
    if (!std::isfinite(v) || v < 0.0) throw TrainingError(std::string(what) + " must be finite and non-negative");
  };
  nonneg(p.min_child_weight, "min_child_weight");
  nonneg(p.reg_lambda, "reg_lambda");
  nonneg(p.reg_alpha, "reg_alpha");
  nonneg(p.max_delta_step, "max_delta_step");
  nonneg(p.gamma, "gamma");
  nonneg(p.min_gain_to_split, "min_gain_to_split");
  if (p.n_monotonic != 0 && p.n_monotonic != features)
    throw TrainingError("monotonic_constraints length must match feature count");
  for (uint32_t i = 0; i < p.n_monotonic; ++i)
    if (p.monotonic_constraints[i] < -1 || p.monotonic_constraints[i] > 1)
      throw TrainingError("monotonic_constraints values must be -1, 0, or 1");
  for (uint32_t g = 0; g < p.n_interaction_groups; ++g) {  // tree_interactions.cpp:57-70
    if (p.interaction_offsets[g + 1] == p.interaction_offsets[g])
      throw TrainingError("interaction constraint groups must be non-empty");
    for (uint32_t i = p.interaction_offsets[g]; i < p.interaction_offsets[g + 1]; ++i)
      if (p.interaction_features[i] >= features)
        throw TrainingError("interaction constraint feature index out of range");
  }
  if (p.split_strategy > 1) throw TrainingError("unknown split strategy");
  if (p.growth_strategy > 1) throw TrainingError("unknown growth strategy");
}

void validate_training_params(const mpsb_train_params& p) {  // trainer.cpp:22-42
  if (p.n_estimators == 0) throw TrainingError("n_estimators must be at least 1");
  if (!std::isfinite(p.learning_rate) || p.learning_rate <= 0.0 || p.learning_rate > 1.0)
    throw TrainingError("learning_rate must be in (0, 1]");
  if (p.max_bins < 2 || p.max_bins > 65536) throw TrainingError("max_bins must be in [2, 65536]");
  if (!std::isfinite(p.objective_alpha) || p.objective_alpha <= 0.0 || p.objective_alpha >= 1.0)
    throw TrainingError("quantile alpha must be in (0, 1)");
  if (!std::isfinite(p.tweedie_variance_power) || p.tweedie_variance_power <= 1.0 ||
      p.tweedie_variance_power >= 2.0)
    throw TrainingError("tweedie variance power must be in (1, 2)");
  if (p.objective > 4) throw TrainingError("unknown training objective");
}

// One pass over the rows: the weight total of ValidateWeights (trainer.cpp:44-66) and,
// for the mean-type objectives (label_mode 1: squared error, finite labels; 2: poisson and
// tweedie, non-negative labels), the weighted label sum of InitialBaseScore
// (trainer.cpp:68-176), both accumulated in row order as the reference does. The two sums
// are independent chains, so one loop costs about one chain. Errors keep the reference's
// order: every weight check before any label check, each at its first failing row.
struct RowSums {
  double total = 0.0;      // sum of weights
  double label_sum = 0.0;  // sum of label * weight (label_mode != 0)
  int label_mode = 0;
};

// The reference's sequential loop, which also finds the first failing row and its error.
RowSums row_sums_checked(const double* w, const double* y, uint64_t n, int label_mode,
                         const char* name) {
  RowSums r;
  r.label_mode = y ? label_mode : 0;
  double total = 0.0, s = 0.0;
  uint64_t w_bad = n, w_ovf = n, y_bad = n, y_ovf = n;
  for (uint64_t i = 0; i < n; ++i) {
    const double x = w ? w[i] : 1.0;
    if (!std::isfinite(x) || x < 0.0) { w_bad = i; break; }
    total += x;
    if (!std::isfinite(total)) { w_ovf = i; break; }
    if (r.label_mode && y_bad == n && y_ovf == n) {
      const double v = y[i];
      if (!std::isfinite(v) || (r.label_mode == 2 && v < 0.0)) {
        y_bad = i;
      } else {
        s += v * x;
        if (!std::isfinite(s)) y_ovf = i;
      }
    }
  }
  if (w_bad < n) throw TrainingError("sample weights must be finite non-negative values");
  if (w_ovf < n) throw TrainingError("sample weight sum overflowed");
  if (total <= 0.0) throw TrainingError("sample weights must contain positive total weight");
  if (y_bad < n) {
    if (r.label_mode == 1) throw TrainingError("Labels must be finite");
    throw TrainingError(std::string(name) + " labels must be non-negative");
  }
  if (y_ovf < n) {
    if (r.label_mode == 1) throw TrainingError("Label accumulation overflowed");
    throw TrainingError(std::string(name) + " label sum overflowed");
  }
  r.total = total;
  r.label_sum = s;
  return r;
}

// Fast path: the two row-order sums in a tight loop (the same additions, so the same
// results) while worker threads check every weight and label; any failed check or
// non-finite sum reruns the sequential loop above for the reference's exact error.
RowSums row_sums(const double* w, const double* y, uint64_t n, int label_mode, const char* name) {
  if (n == 0) throw TrainingError("labels must be non-empty");
  const int mode = y ? label_mode : 0;
  if (!w && !mode) {  // n unit weights: their sum is n exactly
    RowSums r;
    r.total = double(n);
    return r;
  }
  std::atomic<bool> bad{false};
  const uint32_t workers = uint32_t(std::min<uint64_t>(
      std::max(1u, std::min(16u, std::thread::hardware_concurrency())), (n + (1u << 20) - 1) >> 20));
  auto check = [&](uint32_t k, uint32_t of) {
    const uint64_t lo = n * k / of, hi = n * (k + 1) / of;
    bool ok = true;
    for (uint64_t i = lo; i < hi; ++i) {
      const double x = w ? w[i] : 1.0;
      ok &= std::isfinite(x) && !(x < 0.0);
      if (mode) {
        const double v = y[i];
        ok &= std::isfinite(v) && !(mode == 2 && v < 0.0);
      }
    }
    if (!ok) bad.store(true, std::memory_order_relaxed);
  };
  std::vector<std::thread> pool;
  if (workers > 1)
    for (uint32_t k = 0; k < workers; ++k) pool.emplace_back(check, k, workers);
  else
    check(0, 1);
  double total = 0.0, s = 0.0;
  if (mode) {
    for (uint64_t i = 0; i < n; ++i) {
      const double x = w ? w[i] : 1.0;
      total += x;
      s += y[i] * x;
    }
  } else if (w) {
    for (uint64_t i = 0; i < n; ++i) total += w[i];
  } else {
    for (uint64_t i = 0; i < n; ++i) total += 1.0;
  }
  for (auto& t : pool) t.join();
  if (bad.load() || !std::isfinite(total) || !(total > 0.0) || (mode && !std::isfinite(s)))
    return row_sums_checked(w, y, n, label_mode, name);
  RowSums r;
  r.label_mode = mode;
  r.total = total;
  r.label_sum = s;
  return r;
}

double validate_weights(const double* w, uint64_t n) {  // trainer.cpp:44-66
  return row_sums(w, nullptr, n, 0, nullptr).total;
}

// Whether every label is a whole number in [0, limit); `seen` (or null) gets a 1 at each
// that occurs. 2: some are -0.0. A thread per 2^17 rows, at most 16; nothing is thrown.
int class_ids(const double* y, uint64_t n, uint32_t limit, uint8_t* seen) {
  std::atomic<bool> bad{false}, minus{false};
  auto check = [&](uint64_t lo, uint64_t hi) {
    bool ok = true, neg = false;
    for (uint64_t i = lo; i < hi && ok; i += 4096) {
      const uint64_t end = std::min(hi, i + 4096);
      for (uint64_t k = i; k < end; ++k) {
        ok &= (y[k] >= 0.0) & (y[k] < double(limit)) & (std::trunc(y[k]) == y[k]);
        neg |= std::signbit(y[k]);
      }
      for (uint64_t k = i; seen && ok && k < end; ++k) {
        uint8_t* s = seen + uint32_t(y[k]);  // written once: its line stays shared by the threads
        if (!__atomic_load_n(s, __ATOMIC_RELAXED)) __atomic_store_n(s, uint8_t(1), __ATOMIC_RELAXED);
      }
    }
    if (!ok) bad.store(true, std::memory_order_relaxed);
    if (neg) minus.store(true, std::memory_order_relaxed);
  };
  const uint64_t workers = std::max<uint64_t>(
      1, std::min<uint64_t>(std::max(1u, std::min(16u, std::thread::hardware_concurrency())), n >> 17));
  std::thread pool[16];
  for (uint64_t k = 1; k < workers; ++k) {
    const uint64_t lo = n * k / workers, hi = n * (k + 1) / workers;
    try {
      pool[k] = std::thread(check, lo, hi);
    } catch (const std::exception&) {  // no thread, or no memory for one
      check(lo, hi);
    }
  }
  check(0, n / workers);
  for (auto& t : pool)
    if (t.joinable()) t.join();
  return bad.load() ? 0 : (minus.load() ? 2 : 1);
}

const char* count_objective_name(uint32_t objective) {
  return objective == MPSB_POISSON ? "poisson" : "tweedie";
}

// The label mode of row_sums for a boosting objective (0: the base score needs another pass).
int label_mode_of(uint32_t objective) {
  if (objective == MPSB_SQUARED_ERROR) return 1;
  if (objective == MPSB_POISSON || objective == MPSB_TWEEDIE) return 2;
  return 0;
}

// The logistic base score of a positive weight total.
double logistic_base(double pos, double total) {
  const double eps = 1e-15;
  double prob = pos / total;
  prob = std::min(1.0 - eps, std::max(eps, prob));
  return std::log(prob / (1.0 - prob));
}

// InitialBaseScore (trainer.cpp:68-176) on host FP64 in row order. `cls` >= 0 selects the
// one-vs-rest binary labels (label == cls). `pre`: this fit's row sums, when they carry
// the label sum of the objective (cls < 0).
double base_score(const mpsb_train_params& p, const double* y, const double* w, uint64_t n,
                  int64_t cls, const RowSums* pre = nullptr) {
  const int mode = cls < 0 ? label_mode_of(p.objective) : 0;
  if (mode && pre && pre->label_mode == mode) {
    if (mode == 1) return pre->label_sum / pre->total;
    return std::log(std::max(1e-15, pre->label_sum / pre->total));
  }
  if (mode) {
    const RowSums r = row_sums(w, y, n, mode, count_objective_name(p.objective));
    if (mode == 1) return r.label_sum / r.total;
    return std::log(std::max(1e-15, r.label_sum / r.total));
  }
  const double total = pre ? pre->total : validate_weights(w, n);
  auto W = [&](uint64_t i) { return w ? w[i] : 1.0; };
  auto Y = [&](uint64_t i) { return cls >= 0 ? (y[i] == double(cls) ? 1.0 : 0.0) : y[i]; };
  switch (p.objective) {
    case MPSB_BINARY_LOGISTIC: {
      double pos = 0.0;
      for (uint64_t i = 0; i < n; ++i) {
        const double l = Y(i);
        if (l == 0.0) continue;
        if (l == 1.0) { pos += W(i); continue; }
        throw TrainingError("binary-logistic labels must be 0 or 1");
      }
      return logistic_base(pos, total);
    }
    case MPSB_QUANTILE: {
      std::vector<std::pair<double, double>> o(n);
      for (uint64_t i = 0; i < n; ++i) {
        if (!std::isfinite(Y(i))) throw TrainingError("label must be finite");
        o[i] = {Y(i), W(i)};
      }
      std::sort(o.begin(), o.end(), [](const auto& a, const auto& b) { return a.first < b.first; });
      const double thr = p.objective_alpha * total;
      double cum = 0.0;
      for (const auto& it : o) {
        cum += it.second;
        if (cum >= thr) return it.first;
      }
      return o.back().first;
    }
    default:  // squared error, poisson and tweedie take the row_sums path above
      throw TrainingError("unknown training objective");
  }
}

// Runs body(0..count-1) on worker threads (each index once); rethrows the first error.
template <class F>
void parallel_trees(uint32_t count, F&& body) {
  const uint32_t workers = std::min<uint32_t>(count, std::max(1u, std::thread::hardware_concurrency()));
  std::atomic<uint32_t> next{0};
  std::vector<std::exception_ptr> errors(workers);
  auto run = [&](uint32_t w) {
    try {
      for (uint32_t i = next.fetch_add(1); i < count; i = next.fetch_add(1)) body(i);
    } catch (...) {
      errors[w] = std::current_exception();
    }
  };
  std::vector<std::thread> pool;
  for (uint32_t w = 1; w < workers; ++w) pool.emplace_back(run, w);
  if (workers > 0) run(0);
  for (auto& t : pool) t.join();
  for (auto& e : errors)
    if (e) std::rethrow_exception(e);
}

// InitialBaseScore of a mean-type objective (label_mode 1 or 2) over a row multiset in
// row order, row r taken m[r] times: the same sequence of additions as over the expanded
// sample, without expanding it.
double multiset_base_score(const mpsb_train_params& p, const double* y, const double* w,
                           const uint8_t* m, uint64_t n, int mode) {
  // A piece of the expanded sample at a time: the terms are laid out without a branch per
  // draw (four copies written, the count kept), then added in order.
  double total = 0.0, s = 0.0;
  uint64_t drawn = 0;
  bool bad_w = false, bad_y = false;
  constexpr uint32_t kPiece = 4096;
  std::vector<double> ys(kPiece + 256 + 4), ws(w ? kPiece + 256 + 4 : 0);
  for (uint64_t r = 0; r < n;) {
    uint32_t pos = 0;
    for (; r < n && pos < kPiece; ++r) {
      const uint32_t c = m[r];
      const double x = w ? w[r] : 1.0, v = y[r] * x;
      bad_w |= (c != 0) & (!std::isfinite(x) | (x < 0.0));
      bad_y |= (c != 0) & (!std::isfinite(y[r]) | ((mode == 2) & (y[r] < 0.0)));
      for (uint32_t q = 0; q < 4; ++q) ys[pos + q] = v;
      for (uint32_t q = 4; q < c; ++q) ys[pos + q] = v;
      if (w) {
        for (uint32_t q = 0; q < 4; ++q) ws[pos + q] = x;
        for (uint32_t q = 4; q < c; ++q) ws[pos + q] = x;
      }
      pos += c;
    }
    for (uint32_t q = 0; q < pos; ++q) s += ys[q];
    if (w)
      for (uint32_t q = 0; q < pos; ++q) total += ws[q];
    drawn += pos;
  }
  if (!w) total = double(drawn);  // the sum of that many ones, exactly
  if (bad_w || bad_y || !std::isfinite(total) || !(total > 0.0) || !std::isfinite(s)) {
    // The exact error of the reference's sequential checks, over the expanded sample.
    std::vector<double> ys, ws;
    for (uint64_t r = 0; r < n; ++r)
      for (uint32_t c = 0; c < m[r]; ++c) {
        ys.push_back(y[r]);
        if (w) ws.push_back(w[r]);
      }
    return base_score(p, ys.data(), w ? ws.data() : nullptr, ys.size(), -1);
  }
  if (mode == 1) return s / total;
  return std::log(std::max(1e-15, s / total));
}

uint32_t effective_max_leaves(const mpsb_train_params& p) {  // tree_structure.cpp:54-62
  if (p.max_leaves != 0) return p.max_leaves;
  if (p.max_depth >= 31) return 0xFFFFFFFFu;
  return 1u << p.max_depth;
}

// Fixed-point exponents of one set of FP32 pairs (same rule as the round_setup kernel).
void fixed_scales(const float* pairs32, uint64_t n, uint64_t n_rows, int32_t* kg, int32_t* kh) {
  float mg = 0.0f, mh = 0.0f;
  for (uint64_t i = 0; i < n; ++i) {
    mg = std::max(mg, std::fabs(pairs32[2 * i]));
    mh = std::max(mh, std::max(pairs32[2 * i + 1], 0.0f));
  }
  (void)n_rows;
  int e;
  std::frexp(mg, &e);
  *kg = mg > 0.0f ? 30 - e : 0;
  std::frexp(mh, &e);
  *kh = mh > 0.0f ? 30 - e : 0;
}

}  // namespace mpsb

// ======================================================================================
// Backend
// ======================================================================================
extern "C" {

const char* mpsb_cuda_last_error(void) { return g_error.c_str(); }
int mpsb_cuda_abi_version(void) { return MPSB_CUDA_ABI_VERSION; }

int mpsb_cuda_device_count(int* out) {
  return guard([&] {
    if (out == nullptr) throw TrainingError("output pointer must not be null");
    *out = 0;
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess) {  // no driver or no device
      cudaGetLastError();
      return;
    }
    int usable = 0;
    for (int d = 0; d < count; ++d) {
      int major = 0, minor = 0;
      if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, d) == cudaSuccess &&
          cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, d) == cudaSuccess &&
          major == 10 && minor == 3)
        ++usable;
    }
    cudaGetLastError();
    *out = usable;
  });
}

int mpsb_cuda_backend_create(int device, mpsb_cuda_backend** out) {
  return guard([&] {
    if (out == nullptr) throw TrainingError("output pointer must not be null");
    int count = 0;
    CK(cudaGetDeviceCount(&count));
    if (device < 0 || device >= count) throw BackendError("CUDA device index out of range");
    std::unique_ptr<mpsb_cuda_backend> b(new mpsb_cuda_backend);
    b->device = device;
    CK(cudaSetDevice(device));
    CK(cudaGetDeviceProperties(&b->prop, device));
    if (b->prop.major != 10 || b->prop.minor != 3)
      throw BackendError("the CUDA backend is built for sm_103a (GB300); device " +
                         std::string(b->prop.name) + " has compute capability " +
                         std::to_string(b->prop.major) + "." + std::to_string(b->prop.minor));
    b->sm_count = b->prop.multiProcessorCount;
    CK(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
    CK(cudaEventCreate(&b->t0));
    CK(cudaEventCreate(&b->t1));
    b->error.alloc(sizeof(uint32_t));
    CK(cudaMemset(b->error.p, 0, sizeof(uint32_t)));
    b->pool = std::make_shared<DevicePool>(device, b->stream);
    *out = b.release();
  });
}

void mpsb_cuda_backend_destroy(mpsb_cuda_backend* b) { delete b; }

int mpsb_cuda_backend_info(const mpsb_cuda_backend* b, mpsb_cuda_info* out) {
  return guard([&] {
    std::memset(out, 0, sizeof *out);
    out->available = 1;
    out->sm_count = uint32_t(b->sm_count);
    out->cc_major = uint32_t(b->prop.major);
    out->cc_minor = uint32_t(b->prop.minor);
    out->total_memory = b->prop.totalGlobalMem;
    std::snprintf(out->device_name, sizeof out->device_name, "%.95s", b->prop.name);
  });
}

int mpsb_cuda_backend_set_hist_mode(mpsb_cuda_backend* b, int mode) {
  return guard([&] {
    if (mode != MPSB_HIST_FIXED && mode != MPSB_HIST_FLOAT) throw TrainingError("unknown histogram mode");
    b->hist_mode = mode;
  });
}

int mpsb_cuda_timer_begin(mpsb_cuda_backend* b) {
  return guard([&] { CK(cudaEventRecord(b->t0, b->stream)); });
}

int mpsb_cuda_timer_end(mpsb_cuda_backend* b, float* ms) {
  return guard([&] {
    CK(cudaEventRecord(b->t1, b->stream));
    CK(cudaEventSynchronize(b->t1));
    CK(cudaEventElapsedTime(ms, b->t0, b->t1));
  });
}

int mpsb_cuda_backend_trim(mpsb_cuda_backend* b, uint64_t* given_back) {
  return guard([&] {
    if (!b) throw TrainingError("null argument");
    b->activate();
    const size_t bytes = b->pool->trim();
    if (given_back) *given_back = bytes;
  });
}

int mpsb_cuda_synchronize(mpsb_cuda_backend* b) {
  return guard([&] { CK(cudaStreamSynchronize(b->stream)); });
}

int mpsb_cuda_host_register(void* p, uint64_t bytes) {
  return guard([&] { CK(cudaHostRegister(p, bytes, cudaHostRegisterDefault)); });
}

int mpsb_cuda_host_unregister(void* p) {
  return guard([&] { CK(cudaHostUnregister(p)); });
}

// ---- binning ---------------------------------------------------------------------------
int mpsb_quantize_dense(const void* data, int scalar_type, uint64_t rows, uint32_t features,
                        uint64_t rs, uint64_t cs, uint32_t max_bins, uint32_t n_threads,
                        void* bins, uint8_t* missing, float* boundaries,
                        uint64_t* boundary_offset, uint32_t* boundary_count,
                        uint32_t* bin_count, uint64_t* missing_count) {
  return guard([&] {
    mpsb::quantize_dense(data, scalar_type, rows, features, rs, cs, max_bins, n_threads, bins,
                         missing, boundaries, boundary_offset, boundary_count, bin_count,
                         missing_count);
  });
}

int mpsb_transform_dense(const void* data, int scalar_type, uint64_t rows, uint32_t features,
                         uint64_t rs, uint64_t cs, uint32_t max_bins, const float* boundaries,
                         const uint64_t* boundary_offset, const uint32_t* boundary_count,
                         uint32_t n_threads, void* bins, uint8_t* missing) {
  return guard([&] {
    mpsb::transform_dense(data, scalar_type, rows, features, rs, cs, max_bins, boundaries,
                          boundary_offset, boundary_count, n_threads, bins, missing);
  });
}

}  // extern "C"

// ---- dataset ---------------------------------------------------------------------------
namespace mpsb {

void dataset_ready(const mpsb_cuda_dataset* d) {
  if (d == nullptr) return;
  std::lock_guard<std::mutex> lock(d->ready_mutex);
  if (d->pending) {
    d->backend->activate();
    CK(cudaEventSynchronize(d->ready));
    uint32_t e = 0;
    CK(cudaMemcpy(&e, d->pack_error.p, sizeof e, cudaMemcpyDeviceToHost));
    for (int k = 0; k < 2; ++k) {
      d->stage[k].reset();
      d->mstage[k].reset();
    }
    d->pending = false;
    d->invalid = e != 0;
  }
  if (d->invalid) throw DataError("Binned value exceeds the feature histogram range");
}

namespace {

// Allocates the dataset and enqueues its upload and pack; returns before they complete
// (the dataset is pending).
std::unique_ptr<mpsb_cuda_dataset> start_dataset(mpsb_cuda_backend* b, const void* bins,
                                                 uint32_t width, const uint8_t* missing,
                                                 uint64_t rows, uint32_t features,
                                                 const uint32_t* bin_count) {
  if (!b || !bins || !bin_count) throw TrainingError("null argument");
  if (width != 1 && width != 2) throw DataError("bin width must be 1 or 2 bytes");
  if (rows == 0 || features == 0) throw DataError("dataset must contain at least one row and one feature");
  if (rows >= 0xFFFFFFFFull) throw UnsupportedError("the CUDA backend indexes rows with uint32");
  b->activate();
  PhaseTrace trace("dataset");
  std::unique_ptr<mpsb_cuda_dataset> d(new mpsb_cuda_dataset);
  d->backend = b;
  d->n_rows = uint32_t(rows);
  d->features = features;
  d->nfb = (features + kBlockFeatures - 1) / kBlockFeatures;
  d->h_bin_count.assign(bin_count, bin_count + features);
  d->h_has_missing.assign(features, 0);
  if (missing) {
    for (uint32_t f = 0; f < features; ++f) {
      const uint8_t* m = missing + uint64_t(f) * rows;
      for (uint64_t r = 0; r < rows; ++r)
        if (m[r]) { d->h_has_missing[f] = 1; break; }
    }
  }
  d->slots = dataset_slots(bin_count, d->h_has_missing.data(), features);
  const bool wide = d->slots != uint32_t(kSlots);
  trace.mark("bin counts, missing scan");
  d->bin_count.alloc(features * sizeof(uint32_t));
  d->has_missing.alloc(features);
  CK(cudaMemcpyAsync(d->bin_count.p, bin_count, features * sizeof(uint32_t), cudaMemcpyHostToDevice, b->stream));
  CK(cudaMemcpyAsync(d->has_missing.p, d->h_has_missing.data(), features, cudaMemcpyHostToDevice, b->stream));
  if (wide) {
    d->bins16.alloc(size_t(d->nfb) * rows * kBlockFeatures * sizeof(uint16_t));
    d->bins16_fm.alloc(size_t(features) * rows * sizeof(uint16_t));
  } else {
    d->bins.alloc(size_t(d->nfb) * rows * kBlockFeatures);
    d->bins_blocked.alloc(size_t(d->nfb) * rows * kBlockFeatures);
    d->bins_fm.alloc(size_t(features) * rows);
  }
  d->pack_error.alloc(sizeof(uint32_t));
  CK(cudaMemsetAsync(d->pack_error.p, 0, sizeof(uint32_t), b->stream));
  CK(cudaEventCreateWithFlags(&d->ready, cudaEventDisableTiming));
  trace.mark("allocs");
  // Feature block by feature block (32 feature columns, contiguous in the feature-major
  // source): the copy stream uploads block fb + 1 into one staging buffer while the
  // compute stream packs block fb from the other.
  if (!b->copy_stream) CK(cudaStreamCreateWithFlags(&b->copy_stream, cudaStreamNonBlocking));
  const size_t block_cells = size_t(kBlockFeatures) * rows;
  DevBuf* stage = d->stage;
  DevBuf* mstage = d->mstage;
  const int nstage = d->nfb > 1 ? 2 : 1;
  for (int k = 0; k < nstage; ++k) {
    stage[k].alloc(block_cells * width);
    if (missing) mstage[k].alloc(block_cells);
  }
  struct Events {
    cudaEvent_t e[4] = {nullptr, nullptr, nullptr, nullptr};
    ~Events() {
      for (cudaEvent_t x : e)
        if (x) cudaEventDestroy(x);
    }
  } ev;  // copied[2], packed[2]
  for (cudaEvent_t& x : ev.e) CK(cudaEventCreateWithFlags(&x, cudaEventDisableTiming));
  for (uint32_t fb = 0; fb < d->nfb; ++fb) {
    const int k = int(fb & 1);
    const uint32_t nf = std::min<uint32_t>(kBlockFeatures, features - fb * kBlockFeatures);
    const size_t first = size_t(fb) * block_cells;
    if (fb >= 2) CK(cudaStreamWaitEvent(b->copy_stream, ev.e[2 + k], 0));  // block fb-2 packed
    CK(cudaMemcpyAsync(stage[k].p, static_cast<const uint8_t*>(bins) + first * width,
                       size_t(nf) * rows * width, cudaMemcpyHostToDevice, b->copy_stream));
    if (missing)
      CK(cudaMemcpyAsync(mstage[k].p, missing + first, size_t(nf) * rows, cudaMemcpyHostToDevice,
                         b->copy_stream));
    CK(cudaEventRecord(ev.e[k], b->copy_stream));
    CK(cudaStreamWaitEvent(b->stream, ev.e[k], 0));
    if (wide)
      CK(launch_pack_bins16_block(stage[k].p, width, missing ? mstage[k].as<uint8_t>() : nullptr,
                                  d->bin_count.as<uint32_t>(), d->n_rows, features, fb, d->slots,
                                  d->bins16.as<uint16_t>(), d->bins16_fm.as<uint16_t>(),
                                  d->pack_error.as<uint32_t>(), b->stream));
    else
      CK(launch_pack_bins_block(stage[k].p, width, missing ? mstage[k].as<uint8_t>() : nullptr,
                                d->bin_count.as<uint32_t>(), d->n_rows, features, d->nfb, fb,
                                d->bins.as<uint8_t>(), d->bins_blocked.as<uint8_t>(),
                                d->bins_fm.as<uint8_t>(), d->pack_error.as<uint32_t>(), b->stream));
    CK(cudaEventRecord(ev.e[2 + k], b->stream));
  }
  CK(cudaEventRecord(d->ready, b->stream));
  d->pending = true;
  trace.mark("upload + pack (enqueued)");
  attach_bins_tmap(d.get());
  return d;
}

}  // namespace
}  // namespace mpsb

extern "C" {

int mpsb_cuda_dataset_create(mpsb_cuda_backend* b, const void* bins, uint32_t width,
                             const uint8_t* missing, uint64_t rows, uint32_t features,
                             const uint32_t* bin_count, mpsb_cuda_dataset** out) {
  return guard([&] {
    if (!out) throw TrainingError("null argument");
    std::unique_ptr<mpsb_cuda_dataset> d = start_dataset(b, bins, width, missing, rows, features, bin_count);
    PhaseTrace trace("dataset");
    dataset_ready(d.get());
    trace.mark("upload + pack (synchronized)");
    *out = d.release();
  });
}

int mpsb_cuda_dataset_create_async(mpsb_cuda_backend* b, const void* bins, uint32_t width,
                                   const uint8_t* missing, uint64_t rows, uint32_t features,
                                   const uint32_t* bin_count, mpsb_cuda_dataset** out) {
  return guard([&] {
    if (!out) throw TrainingError("null argument");
    *out = start_dataset(b, bins, width, missing, rows, features, bin_count).release();
  });
}

int mpsb_cuda_dataset_wait(const mpsb_cuda_dataset* d) {
  return guard([&] {
    if (!d) throw TrainingError("null argument");
    dataset_ready(d);
  });
}

void mpsb_cuda_dataset_destroy(mpsb_cuda_dataset* d) { delete d; }

int mpsb_cuda_dataset_uses_tma(const mpsb_cuda_dataset* d) { return d && d->has_bins_tmap ? 1 : 0; }

}  // extern "C"

// ======================================================================================
// Autotuned launch shapes, per fit shape
// ======================================================================================
namespace mpsb {

std::mutex g_tune_mutex;
std::map<TuneKey, mpsb_cuda_tuning> g_tune_table;

// The shape of a single-model fit (forests, softmax and one-vs-rest keep the built-in
// launch shape).
bool unit_hessian_fit(const double* weights, const mpsb_train_params& p) {
  bool unit = !weights && (p.objective == MPSB_SQUARED_ERROR || p.objective == MPSB_QUANTILE);
  if (const char* v = std::getenv("MPSB_UNIT_HESS")) unit = unit && std::atoi(v) != 0;
  return unit;
}

// The split scan in two launches: best splits with the FP32 screen's quadratic score.
bool two_launch_scan(const mpsb_train_params& p) {
  return p.split_strategy == 0 && p.reg_alpha == 0.0 && p.reg_lambda > 0.0;
}

TuneKey tune_key_of(const mpsb_cuda_dataset* ds, const double* weights, const mpsb_train_params& p,
                    uint32_t options) {
  return TuneKey{ds->n_rows, ds->features, p.max_depth,
                 uint32_t((options & MPSB_OPT_FLOAT_HIST) ? kModeFloat : kModeFixed),
                 unit_hessian_fit(weights, p) ? 1u : 0u, weights ? 1u : 0u,
                 p.growth_strategy == 1 ? 1u : 0u, ds->slots, two_launch_scan(p) ? 1u : 0u};
}

bool tuned_shape(const TuneKey& k, mpsb_cuda_tuning* out) {
  std::lock_guard<std::mutex> lock(g_tune_mutex);
  const auto it = g_tune_table.find(k);
  if (it == g_tune_table.end()) return false;
  *out = it->second;
  return true;
}

}  // namespace mpsb

// ======================================================================================
// Training session
// ======================================================================================
struct mpsb_cuda_trainer {
  mpsb_cuda_backend* b = nullptr;
  const mpsb_cuda_dataset* ds = nullptr;
  mpsb_train_params params{};
  uint32_t options = 0;
  uint32_t depth = 0;
  uint32_t n_trees = 1;
  bool ovr = false;
  TrainerDev dev{};
  HistConfig hcfg;
  DevArena mem;
  std::vector<double> base_scores;
  // One graph for a full round and one for a round that reuses the roots' count and
  // hessian histograms.
  cudaGraph_t graph[2] = {nullptr, nullptr};
  cudaGraphExec_t graph_exec[2] = {nullptr, nullptr};
  bool leafwise = false;   // growth_strategy leaf_wise: steps instead of depth levels
  uint32_t lw_steps = 0;    // split steps per tree and round (max leaves - 1)
  bool root_reuse = false;  // the hessian does not depend on the prediction
  uint32_t softmax_classes = 0;  // native softmax: one tree per class per round
  bool root_saved = false;  // a round has saved the roots' count/hessian histograms
  std::vector<cudaEvent_t> events;  // 2 per level (histogram build begin/end)
  unsigned long long* level_cells = nullptr;  // device: ctl->cells after each level's build
  std::vector<double> level_ms;
  std::vector<uint64_t> level_cells_total;
  uint32_t rounds_enqueued = 0;
  uint32_t blocked_levels = 2;  // levels built from the column-blocked bins
  uint32_t* limb_votes = nullptr;  // (device) TrainerDev::limb_votes, level by level
  size_t limb_vote_words = 0;      // per level
  mpsb_cuda_stats stats{};
  uint64_t kernels_per_round[2] = {0, 0};
  uint64_t cells_base = 0, rows_base = 0, part_base = 0;
  unsigned long long cells_before_round = 0;

  template <class T>
  T* alloc(size_t count) {
    return static_cast<T*>(mem.alloc(count * sizeof(T)));
  }

  cudaStream_t side = nullptr;                      // work beside the main stream
  cudaEvent_t fork_ev = nullptr, zero_ev = nullptr;  // fork to / join from `side`

  ~mpsb_cuda_trainer() {
    if (fork_ev) cudaEventDestroy(fork_ev);
    if (zero_ev) cudaEventDestroy(zero_ev);
    if (side) {
      cudaStreamSynchronize(side);  // `mem` is reused once the backend's stream is idle
      cudaStreamDestroy(side);
    }
    for (int i = 0; i < 2; ++i) {
      if (graph_exec[i]) cudaGraphExecDestroy(graph_exec[i]);
      if (graph[i]) cudaGraphDestroy(graph[i]);
    }
    for (cudaEvent_t e : events) cudaEventDestroy(e);
  }

  int grid(int per_sm) const { return b->sm_count * per_sm; }

  // The most nodes depth level d can hold, over all trees.
  uint32_t level_nodes(uint32_t d) const {
    return uint32_t(std::min<uint64_t>(dev.max_level_nodes, uint64_t(n_trees) << std::min<uint32_t>(d, 31)));
  }

  // The split scan's CTA size and what follows from it: the one-launch scan writes a record per
  // feature chunk, and its readers step over them by partial_stride.
  void set_scan_threads(uint32_t threads) {
    dev.scan_threads = threads;
    dev.n_fchunks = (dev.features + threads / 32 - 1) / (threads / 32);
    dev.partial_stride = dev.scan_two_phase ? 1u : dev.n_fchunks;
  }

  // Captured rounds bake in the launch shape: drop them after a change.
  void reset_graphs() {
    for (int i = 0; i < 2; ++i) {
      if (graph_exec[i]) cudaGraphExecDestroy(graph_exec[i]);
      if (graph[i]) cudaGraphDestroy(graph[i]);
      graph_exec[i] = nullptr;
      graph[i] = nullptr;
    }
  }

  void apply_shape(const mpsb_cuda_tuning& s) {
    hcfg.threads = int(s.hist_threads);
    hcfg.stages = int(s.hist_stages);
    hcfg.root_threads = int(s.root_threads);
    dev.items_per_sm = s.items_per_sm;
    blocked_levels = s.blocked_levels;
    set_scan_threads(s.scan_threads);
    reset_graphs();
  }

  // Enqueue one boosting round. Returns the number of kernels enqueued. root_gradient_only:
  // the roots' count and hessian histograms come from the fit's first round.
  uint64_t enqueue_round(bool record_events, bool root_gradient_only) {
    cudaStream_t s = b->stream;
    uint64_t k = 0;
    // The roots' slots are cleared beside the gradients.
    CK(cudaEventRecord(fork_ev, s));
    CK(cudaStreamWaitEvent(side, fork_ev, 0));
    CK(launch_zero_root_slots(dev, root_gradient_only, grid(8), side)); ++k;
    CK(cudaEventRecord(zero_ev, side));
    CK(launch_gradients(dev, root_gradient_only,
                        std::max(1, std::min(grid(4), int((dev.seg_stride + 255) / 256))), s)); ++k;
    CK(cudaStreamWaitEvent(s, zero_ev, 0));
    if (leafwise) {
      k += enqueue_leafwise(root_gradient_only);
      CK(launch_apply_leaves(dev, grid(8), s)); k += 2;
      return k;
    }
    const uint32_t levels = std::max<uint32_t>(depth, 1);
    for (uint32_t d = 0; d < levels; ++d) {
      const int parity = int(d & 1);
      if (d > 0) CK(cudaStreamWaitEvent(s, zero_ev, 0));  // its slots were cleared beside the partition
      if (record_events) CK(cudaEventRecord(events[2 * d], s));
      if (options & MPSB_OPT_PER_NODE) {
        k += enqueue_hist_per_node(d);
      } else {
        TrainerDev view = level_view(d);
        if (d == 0 && root_gradient_only) view.mode = kModeFixedG;
        CK(launch_hist_build(view, hcfg, grid(1), s)); ++k;
      }
      if (record_events) {
        CK(cudaEventRecord(events[2 * d + 1], s));
        CK(cudaMemcpyAsync(level_cells + d, &dev.ctl->cells, sizeof(unsigned long long),
                           cudaMemcpyDeviceToDevice, s));
      }
      if (d == 0) {
        k += enqueue_root_stats(root_gradient_only);
      } else if (!dev.fused_sub) {
        CK(launch_subtract(dev, grid(8), s)); ++k;
      }
      if (depth > 0) {
        CK(launch_split_scan(dev, parity, level_nodes(d), d == 0 ? ScanKind::kRoot : ScanKind::kLevel, d + 1 == depth,
                             grid(4), s)); k += split_scan_kernels(dev);
      }
      CK(launch_finalize(dev, parity, d, level_nodes(d), s)); ++k;
      if (d + 1 < depth) {
        // The next level's build slots (named by the finalize) are cleared on the side
        // stream while the partition moves the rows.
        CK(cudaEventRecord(fork_ev, s));
        CK(cudaStreamWaitEvent(side, fork_ev, 0));
        CK(launch_zero_build_slots(dev, grid(8), side)); ++k;
        CK(cudaEventRecord(zero_ev, side));
        CK(launch_partition(dev, level_nodes(d), grid(4), s)); k += partition_kernels(dev, level_nodes(d));
      }
    }
    CK(launch_apply_leaves(dev, grid(8), s)); k += 2;
    return k;
  }

  // After the roots' histograms: their cache in a fit's first round, and their statistics
  // where the split scan does not form them.
  uint64_t enqueue_root_stats(bool root_gradient_only) {
    uint64_t k = 0;
    if (root_reuse && !root_gradient_only) {
      CK(launch_root_cache(dev, grid(4), b->stream)); ++k;
    }
    if (depth == 0 || !scan_forms_root(dev)) {
      CK(launch_root_stats(dev, b->stream)); ++k;
    }
    return k;
  }

  // Leaf-wise round body: the root as a depth-0 level, then lw_steps split steps
  // (select, partition, smaller-child histogram, subtraction, children's split scan,
  // merge), then the leaf segments.
  uint64_t enqueue_leafwise(bool root_gradient_only) {
    cudaStream_t s = b->stream;
    uint64_t k = 0;
    TrainerDev view = level_view(0);
    if (root_gradient_only) view.mode = kModeFixedG;
    CK(launch_hist_build(view, hcfg, grid(1), s)); ++k;
    k += enqueue_root_stats(root_gradient_only);
    if (depth > 0) {
      CK(launch_split_scan(dev, 0, n_trees, ScanKind::kRoot, false, grid(4), s)); k += split_scan_kernels(dev);
    }
    CK(launch_leafwise_init(dev, s)); ++k;
    for (uint32_t step = 0; step < lw_steps && depth > 0; ++step) {
      CK(launch_leafwise_select(dev, s)); ++k;
      // The built child's slot is cleared beside the partition, as between levels.
      CK(cudaEventRecord(fork_ev, s));
      CK(cudaStreamWaitEvent(side, fork_ev, 0));
      CK(launch_zero_build_slots(dev, grid(8), side)); ++k;
      CK(cudaEventRecord(zero_ev, side));
      CK(launch_partition(dev, n_trees, grid(4), s)); k += partition_kernels(dev, n_trees);
      CK(cudaStreamWaitEvent(s, zero_ev, 0));
      CK(launch_hist_build(step_view(), hcfg, grid(1), s)); ++k;
      if (!dev.fused_sub) { CK(launch_subtract(dev, grid(8), s)); ++k; }
      const uint32_t scans = split_scan_kernels(dev);
      CK(launch_split_scan(dev, 1, 2 * n_trees, ScanKind::kActive, false, grid(4), s)); k += scans;
      if (scans == 1) { CK(launch_leafwise_merge(dev, s)); ++k; }
    }
    CK(launch_leafwise_finish(dev, s)); ++k;
    return k;
  }

  // The histogram launch's view: unit-hessian fixed-point builds count and gradient limbs.
  TrainerDev build_view() const {
    TrainerDev v = dev;
    if (v.mode == kModeFixed && v.unit_hess) v.mode = kModeFixedCG;
    return v;
  }

  // A leaf-wise step's view: the packed-limb votes of level 1 stand for every step.
  TrainerDev step_view() const {
    TrainerDev v = build_view();
    if (limb_votes) v.limb_votes = limb_votes + limb_vote_words;
    return v;
  }

  // Dense levels (every row of a node close to the next) read the column-blocked copy of
  // the bins, whose 32-byte block rows are consecutive; sparse levels read the padded
  // row-major copy, whose 128-byte row line serves all feature blocks through L2.
  TrainerDev level_view(uint32_t d) const {
    TrainerDev v = build_view();
    if (limb_votes) v.limb_votes = limb_votes + limb_vote_words * d;
    if (d == 0) v.store_single = 0;
    if (d < blocked_levels && !dev.feature_of) {
      v.bins = ds->bins_blocked.as<uint8_t>();
      v.bins_row_stride = kBlockFeatures;
      v.bins_block_stride = uint64_t(ds->n_rows) * kBlockFeatures;
    }
    return v;
  }

  // Plain path: the host reads the level's build list and launches one histogram build
  // per node, waiting for each level (the per-node submit/wait of mps_histogram.mm:62-80).
  uint64_t enqueue_hist_per_node(uint32_t d) {
    cudaStream_t s = b->stream;
    Control c;
    CK(cudaMemcpyAsync(&c, dev.ctl, sizeof c, cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    std::vector<uint32_t> prefix(c.n_build + 1);
    CK(cudaMemcpyAsync(prefix.data(), dev.build_prefix, prefix.size() * sizeof(uint32_t),
                       cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    uint64_t k = 0;
    for (uint32_t e = 0; e < c.n_build; ++e) {
      TrainerDev one = level_view(d);
      one.item_begin = prefix[e] * dev.nfb;
      one.item_end = prefix[e + 1] * dev.nfb;
      CK(cudaMemsetAsync(&dev.ctl->hist_counter, 0, sizeof(uint32_t), s));
      CK(launch_hist_build(one, hcfg, grid(1), s));
      ++k;
      CK(cudaStreamSynchronize(s));
    }
    return k;
  }

  void run(uint32_t rounds) {
    b->activate();
    if (rounds_enqueued + rounds > dev.max_rounds)
      throw TrainingError("training session round capacity exceeded");
    const bool timing = (options & MPSB_OPT_TIMING) && !leafwise;  // events are per depth level
    // Events captured into a graph cannot be timed, so timing runs launch directly.
    const bool use_graph = !(options & (MPSB_OPT_NO_GRAPH | MPSB_OPT_PER_NODE | MPSB_OPT_TIMING));
    PhaseTrace capture_trace("run");
    for (uint32_t r = 0; r < rounds; ++r) {
      const bool g_only = root_reuse && root_saved;
      const int gi = g_only ? 1 : 0;
      if (use_graph) {
        if (!graph_exec[gi]) {
          std::lock_guard<std::mutex> capture(b->pool->capturing);
          CK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
          uint64_t k = 0;
          try {
            k = enqueue_round(timing, g_only);
          } catch (...) {
            cudaGraph_t g = nullptr;
            cudaStreamEndCapture(b->stream, &g);
            if (g) cudaGraphDestroy(g);
            throw;
          }
          CK(cudaStreamEndCapture(b->stream, &graph[gi]));
          CK(cudaGraphInstantiate(&graph_exec[gi], graph[gi], 0));
          kernels_per_round[gi] = k;
          capture_trace.mark(gi ? "capture + instantiate (1)" : "capture + instantiate (0)");
        }
        CK(cudaGraphLaunch(graph_exec[gi], b->stream));
        stats.kernel_launches += kernels_per_round[gi];
      } else {
        stats.kernel_launches += enqueue_round(timing, g_only);
      }
      root_saved = root_reuse;
      stats.hist_launches += (options & MPSB_OPT_PER_NODE) ? 0 : std::max<uint32_t>(depth, 1);
      ++rounds_enqueued;
      ++stats.rounds;
      if (timing) {
        CK(cudaStreamSynchronize(b->stream));
        const uint32_t levels = std::max<uint32_t>(depth, 1);
        std::vector<unsigned long long> after(levels);
        CK(cudaMemcpy(after.data(), level_cells, levels * sizeof(unsigned long long),
                      cudaMemcpyDeviceToHost));
        level_ms.resize(levels, 0.0);
        level_cells_total.resize(levels, 0);
        for (uint32_t d = 0; d < levels; ++d) {
          float ms = 0.0f;
          CK(cudaEventElapsedTime(&ms, events[2 * d], events[2 * d + 1]));
          stats.hist_ms += ms;
          ++stats.hist_timed_launches;
          level_ms[d] += ms;
          level_cells_total[d] += after[d] - (d ? after[d - 1] : cells_before_round);
        }
        cells_before_round = after[levels - 1];
      }
    }
  }

  void synchronize() {
    b->activate();
    CK(cudaStreamSynchronize(b->stream));
    Control c;
    CK(cudaMemcpy(&c, dev.ctl, sizeof c, cudaMemcpyDeviceToHost));
    stats.hist_cells = c.cells - cells_base;
    stats.hist_rows = c.rows_built - rows_base;
    stats.part_rows = c.rows_partitioned - part_base;
    if (c.error) throw TrainingError(describe_device_error(c.error));
  }
};

namespace {

// A batch of forest trees: per tree its sample (a multiset of rows, given as the number of
// times each was drawn), feature subset, random-threshold seed and base score. Compact: the
// trees train on their own features, numbered within their ascending subsets.
struct ForestSpec {
  uint32_t n_trees = 0;
  uint32_t cap = 0;                   // largest sample
  const uint8_t* row_counts = nullptr;  // [n_trees][rows] (host)
  std::vector<uint32_t> count;        // [n_trees]
  bool compact = false;
  uint32_t features = 0;              // the dataset's, or (compact) the largest subset
  std::vector<uint32_t> feature_of;   // compact: [n_trees][features], 0xffffffff past a subset
  std::vector<uint32_t> masks;        // [n_trees][path_words]
  std::vector<uint32_t> ranks;        // [n_trees][features] (compact: empty, rank = number)
  std::vector<uint32_t> seeds;        // [n_trees] or empty
  std::vector<double> base_scores;    // [n_trees]
};

void setup_trainer(mpsb_cuda_trainer* t, mpsb_cuda_backend* b, const mpsb_cuda_dataset* ds,
                   const double* labels, const double* weights, uint64_t n,
                   const mpsb_train_params* p, uint32_t options, uint32_t n_classes,
                   const ForestSpec* forest = nullptr, uint32_t softmax_classes = 0) {
  if (!b || !ds || !labels || !p) throw TrainingError("null argument");
  PhaseTrace trace("setup");
  validate_training_params(*p);
  validate_tree_params(*p, ds->features);
  if (n != ds->n_rows) throw TrainingError("Training data, labels, or max_bins contract does not match");
  // Weight checks and total; for a single boosted tree of a mean-type objective also the
  // base score's label sum, in the same pass.
  const bool single_mean = !forest && !softmax_classes && n_classes == 0 && label_mode_of(p->objective) != 0;
  const RowSums sums = row_sums(weights, single_mean ? labels : nullptr, n, label_mode_of(p->objective),
                                count_objective_name(p->objective));
  trace.mark("validate weights, label sum");
  // An asynchronous dataset upload ran beside the host passes above.
  dataset_ready(ds);
  trace.mark("dataset upload complete");
  b->activate();
  t->b = b;
  t->mem.pool = b->pool;
  t->ds = ds;
  CK(cudaStreamCreateWithFlags(&t->side, cudaStreamNonBlocking));
  CK(cudaEventCreateWithFlags(&t->fork_ev, cudaEventDisableTiming));
  CK(cudaEventCreateWithFlags(&t->zero_ev, cudaEventDisableTiming));
  t->params = *p;
  t->options = options;
  t->depth = p->max_depth;
  t->leafwise = p->growth_strategy == 1;
  if (t->leafwise && (forest || n_classes > 1024))
    throw UnsupportedError("leaf-wise growth on the CUDA backend trains boosting, one-vs-rest (<= 1024 classes) and softmax models");
  t->ovr = n_classes > 0;
  t->n_trees = forest ? forest->n_trees : (t->ovr ? n_classes : 1);
  if (t->ovr && p->objective != MPSB_BINARY_LOGISTIC)
    throw TrainingError("one-vs-rest training uses the binary_logistic objective");
  const uint32_t T = t->n_trees;
  const uint32_t F = forest ? forest->features : ds->features;  // a tree's feature numbers
  const bool compact = forest && forest->compact;
  const uint32_t D = p->max_depth;
  if (D > 24) throw UnsupportedError("max_depth above 24 is not supported by the CUDA backend");
  const uint64_t max_leaves_eff = effective_max_leaves(*p);
  const uint64_t seg_rows = forest ? forest->cap : n;  // positions per tree
  const uint64_t by_rows = std::max<uint64_t>(1, (seg_rows + p->min_samples_leaf - 1) / p->min_samples_leaf);
  const uint64_t leaves = std::min<uint64_t>({uint64_t(1) << std::min<uint32_t>(D, 30), max_leaves_eff, by_rows});
  const uint64_t level_nodes = std::max<uint64_t>(1, std::min<uint64_t>(D ? (uint64_t(1) << (D - 1)) : 1, leaves));
  const uint64_t tree_nodes = 2 * leaves + 1;
  TrainerDev& a = t->dev;
  a = TrainerDev{};
  a.bins = ds->bins.as<uint8_t>();
  a.bins_row_stride = uint64_t(ds->nfb) * kBlockFeatures;
  a.bins_block_stride = kBlockFeatures;
  a.bins_fm = ds->bins_fm.as<uint8_t>();
  a.slots = ds->slots;
  a.scan_two_phase = two_launch_scan(*p);
  // The split scan forms each sibling's histogram (MPSB_FUSED_SUB=0: subtract_kernel
  // does); the one-launch scan on level-wise u8 datasets only.
  a.fused_sub = a.scan_two_phase || (ds->slots == uint32_t(kSlots) && p->growth_strategy != 1);
  if (const char* v = std::getenv("MPSB_FUSED_SUB")) a.fused_sub = a.fused_sub && std::atoi(v) != 0;
  a.bins16 = ds->bins16.as<uint16_t>();
  a.bins16_fm = ds->bins16_fm.as<uint16_t>();
  a.bin_count = ds->bin_count.as<uint32_t>();
  a.sm_count = uint32_t(b->sm_count);
  a.has_missing = ds->has_missing.as<uint8_t>();
  a.n_rows = ds->n_rows;
  a.seg_stride = uint32_t(seg_rows);
  a.features = F;
  a.nfb = (F + kBlockFeatures - 1) / kBlockFeatures;
  a.n_trees = T;
  a.objective = p->objective;
  a.ovr = t->ovr ? 1 : 0;
  a.n_classes = softmax_classes;
  t->softmax_classes = softmax_classes;
  a.mode = (options & MPSB_OPT_FLOAT_HIST) ? kModeFloat : kModeFixed;
  // Four features (warps) per split-scan CTA spread a shallow level's few nodes over many
  // SMs; MPSB_SCAN_THREADS overrides (a multiple of 32, at most 512).
  a.scan_threads = 128;
  // rows per histogram work item: chosen per level on the device (about three items per
  // SM, one for wide datasets, within the 2^16-row limb bound)
  a.item_rows = 0;
  // Squared error and quantile have h = 1 per row; without weights every row's quantized
  // hessian is the same unit (MPSB_UNIT_HESS=0 builds the hessian limbs anyway).
  a.unit_hess = !softmax_classes && n_classes == 0 && unit_hessian_fit(weights, *p);
  {
    // A shape the autotuner chose for this kind of fit.
    mpsb_cuda_tuning tuned{};
    if (!forest && !softmax_classes && n_classes == 0 &&
        tuned_shape(tune_key_of(ds, weights, *p, options), &tuned)) {
      t->hcfg.threads = int(tuned.hist_threads);
      t->hcfg.stages = int(tuned.hist_stages);
      t->hcfg.root_threads = int(tuned.root_threads);
      a.items_per_sm = tuned.items_per_sm;
      t->blocked_levels = tuned.blocked_levels;
      a.scan_threads = tuned.scan_threads;
    }
  }
  t->hcfg.bins_tmap = ds->has_bins_tmap && !compact ? &ds->bins_tmap : nullptr;
  // Launch-shape overrides (tuning sweeps): threads per CTA, pipeline stages, rows per work
  // item, split-scan CTA size.
  if (const char* v = std::getenv("MPSB_SCAN_THREADS"))
    a.scan_threads = uint32_t(std::min(512, std::max(32, std::atoi(v) / 32 * 32)));
  t->set_scan_threads(a.scan_threads);
  if (const char* v = std::getenv("MPSB_HIST_THREADS")) t->hcfg.threads = std::atoi(v);
  if (const char* v = std::getenv("MPSB_HIST_STAGES")) t->hcfg.stages = std::atoi(v);
  t->hcfg.direct = true;
  if (const char* v = std::getenv("MPSB_HIST_DIRECT")) t->hcfg.direct = std::atoi(v) != 0;
  if (const char* v = std::getenv("MPSB_ROOT_THREADS")) t->hcfg.root_threads = std::atoi(v);
  if (const char* v = std::getenv("MPSB_WIDE_THREADS")) t->hcfg.wide_threads = std::atoi(v);
  if (const char* v = std::getenv("MPSB_BLOCKED_LEVELS")) t->blocked_levels = uint32_t(std::atoi(v));
  if (const char* v = std::getenv("MPSB_ITEMS_PER_SM")) a.items_per_sm = uint32_t(std::max(1, std::atoi(v)));
  if (const char* v = std::getenv("MPSB_ITEM_ROWS"))
    a.item_rows = uint32_t(std::min<long>(std::max<long>(std::atol(v), 512), long(kItemRowsMax)));
  // Squared error and quantile have hessian = sample weight, the same in every round: the
  // roots' count and hessian histograms are built once per fit (MPSB_ROOT_REUSE=0 builds
  // them every round).
  t->root_reuse = !forest && !softmax_classes && a.mode == kModeFixed && !(options & MPSB_OPT_PER_NODE) &&
                  (p->objective == MPSB_SQUARED_ERROR || p->objective == MPSB_QUANTILE);
  if (const char* v = std::getenv("MPSB_ROOT_REUSE")) t->root_reuse = t->root_reuse && std::atoi(v) != 0;
  if (t->root_reuse) {
    a.root_cache = t->alloc<unsigned long long>(size_t(T) * F * ds->slots * 2);
    a.root_cache_kh = t->alloc<int>(T);
  }
  TreeParams& tp = a.params;
  tp.min_samples_leaf = p->min_samples_leaf;
  tp.min_child_weight = p->min_child_weight;
  tp.reg_lambda = p->reg_lambda;
  tp.reg_alpha = p->reg_alpha;
  tp.max_delta_step = p->max_delta_step;
  tp.gamma = p->gamma;
  tp.min_gain_to_split = p->min_gain_to_split;
  tp.learning_rate = p->learning_rate;
  tp.max_depth = D;
  tp.max_leaves = uint32_t(std::min<uint64_t>(max_leaves_eff, 0xFFFFFFFFull));
  tp.split_strategy = p->split_strategy;
  tp.random_seed = p->random_seed;
  tp.has_monotonic = p->n_monotonic ? 1 : 0;
  tp.n_groups = p->n_interaction_groups;
  tp.path_words = (F + 31) / 32;
  tp.objective = p->objective;
  tp.objective_alpha = p->objective_alpha;
  tp.tweedie_variance_power = p->tweedie_variance_power;
  set_screen_constants(tp);
  cudaStream_t s = b->stream;
  const uint32_t W = tp.path_words;

  a.store_single = a.mode == kModeFixed && ds->slots == uint32_t(kSlots) && t->hcfg.direct && !t->hcfg.bins_tmap;
  trace.mark("parameters, root cache");
  // inputs
  double* d_labels = t->alloc<double>(n);
  CK(cudaMemcpyAsync(d_labels, labels, n * sizeof(double), cudaMemcpyHostToDevice, s));
  a.labels = d_labels;
  if (weights) {
    double* d_w = t->alloc<double>(n);
    CK(cudaMemcpyAsync(d_w, weights, n * sizeof(double), cudaMemcpyHostToDevice, s));
    a.weights = d_w;
  }

  // Unweighted class fits: the rows of each class, counted on the device. With a label that
  // is no class id the host passes below report it.
  std::vector<unsigned long long> class_rows;
  if (!weights && !forest && (softmax_classes || p->objective == MPSB_BINARY_LOGISTIC)) {
    const uint32_t K = softmax_classes ? softmax_classes : (t->ovr ? n_classes : 2u);
    if (K <= kLabelCountMax) {
      unsigned long long* d_counts = t->alloc<unsigned long long>(K + 1);
      CK(cudaMemsetAsync(d_counts, 0, (K + 1) * sizeof(unsigned long long), s));
      CK(launch_label_counts(d_labels, n, K, d_counts, s));
      class_rows.resize(K + 1);
      CK(cudaMemcpyAsync(class_rows.data(), d_counts, (K + 1) * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
      CK(cudaStreamSynchronize(s));
      if (class_rows[K] != 0) class_rows.clear();
    }
  }
  if (softmax_classes) {
    // Margins [K][n] from the class priors (WeightedClassBaseScores,
    // multiclass_trainer.cpp:39-67); labels must be class ids (22-37).
    const uint32_t K = softmax_classes;
    const double total = sums.total;
    std::vector<double> cw(K, 0.0);
    for (uint32_t k = 0; k < K && !class_rows.empty(); ++k) cw[k] = double(class_rows[k]);
    for (uint64_t i = 0; i < n && class_rows.empty(); ++i) {
      const double y = labels[i];
      if (!std::isfinite(y)) throw TrainingError("softmax labels must be finite");
      if (std::floor(y) != y || y < 0.0 || y >= double(K))
        throw TrainingError("softmax labels must be encoded class ids");
      cw[uint32_t(y)] += weights ? weights[i] : 1.0;
      if (!std::isfinite(cw[uint32_t(y)])) throw TrainingError("softmax class prior overflowed");
    }
    t->base_scores.resize(K);
    for (uint32_t k = 0; k < K; ++k) {
      t->base_scores[k] = std::log(std::max(1e-15, cw[k] / total));
      if (!std::isfinite(t->base_scores[k])) throw TrainingError("softmax base score is not finite");
    }
    a.preds = t->alloc<double>(size_t(K) * n);
    for (uint32_t k = 0; k < K; ++k) CK(launch_fill_f64(a.preds + size_t(k) * n, n, t->base_scores[k], s));
  }
  trace.mark("label/weight upload");
  if (!softmax_classes) t->base_scores.resize(T);
  if (forest) {  // single-round trees: every row's prediction is the base score
    t->base_scores = forest->base_scores;
    double* d_base = t->alloc<double>(T);
    CK(cudaMemcpyAsync(d_base, t->base_scores.data(), size_t(T) * sizeof(double), cudaMemcpyHostToDevice, s));
    a.tree_base = d_base;
  }
  if (!softmax_classes && !forest) a.preds = t->alloc<double>(size_t(T) * n);
  for (uint32_t k = 0; k < T && !softmax_classes && !forest; ++k) {
    t->base_scores[k] = !class_rows.empty()
                            ? logistic_base(double(class_rows[t->ovr ? k : 1u]), sums.total)
                            : base_score(*p, labels, weights, n, t->ovr ? int64_t(k) : -1, &sums);
    CK(launch_fill_f64(a.preds + size_t(k) * n, n, t->base_scores[k], s));
  }
  trace.mark("base scores, predictions");
  if (p->n_monotonic) {
    int8_t* m = t->alloc<int8_t>(ds->features);
    CK(cudaMemcpyAsync(m, p->monotonic_constraints, ds->features, cudaMemcpyHostToDevice, s));
    a.monotonic = m;
  }
  if (p->n_interaction_groups) {
    std::vector<uint32_t> masks(size_t(p->n_interaction_groups) * W, 0);
    for (uint32_t g = 0; g < p->n_interaction_groups; ++g)
      for (uint32_t i = p->interaction_offsets[g]; i < p->interaction_offsets[g + 1]; ++i) {
        const uint32_t f = p->interaction_features[i];
        masks[size_t(g) * W + f / 32] |= 1u << (f % 32);
      }
    uint32_t* gm = t->alloc<uint32_t>(masks.size());
    CK(cudaMemcpyAsync(gm, masks.data(), masks.size() * 4, cudaMemcpyHostToDevice, s));
    CK(cudaStreamSynchronize(s));
    a.group_masks = gm;
  }
  if (forest) {
    uint32_t* d_sample = t->alloc<uint32_t>(size_t(T) * forest->cap);
    DevArena samples;  // released once the samples are written
    samples.pool = b->pool;
    uint8_t* counts = static_cast<uint8_t*>(samples.alloc(size_t(T) * n));
    uint32_t* chunk_sums = static_cast<uint32_t*>(
        samples.alloc(size_t(T) * ((n + kExpandChunk - 1) / kExpandChunk) * sizeof(uint32_t)));
    CK(cudaMemcpyAsync(counts, forest->row_counts, size_t(T) * n, cudaMemcpyHostToDevice, s));
    CK(launch_expand_samples(counts, uint32_t(n), T, chunk_sums, forest->cap, d_sample, s));
    uint32_t* d_count = t->alloc<uint32_t>(T);
    CK(cudaMemcpyAsync(d_count, forest->count.data(), size_t(T) * 4, cudaMemcpyHostToDevice, s));
    uint32_t* d_masks = t->alloc<uint32_t>(size_t(T) * W);
    CK(cudaMemcpyAsync(d_masks, forest->masks.data(), size_t(T) * W * 4, cudaMemcpyHostToDevice, s));
    if (compact) {
      uint32_t* d_of = t->alloc<uint32_t>(size_t(T) * F);
      CK(cudaMemcpyAsync(d_of, forest->feature_of.data(), size_t(T) * F * 4, cudaMemcpyHostToDevice, s));
      uint8_t* d_bins = t->alloc<uint8_t>(size_t(T) * n * a.nfb * kBlockFeatures);
      CK(launch_pack_tree_bins(ds->bins_fm.as<uint8_t>(), uint32_t(n), d_of, F, a.nfb, T, d_bins, s));
      a.feature_of = d_of;
      a.bins = d_bins;
      a.bins_row_stride = uint64_t(a.nfb) * kBlockFeatures;
      a.bins_tree_stride = uint64_t(n) * a.nfb * kBlockFeatures;
    } else {
      uint32_t* d_ranks = t->alloc<uint32_t>(size_t(T) * F);
      CK(cudaMemcpyAsync(d_ranks, forest->ranks.data(), size_t(T) * F * 4, cudaMemcpyHostToDevice, s));
      a.feature_rank = d_ranks;
    }
    a.sample_rows = d_sample;
    a.sample_count = d_count;
    a.tree_feature_masks = d_masks;
    if (!forest->seeds.empty()) {
      uint32_t* d_seeds = t->alloc<uint32_t>(T);
      CK(cudaMemcpyAsync(d_seeds, forest->seeds.data(), size_t(T) * 4, cudaMemcpyHostToDevice, s));
      a.tree_seeds = d_seeds;
    }
    a.skip_apply = 1;
    CK(cudaStreamSynchronize(s));
  }
  // working state
  a.gh = t->alloc<float2>(size_t(T) * 2 * seg_rows);
  a.gh_ordered = 1;
  a.rows = t->alloc<uint32_t>(size_t(T) * 2 * seg_rows);
  a.trees = t->alloc<TreeState>(T);
  CK(cudaMemsetAsync(a.trees, 0, size_t(T) * sizeof(TreeState), s));
  a.max_level_nodes = uint32_t(T * level_nodes);
  a.n_slots = a.max_level_nodes;
  if (t->leafwise) {
    // Active leaves <= leaves; each active leaf above max_depth keeps a histogram slot
    // from its tree's stack (slot t is the root's).
    const uint64_t max_active = p->max_active_leaves ? p->max_active_leaves : max_leaves_eff;
    a.lw_max_leaves = uint32_t(std::min<uint64_t>(max_leaves_eff, 0xFFFFFFFFull));
    a.lw_max_active = uint32_t(std::min<uint64_t>(max_active, 0xFFFFFFFFull));
    a.lw_cap = uint32_t(std::min<uint64_t>(max_active, leaves) + 2);
    a.lw_slot_cap = uint32_t(std::min<uint64_t>(max_active, leaves) + 1);
    a.n_slots = T + T * a.lw_slot_cap;
    a.max_level_nodes = std::max<uint32_t>(a.max_level_nodes, 2 * T);
    a.lw_active = t->alloc<LeafActive>(size_t(T) * a.lw_cap);
    a.lw_path = t->alloc<uint32_t>(size_t(T) * a.lw_cap * W);
    a.lw_allowed = t->alloc<uint32_t>(size_t(T) * a.lw_cap * W);
    a.lw_count = t->alloc<uint32_t>(T);
    a.lw_done = t->alloc<uint32_t>(T);
    a.lw_slots = t->alloc<uint32_t>(size_t(T) * a.lw_slot_cap);
    a.lw_slot_top = t->alloc<uint32_t>(T);
    a.lw_scan_map = t->alloc<uint32_t>(2 * size_t(T));
    t->lw_steps = uint32_t(leaves > 0 ? leaves - 1 : 0);
  }
  const uint64_t slot_words = uint64_t(F) * ds->slots * 3;
  a.hist = t->alloc<unsigned long long>(uint64_t(a.n_slots) * slot_words);
  a.free_stack = t->alloc<uint32_t>(a.n_slots);
  for (int q = 0; q < 2; ++q) {
    a.nodes[q] = t->alloc<NodeRec>(a.max_level_nodes);
    a.node_path[q] = t->alloc<uint32_t>(size_t(a.max_level_nodes) * W);
    a.node_allowed[q] = t->alloc<uint32_t>(size_t(a.max_level_nodes) * W);
  }
  a.partial = t->alloc<SplitRec>(size_t(a.max_level_nodes) * a.partial_stride);
  a.node_screen = t->alloc<uint32_t>(a.max_level_nodes);
  if (a.scan_two_phase) a.feature_screen = t->alloc<uint32_t>(size_t(a.max_level_nodes) * F);
  if (a.scan_two_phase && F > kExactFeatures) {
    a.exact_cap = a.sm_count * kScanCtasPerSm;
    a.exact_part = t->alloc<SplitRec>(a.exact_cap);
    a.exact_done = t->alloc<uint32_t>(a.exact_cap);
    CK(cudaMemsetAsync(a.exact_done, 0, a.exact_cap * sizeof(uint32_t), s));
  }
  a.build = t->alloc<BuildEntry>(a.max_level_nodes);
  a.build_prefix = t->alloc<uint32_t>(a.max_level_nodes + 1);
  a.sub = t->alloc<SubEntry>(a.max_level_nodes);
  a.part = t->alloc<PartEntry>(a.max_level_nodes);
  a.part_prefix = t->alloc<uint32_t>(a.max_level_nodes + 1);
  a.max_part_chunks = uint32_t(T * ((seg_rows + kPartChunk - 1) / kPartChunk + level_nodes + 1));
  a.part_counts = t->alloc<uint32_t>(a.max_part_chunks);
  a.part_offsets = t->alloc<uint32_t>(a.max_part_chunks);
  a.part_flags = t->alloc<uint32_t>(size_t(a.max_part_chunks) * (kPartChunk / 32));
  a.max_leafsegs = uint32_t(T * (leaves + 1));
  // Leaf chunks of 4,096 rows; a quarter of that where they would leave SMs idle.
  a.apply_chunk = uint64_t(T) * seg_rows <= (1u << 20) ? 1024u : 4096u;
  a.leafseg = t->alloc<LeafSeg>(a.max_leafsegs);
  a.leaf_prefix = t->alloc<uint32_t>(a.max_leafsegs + 1);
  if (!a.skip_apply) {
    a.leaf_of = t->alloc<uint32_t>(size_t(T) * n);
    CK(cudaMemsetAsync(a.leaf_of, 0xff, size_t(T) * n * sizeof(uint32_t), s));  // no leaf yet
    a.leaf_steps = t->alloc<double>(2 * size_t(a.max_leafsegs));
  }
  a.max_tree_nodes = uint32_t(tree_nodes);
  a.tree_nodes = t->alloc<TreeNodeOut>(size_t(T) * tree_nodes);
  a.ctl = t->alloc<Control>(1);
  CK(cudaMemsetAsync(a.ctl, 0, sizeof(Control), s));
  a.early_launch = 1;
  // Packed histogram limbs (MPSB_PACKED=0: split limbs only). A wide fixed-point cell packs
  // at most 127 rows of an item: items are kept to about 32 rows a bin.
  const char* packed = std::getenv("MPSB_PACKED");
  if (a.mode == kModeFixed && !(packed && std::atoi(packed) == 0)) {
    if (ds->slots != uint32_t(kSlots))
      a.item_rows_max = std::min<uint32_t>(kItemRowsMax, std::max<uint32_t>(4096u, 32u * ds->slots));
    t->limb_vote_words = size_t(a.nfb) * 2 * (ds->slots == uint32_t(kSlots) ? 1 : kWideVotePasses);
    const size_t votes = size_t(std::max<uint32_t>(D, 2)) * t->limb_vote_words;
    t->limb_votes = t->alloc<uint32_t>(votes);
    CK(cudaMemsetAsync(t->limb_votes, 0, votes * sizeof(uint32_t), s));
  }
  a.scratch_flags = t->alloc<uint32_t>(a.max_level_nodes);
  a.scratch_prefix = t->alloc<uint32_t>(a.max_level_nodes);
  a.scratch_aux = t->alloc<uint32_t>(a.max_level_nodes);
  a.tree_scratch = t->alloc<uint32_t>(size_t(T) * 4);
  a.max_rounds = p->n_estimators * (softmax_classes ? softmax_classes : 1);
  a.model_nodes = t->alloc<TreeNodeOut>(size_t(a.max_rounds) * T * tree_nodes);
  a.model_counts = t->alloc<uint32_t>(size_t(a.max_rounds) * T);
  a.round_counter = t->alloc<uint32_t>(1);
  CK(cudaMemsetAsync(a.round_counter, 0, sizeof(uint32_t), s));
  a.item_begin = a.item_end = 0;
  if (options & MPSB_OPT_TIMING) {
    t->events.resize(2 * std::max<uint32_t>(D, 1));
    for (auto& e : t->events) CK(cudaEventCreate(&e));
    t->level_cells = t->alloc<unsigned long long>(std::max<uint32_t>(D, 1));
  }
  CK(cudaStreamSynchronize(s));
  trace.mark("working state");
}

// A trainer's finished trees on the host: their sizes and, where all of them with the room
// between them are at most 1 MB, their nodes. One copy of 490 KB takes 20 us; 20 trees copied
// one by one take 220.
struct TreeDownload {
  uint32_t rounds = 0;
  std::vector<uint32_t> counts;          // [rounds][n_trees]
  std::vector<mpsb_tree_node> nodes;     // [rounds][n_trees][max_tree_nodes], or empty

  explicit TreeDownload(const TrainerDev& a) {
    CK(cudaMemcpy(&rounds, a.round_counter, sizeof rounds, cudaMemcpyDeviceToHost));
    counts.resize(size_t(rounds) * a.n_trees);
    if (counts.empty()) return;
    CK(cudaMemcpy(counts.data(), a.model_counts, counts.size() * 4, cudaMemcpyDeviceToHost));
    const uint64_t all = uint64_t(counts.size()) * a.max_tree_nodes;
    if (all * sizeof(mpsb_tree_node) > (1u << 20)) return;
    nodes.resize(all);
    CK(cudaMemcpy(nodes.data(), a.model_nodes, all * sizeof(mpsb_tree_node), cudaMemcpyDeviceToHost));
  }
};

mpsb_cuda_model* export_model(mpsb_cuda_trainer* t, uint32_t tree_index, const TreeDownload& down,
                              bool with_predictions = true) {
  const TrainerDev& a = t->dev;
  PhaseTrace trace("export");
  const uint32_t rounds = down.rounds;
  std::unique_ptr<mpsb_cuda_model> m(new mpsb_cuda_model);
  m->base = t->base_scores[tree_index];
  m->learning_rate = t->params.learning_rate;
  m->objective = t->params.objective;
  m->objective_alpha = t->params.objective_alpha;
  m->tweedie_variance_power = t->params.tweedie_variance_power;
  const mpsb_cuda_dataset* ds = t->ds;
  if (ds->has_schema) {  // a device-quantized dataset carries the file's schema
    m->has_schema = true;
    m->features = ds->features;
    m->max_bins = ds->max_bins;
    m->boundaries = ds->boundaries;
    m->boundary_offset = ds->boundary_offset;
    m->boundary_count = ds->boundary_count;
    m->bin_count = ds->h_bin_count;
    m->missing_count = ds->missing_count;
  }
  m->n_trees = rounds;
  m->trees.resize(rounds);
  for (uint32_t r = 0; r < rounds; ++r) {
    const size_t k = size_t(r) * a.n_trees + tree_index;
    const uint32_t c = down.counts[k];
    if (!down.nodes.empty()) {
      const mpsb_tree_node* nodes = down.nodes.data() + k * a.max_tree_nodes;
      m->trees[r].assign(nodes, nodes + c);
      continue;
    }
    m->trees[r].resize(c);
    CK(cudaMemcpy(m->trees[r].data(), a.model_nodes + k * a.max_tree_nodes, size_t(c) * sizeof(mpsb_tree_node),
                  cudaMemcpyDeviceToHost));
  }
  trace.mark("trees");
  if (with_predictions) {
    const size_t bytes = size_t(a.n_rows) * sizeof(double);
    m->device_predictions.alloc(bytes);
    m->device_prediction_count = a.n_rows;
    m->device = t->b->device;
    CK(cudaMemcpyAsync(m->device_predictions.p, a.preds + size_t(tree_index) * a.n_rows, bytes,
                       cudaMemcpyDeviceToDevice, t->b->stream));
    CK(cudaStreamSynchronize(t->b->stream));
    trace.mark("prediction copy (device)");
  }
  return m.release();
}

// A softmax model: K base scores, the trees of every (round, class) in that order, and
// the training margins [rows][K].
mpsb_cuda_model* export_softmax(mpsb_cuda_trainer* t) {
  mpsb_cuda_model* m = export_model(t, 0, TreeDownload(t->dev), false);
  const uint32_t K = t->softmax_classes;
  const TrainerDev& a = t->dev;
  m->class_count = K;
  m->base_scores = t->base_scores;
  m->base = 0.0;
  m->class_labels.resize(K);
  for (uint32_t k = 0; k < K; ++k) m->class_labels[k] = double(k);
  std::vector<double> margins(size_t(K) * a.n_rows);
  CK(cudaMemcpy(margins.data(), a.preds, margins.size() * sizeof(double), cudaMemcpyDeviceToHost));
  m->train_predictions.resize(margins.size());
  for (uint32_t k = 0; k < K; ++k)
    for (uint32_t r = 0; r < a.n_rows; ++r)
      m->train_predictions[size_t(r) * K + k] = margins[size_t(k) * a.n_rows + r];
  return m;
}

static_assert(sizeof(mpsb_tree_node) == sizeof(TreeNodeOut), "tree node layout");

}  // namespace

extern "C" {

int mpsb_cuda_trainer_create(mpsb_cuda_backend* b, const mpsb_cuda_dataset* ds,
                             const double* labels, const double* weights, uint64_t n,
                             const mpsb_train_params* p, uint32_t options,
                             mpsb_cuda_trainer** out) {
  return guard([&] {
    std::unique_ptr<mpsb_cuda_trainer> t(new mpsb_cuda_trainer);
    setup_trainer(t.get(), b, ds, labels, weights, n, p, options, 0);
    *out = t.release();
  });
}

int mpsb_cuda_trainer_run(mpsb_cuda_trainer* t, uint32_t rounds) {
  return guard([&] { t->run(rounds); });
}

int mpsb_cuda_trainer_synchronize(mpsb_cuda_trainer* t) {
  return guard([&] { t->synchronize(); });
}

int mpsb_cuda_trainer_stats(const mpsb_cuda_trainer* t, mpsb_cuda_stats* out) {
  return guard([&] { *out = t->stats; });
}

int mpsb_cuda_trainer_reset_stats(mpsb_cuda_trainer* t) {
  return guard([&] {
    t->synchronize();
    Control c;
    CK(cudaMemcpy(&c, t->dev.ctl, sizeof c, cudaMemcpyDeviceToHost));
    t->cells_base = c.cells;
    t->rows_base = c.rows_built;
    t->part_base = c.rows_partitioned;
    t->cells_before_round = c.cells;
    t->stats = mpsb_cuda_stats{};
    t->level_ms.assign(t->level_ms.size(), 0.0);
    t->level_cells_total.assign(t->level_cells_total.size(), 0);
  });
}

int mpsb_cuda_trainer_level_stats(const mpsb_cuda_trainer* t, uint32_t n_levels, double* ms,
                                  uint64_t* cells) {
  return guard([&] {
    for (uint32_t d = 0; d < n_levels; ++d) {
      ms[d] = d < t->level_ms.size() ? t->level_ms[d] : 0.0;
      cells[d] = d < t->level_cells_total.size() ? t->level_cells_total[d] : 0;
    }
  });
}

int mpsb_cuda_trainer_export(mpsb_cuda_trainer* t, mpsb_cuda_model** out) {
  return guard([&] {
    t->synchronize();
    *out = export_model(t, 0, TreeDownload(t->dev));
  });
}

void mpsb_cuda_trainer_destroy(mpsb_cuda_trainer* t) { delete t; }

int mpsb_cuda_autotune(mpsb_cuda_backend* b, const mpsb_cuda_dataset* ds, const double* labels,
                       const double* weights, uint64_t n, const mpsb_train_params* p,
                       uint32_t options, uint32_t rounds_per_trial, mpsb_cuda_tuning* out) {
  return guard([&] {
    if (!b || !ds || !labels || !p || !out) throw TrainingError("null argument");
    dataset_ready(ds);
    if (options & (MPSB_OPT_PER_NODE | MPSB_OPT_TIMING | MPSB_OPT_NO_GRAPH))
      throw UnsupportedError("the autotuner times the batched, graph-captured rounds");
    const uint32_t R = std::max(1u, rounds_per_trial);
    constexpr uint32_t kMaxTrials = 16, kConfirmTrials = 4;
    mpsb_train_params tp = *p;
    tp.n_estimators = (kMaxTrials + kConfirmTrials) * (R + 1) + 1;
    std::unique_ptr<mpsb_cuda_trainer> t(new mpsb_cuda_trainer);
    const TuneKey key = tune_key_of(ds, weights, *p, options);
    {
      // The session starts from the built-in shape, not from an earlier tuning.
      std::lock_guard<std::mutex> lock(g_tune_mutex);
      g_tune_table.erase(key);
    }
    setup_trainer(t.get(), b, ds, labels, weights, n, &tp, options, 0);
    mpsb_cuda_tuning cur{};
    cur.hist_threads = uint32_t(t->hcfg.threads);
    cur.hist_stages = uint32_t(t->hcfg.stages);
    cur.root_threads = uint32_t(t->hcfg.root_threads);
    cur.items_per_sm = t->dev.items_per_sm ? t->dev.items_per_sm : default_items_per_sm(ds->slots);
    cur.blocked_levels = t->blocked_levels;
    cur.scan_threads = t->dev.scan_threads;
    const uint32_t min_scan = t->dev.scan_threads;  // the chunk tables are sized for it
    const mpsb_cuda_tuning built_in_shape = cur;
    auto same_shape = [](const mpsb_cuda_tuning& x, const mpsb_cuda_tuning& y) {
      return x.hist_threads == y.hist_threads && x.hist_stages == y.hist_stages &&
             x.root_threads == y.root_threads && x.items_per_sm == y.items_per_sm &&
             x.blocked_levels == y.blocked_levels && x.scan_threads == y.scan_threads;
    };
    cudaEvent_t e0, e1;
    CK(cudaEventCreate(&e0));
    CK(cudaEventCreate(&e1));
    uint32_t trials = 0;
    auto measure = [&](const mpsb_cuda_tuning& s) -> double {
      t->apply_shape(s);
      t->run(1);  // captures the round graphs of this shape (and the roots' reuse)
      CK(cudaEventRecord(e0, b->stream));
      t->run(R);
      CK(cudaEventRecord(e1, b->stream));
      t->synchronize();
      float ms = 0.0f;
      CK(cudaEventElapsedTime(&ms, e0, e1));
      ++trials;
      return double(ms) / R;
    };
    try {
      double best = measure(cur);
      const double built_in = best;
      // Coordinate descent over the shape, one parameter at a time.
      auto try_values = [&](auto set, std::initializer_list<uint32_t> values) {
        for (uint32_t v : values) {
          if (trials >= kMaxTrials) return;
          mpsb_cuda_tuning cand = cur;
          if (!set(cand, v)) continue;
          const double ms = measure(cand);
          if (ms < best) {
            best = ms;
            cur = cand;
          }
        }
      };
      try_values([&](mpsb_cuda_tuning& c, uint32_t v) {
        if (v == c.hist_threads) return false;
        c.hist_threads = v;
        c.hist_stages = 2;
        return true;
      }, {768, 640, 512});
      try_values([&](mpsb_cuda_tuning& c, uint32_t v) {
        if (c.hist_threads != 512 || v == c.hist_stages) return false;
        c.hist_stages = v;
        return true;
      }, {3});
      try_values([&](mpsb_cuda_tuning& c, uint32_t v) {
        if (v == c.items_per_sm) return false;
        c.items_per_sm = v;
        return true;
      }, {1, 2, 3, 4});
      try_values([&](mpsb_cuda_tuning& c, uint32_t v) {
        if (v == c.blocked_levels) return false;
        c.blocked_levels = v;
        return true;
      }, {1, 2, 3});
      try_values([&](mpsb_cuda_tuning& c, uint32_t v) {
        // The two-launch scan's CTAs have one size.
        if (t->dev.scan_two_phase || v == c.scan_threads || v < min_scan) return false;
        c.scan_threads = v;
        return true;
      }, {128, 256});
      try_values([&](mpsb_cuda_tuning& c, uint32_t v) {
        if (v == c.root_threads) return false;
        c.root_threads = v;
        return true;
      }, {1024, 768});
      // Rounds differ a little from tree to tree: confirm the winner against the built-in
      // shape with alternating measurements before keeping it.
      mpsb_cuda_tuning chosen = cur;
      double chosen_ms = best, default_ms = built_in;
      if (!same_shape(cur, built_in_shape)) {
        double d = 0.0, c = 0.0;
        for (uint32_t i = 0; i < kConfirmTrials / 2; ++i) {
          d += measure(built_in_shape);
          c += measure(cur);
        }
        default_ms = d / (kConfirmTrials / 2);
        chosen_ms = c / (kConfirmTrials / 2);
        if (!(chosen_ms < default_ms)) {
          chosen = built_in_shape;
          chosen_ms = default_ms;
        }
      }
      cur = chosen;
      cur.ms_per_round = chosen_ms;
      cur.default_ms_per_round = default_ms;
      cur.trials = trials;
    } catch (...) {
      cudaEventDestroy(e0);
      cudaEventDestroy(e1);
      throw;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    {
      std::lock_guard<std::mutex> lock(g_tune_mutex);
      g_tune_table[key] = cur;
    }
    *out = cur;
  });
}

int mpsb_cuda_class_ids(const double* labels, uint64_t n, uint32_t limit, uint8_t* seen) {
  if (!labels || !seen) return 0;
  return class_ids(labels, n, limit, seen);
}

void mpsb_cuda_touch_pages(void* p, uint64_t bytes) {
  const uintptr_t page = uintptr_t(sysconf(_SC_PAGESIZE)), end = uintptr_t(p) + bytes;
  for (uintptr_t at = uintptr_t(p); at < end; at = (at / page + 1) * page)
    *reinterpret_cast<volatile unsigned char*>(at) = 0;
}

void mpsb_cuda_autotune_clear(void) {
  std::lock_guard<std::mutex> lock(g_tune_mutex);
  g_tune_table.clear();
}

int mpsb_cuda_train_regressor(mpsb_cuda_backend* b, const mpsb_cuda_dataset* ds,
                              const double* labels, const double* weights, uint64_t n,
                              const mpsb_train_params* p, uint32_t options,
                              mpsb_cuda_model** out) {
  return guard([&] {
    std::unique_ptr<mpsb_cuda_trainer> t(new mpsb_cuda_trainer);
    setup_trainer(t.get(), b, ds, labels, weights, n, p, options, 0);
    t->run(p->n_estimators);
    t->synchronize();
    *out = export_model(t.get(), 0, TreeDownload(t->dev));
  });
}

int mpsb_cuda_train_ovr(mpsb_cuda_backend* b, const mpsb_cuda_dataset* ds,
                        const double* labels, const double* weights, uint64_t n,
                        uint32_t n_classes, const mpsb_train_params* p, uint32_t options,
                        mpsb_cuda_model** out) {
  return guard([&] {
    if (n_classes < 2) throw TrainingError("one-vs-rest needs at least two classes");
    if (labels && !class_ids(labels, n, n_classes, nullptr)) throw TrainingError("one-vs-rest labels must be class ids in [0, n_classes)");
    std::unique_ptr<mpsb_cuda_trainer> t(new mpsb_cuda_trainer);
    setup_trainer(t.get(), b, ds, labels, weights, n, p, options, n_classes);
    t->run(p->n_estimators);
    t->synchronize();
    const TreeDownload down(t->dev);
    for (uint32_t k = 0; k < n_classes; ++k) out[k] = export_model(t.get(), k, down);
  });
}

int mpsb_cuda_train_softmax(mpsb_cuda_backend* b, const mpsb_cuda_dataset* ds,
                            const double* labels, const double* weights, uint64_t n,
                            const mpsb_train_params* p, uint32_t class_count, uint32_t options,
                            mpsb_cuda_model** out) {
  return guard([&] {
    if (!out) throw TrainingError("null argument");
    if (class_count < 2) throw TrainingError("softmax class_count must be at least two");
    std::unique_ptr<mpsb_cuda_trainer> t(new mpsb_cuda_trainer);
    setup_trainer(t.get(), b, ds, labels, weights, n, p, options, 0, nullptr, class_count);
    t->run(p->n_estimators * class_count);
    t->synchronize();
    *out = export_softmax(t.get());
  });
}

int mpsb_cuda_train_forest(mpsb_cuda_backend* b, const mpsb_cuda_dataset* ds,
                           const double* labels, const double* weights, uint64_t n,
                           const mpsb_train_params* p, uint32_t n_trees,
                           const uint8_t* row_counts, const uint32_t* feature_offsets,
                           const uint32_t* features, const uint32_t* seeds, uint32_t options,
                           mpsb_cuda_model** out) {
  return guard([&] {
    if (!b || !ds || !labels || !p || !row_counts || !feature_offsets || !features || !out)
      throw TrainingError("null argument");
    if (n_trees == 0) throw TrainingError("n_estimators must be at least 1");
    if (n != ds->n_rows) throw TrainingError("Training data, labels, or max_bins contract does not match");
    if (p->n_interaction_groups)
      throw UnsupportedError("forest training on the CUDA backend takes no interaction constraints");
    validate_training_params(*p);
    validate_tree_params(*p, ds->features);
    validate_weights(weights, n);
    const uint32_t F = ds->features;
    // Trees per trainer: the histogram slots of a tree's widest level dominate its device
    // memory, so batch as many trees as fit in half of the free memory.
    mpsb_train_params tp = *p;
    tp.n_estimators = 1;
    PhaseTrace trace("forest");
    // Sample sizes of every tree (independent trees: worker threads).
    std::vector<uint64_t> sample_size(n_trees, 0);
    parallel_trees(n_trees, [&](uint32_t t) {
      uint64_t c = 0;
      const uint8_t* m = row_counts + size_t(t) * n;
      for (uint64_t r = 0; r < n; ++r) c += m[r];
      sample_size[t] = c;
    });
    trace.mark("sample sizes");
    uint64_t cap_all = 1;
    uint32_t widest = 1;  // the largest subset
    for (uint32_t t = 0; t < n_trees; ++t) {
      const uint64_t c = sample_size[t];
      if (c == 0) throw TrainingError("a forest tree's row sample must not be empty");
      if (c >= 0x80000000ull) throw UnsupportedError("a forest tree's row sample exceeds 2^31 rows");
      cap_all = std::max(cap_all, c);
      const uint32_t f0 = feature_offsets[t], f1 = feature_offsets[t + 1];
      if (f1 <= f0) throw TrainingError("a forest tree's feature subset must not be empty");
      widest = std::max(widest, f1 - f0);
      std::vector<uint8_t> seen(F, 0);
      for (uint32_t i = f0; i < f1; ++i) {
        if (features[i] >= F) throw TrainingError("forest feature index out of range");
        if (seen[features[i]]++) throw TrainingError("forest feature subsets must not repeat a feature");
      }
    }
    const uint64_t leaves = std::min<uint64_t>(
        {uint64_t(1) << std::min<uint32_t>(p->max_depth, 30), std::max<uint64_t>(effective_max_leaves(*p), 2),
         std::max<uint64_t>(1, (cap_all + p->min_samples_leaf - 1) / p->min_samples_leaf)});
    // Trees of few features train on a copy of their own (compact) where that is at most half
    // of the dataset's: histograms, their slots and the scans then hold no other feature.
    const bool compact = ds->slots == uint32_t(kSlots) && widest * 2 <= F;
    const uint32_t FT = compact ? widest : F, W = (FT + 31) / 32;
    const uint64_t per_tree = leaves * uint64_t(FT) * ds->slots * 24 + cap_all * (2 * 12 + 4) + n +
                              (compact ? n * W * kBlockFeatures : 0) + uint64_t(2 * leaves + 1) * 64 * 8;
    size_t free_b = 0, total_b = 0;
    b->activate();
    CK(cudaMemGetInfo(&free_b, &total_b));
    free_b += b->pool->kept();
    uint64_t batch = std::max<uint64_t>(1, (free_b / 2) / std::max<uint64_t>(per_tree, 1));
    if (const char* v = std::getenv("MPSB_FOREST_BATCH")) batch = std::max(1, std::atoi(v));
    batch = std::min<uint64_t>(batch, n_trees);
    for (uint32_t t0 = 0; t0 < n_trees; t0 += uint32_t(batch)) {
      const uint32_t B = std::min<uint32_t>(uint32_t(batch), n_trees - t0);
      ForestSpec fs;
      fs.n_trees = B;
      fs.count.resize(B);
      for (uint32_t k = 0; k < B; ++k) {
        fs.count[k] = uint32_t(sample_size[t0 + k]);
        fs.cap = std::max<uint32_t>(fs.cap, fs.count[k]);
      }
      fs.row_counts = row_counts + size_t(t0) * n;
      fs.compact = compact;
      fs.features = FT;
      fs.masks.assign(size_t(B) * W, 0);
      if (compact) fs.feature_of.assign(size_t(B) * FT, 0xffffffffu);
      else fs.ranks.assign(size_t(B) * F, 0);
      fs.base_scores.resize(B);
      if (seeds) fs.seeds.assign(seeds + t0, seeds + t0 + B);
      const int mode = label_mode_of(tp.objective);
      parallel_trees(B, [&](uint32_t k) {
        const uint8_t* m = row_counts + size_t(t0 + k) * n;
        // The reference fits the tree on its sample: base score over the sample's rows in
        // order (each row as often as it was drawn).
        if (mode) {
          fs.base_scores[k] = multiset_base_score(tp, labels, weights, m, n, mode);
        } else {
          std::vector<double> ys, ws;
          ys.reserve(fs.count[k]);
          if (weights) ws.reserve(fs.count[k]);
          for (uint64_t r = 0; r < n; ++r)
            for (uint32_t c = 0; c < m[r]; ++c) {
              ys.push_back(labels[r]);
              if (weights) ws.push_back(weights[r]);
            }
          fs.base_scores[k] = base_score(tp, ys.data(), weights ? ws.data() : nullptr, ys.size(), -1);
        }
        std::vector<uint32_t> sub(features + feature_offsets[t0 + k], features + feature_offsets[t0 + k + 1]);
        std::sort(sub.begin(), sub.end());
        for (uint32_t i = 0; i < sub.size(); ++i) {  // i: position in the tree's ascending subset
          const uint32_t f = compact ? i : sub[i];
          fs.masks[size_t(k) * W + f / 32] |= 1u << (f % 32);
          if (compact) fs.feature_of[size_t(k) * FT + i] = sub[i];
          else fs.ranks[size_t(k) * F + f] = i;
        }
      });
      trace.mark("base scores, subsets");
      std::unique_ptr<mpsb_cuda_trainer> t(new mpsb_cuda_trainer);
      setup_trainer(t.get(), b, ds, labels, weights, n, &tp, options | MPSB_OPT_NO_GRAPH, 0, &fs);
      trace.mark("setup");
      t->run(1);
      t->synchronize();
      trace.mark("growth");
      const TreeDownload down(t->dev);
      for (uint32_t k = 0; k < B; ++k) out[t0 + k] = export_model(t.get(), k, down, false);
      trace.mark("export");
      t.reset();
      trace.mark("release");
    }
  });
}

int mpsb_cuda_model_create(double base, double lr, uint32_t n_trees, const uint32_t* counts,
                           const mpsb_tree_node* nodes, mpsb_cuda_model** out) {
  return guard([&] {
    if (!std::isfinite(base) || !std::isfinite(lr) || lr <= 0.0 || lr > 1.0)
      throw TrainingError("Model base score, learning rate, or tree count is invalid");
    std::unique_ptr<mpsb_cuda_model> m(new mpsb_cuda_model);
    m->base = base;
    m->learning_rate = lr;
    m->n_trees = n_trees;
    m->trees.resize(n_trees);
    size_t k = 0;
    for (uint32_t t = 0; t < n_trees; ++t) {
      if (counts[t] == 0) throw TrainingError("Tree model has no root node");
      m->trees[t].assign(nodes + k, nodes + k + counts[t]);
      k += counts[t];
    }
    *out = m.release();
  });
}

uint32_t mpsb_cuda_model_tree_count(const mpsb_cuda_model* m) { return m->n_trees; }
double mpsb_cuda_model_base_score(const mpsb_cuda_model* m) { return m->base; }
double mpsb_cuda_model_learning_rate(const mpsb_cuda_model* m) { return m->learning_rate; }
uint32_t mpsb_cuda_model_tree_node_count(const mpsb_cuda_model* m, uint32_t t) {
  return t < m->trees.size() ? uint32_t(m->trees[t].size()) : 0;
}
int mpsb_cuda_model_tree_nodes(const mpsb_cuda_model* m, uint32_t t, mpsb_tree_node* out) {
  return guard([&] {
    if (t >= m->trees.size()) throw TrainingError("tree index out of range");
    std::memcpy(out, m->trees[t].data(), m->trees[t].size() * sizeof(mpsb_tree_node));
  });
}
int mpsb_cuda_model_train_predictions(const mpsb_cuda_model* m, double* out) {
  return guard([&] {
    if (m->device_prediction_count) {
      CK(cudaSetDevice(m->device));
      CK(cudaMemcpy(out, m->device_predictions.p, m->device_prediction_count * sizeof(double),
                    cudaMemcpyDeviceToHost));
      return;
    }
    if (m->train_predictions.empty())
      throw TrainingError("this model holds no training predictions (forest tree or loaded model)");
    std::memcpy(out, m->train_predictions.data(), m->train_predictions.size() * sizeof(double));
  });
}

}  // extern "C"

namespace {

// The trees in launch_predict_packed's node format; false where one does not fit it: too
// many nodes or features, or a child that does not follow its parent (the general kernel
// then walks the trees and reports a bad index or a cycle where a row meets it).
struct HostForest {
  std::vector<uint2> nodes;
  std::vector<double> steps;
  std::vector<uint4> trees;
  std::vector<uint32_t> groups;
};

bool pack_forest(const std::vector<const std::vector<mpsb_tree_node>*>& trees, double lr,
                 const mpsb_cuda_dataset* ds, HostForest& f) {
  if (ds->features >= 32768) return false;
  f.groups.push_back(0);
  std::vector<uint32_t> ref;
  for (size_t t = 0; t < trees.size(); ++t) {
    const std::vector<mpsb_tree_node>& tree = *trees[t];
    uint32_t inner = 0, leaves = 0;
    ref.resize(tree.size());
    for (size_t i = 0; i < tree.size(); ++i) ref[i] = (tree[i].flags & 1u) ? kPackedLeaf | leaves++ : inner++;
    if (tree.empty() || inner > kPredictNodes || leaves > kPredictLeaves) return false;
    const uint4 at = make_uint4(uint32_t(f.nodes.size()), uint32_t(f.steps.size()), ref[0], 0);
    if (at.x + inner - (f.trees.empty() ? 0 : f.trees[f.groups.back()].x) > kPredictNodes ||
        at.y + leaves - (f.trees.empty() ? 0 : f.trees[f.groups.back()].y) > kPredictLeaves)
      f.groups.push_back(uint32_t(t));
    f.trees.push_back(at);
    for (size_t i = 0; i < tree.size(); ++i) {
      const mpsb_tree_node& nd = tree[i];
      if (nd.flags & 1u) {
        f.steps.push_back(lr * nd.leaf_value);
        continue;
      }
      if (nd.left_child <= i || nd.right_child <= i || nd.left_child >= tree.size() ||
          nd.right_child >= tree.size() || nd.threshold_bin > 0xFFFFu)
        return false;
      const uint32_t missing_left = ds->h_has_missing[nd.feature_index] && nd.default_left ? 1u : 0u;
      // A missing row's bin is above every threshold but the largest bin's, and goes by the
      // node's direction there too.
      if (ds->h_has_missing[nd.feature_index] && nd.threshold_bin >= ds->slots - 1) return false;
      f.nodes.push_back(make_uint2(nd.feature_index << 17 | missing_left << 16 | nd.threshold_bin,
                                   ref[nd.left_child] | ref[nd.right_child] << 16));
    }
  }
  f.groups.push_back(uint32_t(trees.size()));
  f.trees.push_back(make_uint4(uint32_t(f.nodes.size()), uint32_t(f.steps.size()), 0, 0));
  return true;
}

// base + lr * sum of the given trees' leaves for every row, on the device.
void predict_trees(mpsb_cuda_backend* b, const std::vector<const std::vector<mpsb_tree_node>*>& trees,
                   double base, double lr, const mpsb_cuda_dataset* ds, double* out) {
  dataset_ready(ds);
  std::vector<uint32_t> offsets(trees.size() + 1, 0);
  uint64_t visits = 0;  // of a row, were every tree balanced
  for (size_t t = 0; t < trees.size(); ++t) {
    offsets[t + 1] = offsets[t] + uint32_t(trees[t]->size());
    uint32_t leaves = 0;
    for (const mpsb_tree_node& nd : *trees[t]) {
      if (nd.flags & 1u) ++leaves;
      else if (nd.feature_index >= ds->features)
        throw TrainingError("Prediction feature count does not match the tree model");
    }
    while (leaves >>= 1) ++visits;
  }
  HostForest packed;
  if (!trees.empty() &&
      predict_packed_pays(ds->n_rows, ds->features, ds->slots == uint32_t(kSlots) ? 1 : 2, offsets.back(), visits) &&
      pack_forest(trees, lr, ds, packed)) {
    // One upload and one buffer: nodes, leaf steps, tree and group tables, predictions.
    const size_t nb = packed.nodes.size() * sizeof(uint2), sb = packed.steps.size() * sizeof(double),
                 tb = packed.trees.size() * sizeof(uint4), gb = packed.groups.size() * sizeof(uint32_t);
    const size_t at_s = (nb + 15) / 16 * 16, at_t = (at_s + sb + 15) / 16 * 16, at_g = at_t + tb,
                 at_out = (at_g + gb + 15) / 16 * 16;
    std::vector<unsigned char> host(at_out);
    std::memcpy(host.data(), packed.nodes.data(), nb);
    std::memcpy(host.data() + at_s, packed.steps.data(), sb);
    std::memcpy(host.data() + at_t, packed.trees.data(), tb);
    std::memcpy(host.data() + at_g, packed.groups.data(), gb);
    DevArena mem;
    mem.pool = b->pool;
    unsigned char* p = static_cast<unsigned char*>(mem.alloc(at_out + size_t(ds->n_rows) * sizeof(double)));
    double* d_out = reinterpret_cast<double*>(p + at_out);
    cudaStream_t s = b->stream;
    CK(cudaMemcpyAsync(p, host.data(), at_out, cudaMemcpyHostToDevice, s));
    const PackedForest f{reinterpret_cast<const uint2*>(p), reinterpret_cast<const double*>(p + at_s),
                         reinterpret_cast<const uint4*>(p + at_t), reinterpret_cast<const uint32_t*>(p + at_g),
                         uint32_t(packed.groups.size() - 1)};
    CK(launch_predict_packed(ds->bins_fm.as<uint8_t>(), ds->bins16_fm.as<uint16_t>(), ds->slots, ds->n_rows,
                             ds->features, f, base, d_out, s));
    CK(cudaMemcpyAsync(out, d_out, size_t(ds->n_rows) * sizeof(double), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    return;
  }
  std::vector<mpsb_tree_node> flat(offsets.back() ? offsets.back() : 1);
  for (size_t t = 0; t < trees.size(); ++t)
    std::copy(trees[t]->begin(), trees[t]->end(), flat.begin() + offsets[t]);
  DevArena mem;
  mem.pool = b->pool;
  TreeNodeOut* d_nodes = static_cast<TreeNodeOut*>(mem.alloc(flat.size() * sizeof(mpsb_tree_node)));
  uint32_t* d_off = static_cast<uint32_t*>(mem.alloc(offsets.size() * sizeof(uint32_t)));
  double* d_out = static_cast<double*>(mem.alloc(size_t(ds->n_rows) * sizeof(double)));
  cudaStream_t s = b->stream;
  CK(cudaMemcpyAsync(d_nodes, flat.data(), flat.size() * sizeof(mpsb_tree_node), cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(d_off, offsets.data(), offsets.size() * 4, cudaMemcpyHostToDevice, s));
  CK(launch_predict(ds->bins_fm.as<uint8_t>(), ds->bins16_fm.as<uint16_t>(), ds->slots, ds->n_rows,
                    ds->nfb, ds->has_missing.as<uint8_t>(),
                    d_nodes, d_off, uint32_t(trees.size()), base, lr, d_out, b->error.as<uint32_t>(), s));
  CK(cudaMemcpyAsync(out, d_out, size_t(ds->n_rows) * sizeof(double), cudaMemcpyDeviceToHost, s));
  if (b->take_error()) throw TrainingError("Tree node index is out of bounds or the structure contains a cycle");
}

}  // namespace

extern "C" {

int mpsb_cuda_model_predict(mpsb_cuda_backend* b, const mpsb_cuda_model* m,
                            const mpsb_cuda_dataset* ds, double* out) {
  return guard([&] {
    if (m->class_count) throw TrainingError("a softmax model predicts margins (mpsb_cuda_model_predict_margins)");
    b->activate();
    std::vector<const std::vector<mpsb_tree_node>*> trees;
    for (const auto& t : m->trees) trees.push_back(&t);
    predict_trees(b, trees, m->base, m->learning_rate, ds, out);
  });
}

int mpsb_cuda_model_predict_margins(mpsb_cuda_backend* b, const mpsb_cuda_model* m,
                                    const mpsb_cuda_dataset* ds, double* out) {
  return guard([&] {
    if (!m->class_count) throw TrainingError("not a softmax model");
    b->activate();
    const uint32_t K = m->class_count;
    std::vector<double> col(ds->n_rows);
    for (uint32_t k = 0; k < K; ++k) {  // class k owns trees k, k + K, ... (PredictMargins)
      std::vector<const std::vector<mpsb_tree_node>*> trees;
      for (size_t t = k; t < m->trees.size(); t += K) trees.push_back(&m->trees[t]);
      predict_trees(b, trees, m->base_scores[k], m->learning_rate, ds, col.data());
      for (uint32_t r = 0; r < ds->n_rows; ++r) out[size_t(r) * K + k] = col[r];
    }
  });
}

uint32_t mpsb_cuda_model_class_count(const mpsb_cuda_model* m) { return m->class_count; }

int mpsb_cuda_model_class_base_scores(const mpsb_cuda_model* m, double* out) {
  return guard([&] {
    if (!m->class_count) throw TrainingError("not a softmax model");
    std::copy(m->base_scores.begin(), m->base_scores.end(), out);
  });
}

int mpsb_cuda_model_class_labels(const mpsb_cuda_model* m, double* out) {
  return guard([&] {
    if (!m->class_count) throw TrainingError("not a softmax model");
    std::copy(m->class_labels.begin(), m->class_labels.end(), out);
  });
}

int mpsb_cuda_model_create_softmax(uint32_t class_count, double lr, const double* base_scores,
                                   const double* class_labels, uint32_t n_trees,
                                   const uint32_t* counts, const mpsb_tree_node* nodes,
                                   mpsb_cuda_model** out) {
  return guard([&] {
    if (class_count < 2 || n_trees == 0 || n_trees % class_count != 0 || !std::isfinite(lr) ||
        lr <= 0.0 || lr > 1.0)
      throw TrainingError("softmax model metadata is invalid");
    std::unique_ptr<mpsb_cuda_model> m(new mpsb_cuda_model);
    m->class_count = class_count;
    m->learning_rate = lr;
    m->base_scores.assign(base_scores, base_scores + class_count);
    for (double v : m->base_scores)
      if (!std::isfinite(v)) throw TrainingError("softmax model class metadata is not finite");
    m->class_labels.resize(class_count);
    for (uint32_t k = 0; k < class_count; ++k) {
      m->class_labels[k] = class_labels ? class_labels[k] : double(k);
      if (!std::isfinite(m->class_labels[k])) throw TrainingError("softmax model class metadata is not finite");
      if (k > 0 && !(m->class_labels[k - 1] < m->class_labels[k]))
        throw TrainingError("softmax model class labels must be strictly increasing");
    }
    m->n_trees = n_trees;
    m->trees.resize(n_trees);
    size_t off = 0;
    for (uint32_t t = 0; t < n_trees; ++t) {
      m->trees[t].assign(nodes + off, nodes + off + counts[t]);
      off += counts[t];
    }
    *out = m.release();
  });
}

void mpsb_cuda_model_destroy(mpsb_cuda_model* m) { delete m; }

}  // extern "C"
