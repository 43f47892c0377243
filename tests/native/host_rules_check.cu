// Host checks of device.cuh's plain rules. Exit status 0 when every one holds.
#include <cstdint>
#include <cstdio>

#include "device.cuh"
#include "host_types.h"

using namespace mpsb;

// Child counts stay what they are where they add up, and are cut to the node's rows where they
// do not: never past the segment, never wrapped.
static bool children() {
  const uint64_t counts[] = {0, 1, 7, 4095, 4096, 0xFFFFFFFEull, 0xFFFFFFFFull, 1ull << 32, (1ull << 63) + 5, ~0ull};
  for (uint32_t rows : {0u, 1u, 8u, 4096u, 0xFFFFFFFFu})
    for (uint64_t l : counts)
      for (uint64_t r : counts) {
        uint64_t left = l, right = r;
        const bool want = l <= rows && r <= rows && l + r == rows;
        if (fit_children(rows, left, right) != want || left > rows || right > rows || left + right != rows ||
            (want && (left != l || right != r))) {
          std::printf("children of %u rows: %llu %llu -> %llu %llu\n", rows, (unsigned long long)l,
                      (unsigned long long)r, (unsigned long long)left, (unsigned long long)right);
          return false;
        }
      }
  return true;
}

// Fits that differ in any one property keep tuned shapes of their own: a u8 and a u16 dataset of
// the same rows, features and depth (slots), and the two kinds of split scan, among them.
static bool tune_keys() {
  constexpr int kFields = 9;
  static_assert(sizeof(TuneKey) == kFields * sizeof(uint32_t), "a field is not compared here");
  const TuneKey base{1000, 8, 6, 0, 1, 0, 0, 256, 1};
  for (int i = 0; i < kFields; ++i) {
    TuneKey other = base;
    reinterpret_cast<uint32_t*>(&other)[i] += 1;
    if (!(base < other) || other < base) {
      std::printf("tune key: field %d is not told apart\n", i);
      return false;
    }
  }
  return !(base < base);
}

// The prediction kernel's rule at the sizes it was measured at: complete trees of a depth.
static bool predict_rule() {
  struct {
    uint32_t rows, features, trees, depth;
    bool packed;
  } at[] = {{1000, 64, 1, 6, true},         {1000, 256, 1, 6, true},        {1000, 64, 64, 6, true},
            {1'000'000, 128, 1, 6, false},  {1'000'000, 128, 4, 6, false},  {1'000'000, 128, 16, 6, true},
            {1'000'000, 64, 8, 11, true},   {30'000, 64, 16, 10, false},    {30'000, 64, 64, 8, true},
            {30'000, 512, 1, 6, false},     {30'000, 512, 256, 6, true},    {300'000, 1000, 1, 6, false},
            {300'000, 1000, 256, 6, false}, {300'000, 512, 256, 6, false},  {1'000'000, 256, 1, 6, false},
            {1'000'000, 256, 64, 6, true},  {1'000'000, 2000, 256, 6, false}, {1, 1, 1, 0, true}};
  for (const auto& c : at) {
    const uint64_t entries = uint64_t(c.trees) * ((2ull << c.depth) - 1), visits = uint64_t(c.trees) * c.depth;
    if (predict_packed_pays(c.rows, c.features, 1, entries, visits) != c.packed) {
      std::printf("prediction of %u x %u by %u trees of depth %u\n", c.rows, c.features, c.trees, c.depth);
      return false;
    }
  }
  return true;
}

int main() { return children() && tune_keys() && predict_rule() ? 0 : 1; }
