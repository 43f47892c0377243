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

int main() { return children() && tune_keys() ? 0 : 1; }
