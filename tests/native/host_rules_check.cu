// Host checks of device.cuh's plain rules. Exit status 0 when every one holds.
#include <cstdint>
#include <cstdio>

#include "device.cuh"

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

int main() { return children() ? 0 : 1; }
