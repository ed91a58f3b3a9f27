// A frame field's solve whose memory cannot be had, one allocation after the
// other: it has put nothing on its stream when it fails (a next solve may come
// on another one), and the next solve is whole.
#include "fake_cudart.h"
#include "gm_internal.h"

int main() {
  int failed = 0;
  for (int res : {8, 40}) {
    const int64_t nodes[5] = {0, 5, 77, 100, 301};
    const float rhs[20] = {};
    auto solve = [&](gm::FrameFieldGpu& f, int points) {
      int rounds = 0;
      return gm::frame_field_solve(f, nodes, rhs, points, 1e-10, &rounds, nullptr, nullptr);
    };
    for (int before = 0; before < 2; before++) {  // the first solve, and one with more points
      long whole = 0;
      for (long k = -1, done = 0; !done; k++) {
        gm::FrameFieldGpu f;
        if (gm::frame_field_alloc(f, res) != cudaSuccess || (before && solve(f, 2) != cudaSuccess)) failed = 1;
        fake::allocs = fake::launches = 0;
        fake::fail_alloc_at = k;
        const cudaError_t e = solve(f, 5);
        fake::fail_alloc_at = -1;
        if (k < 0) whole = fake::launches;
        done = k >= 0 && fake::allocs <= k;
        if (e != cudaSuccess && fake::launches)
          printf("res %d, allocation %ld: failed after %ld launches\n", res, k, fake::launches), failed = 1;
        fake::launches = 0;
        if (k >= 0 && !done && (e == cudaSuccess || solve(f, 5) != cudaSuccess || fake::launches != whole))
          printf("res %d, allocation %ld: %ld launches after it, not %ld\n", res, k, fake::launches, whole), failed = 1;
        gm::frame_field_free(f);
      }
    }
  }
  return failed;
}
