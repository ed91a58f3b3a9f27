// A batch whose allocations fail, one after the other, and a smaller batch
// after it: no buffer that could not be allocated is taken for an older one.
#include <vector>

#include "fake_cudart.h"
#include "gm_internal.h"

int main() {
  static uint8_t grid[16];
  auto batch = [&](int n, bool field) {
    std::vector<gm_batch_item> items(n, gm_batch_item{});
    for (auto& it : items) {
      it.desc.res = 64;
      for (int a = 0; a < 3; a++) it.desc.data_res[a] = 64;
      it.desc.cell_size = 1.f / 64;
      it.d_input = it.d_closing = grid;
      it.d_scale = field ? reinterpret_cast<const int8_t*>(grid) : nullptr;
      it.uniform_radius = 10;
    }
    return items;
  };
  int failed = 0;
  fake::read_back = 10;
  for (int lanes : {2, GM_BATCH_GROUPED})
    for (bool field : {false, true}) {
      auto run = [&](void** state, int n) {
        std::vector<gm_batch_item> items = batch(n, field);
        std::vector<gm_mesh_view> meshes(n);
        return gm::batch_run(state, n, items.data(), 0, 0, 3, lanes, meshes.data(), 152, nullptr, nullptr);
      };
      bool all_given = false;
      for (long k = 0; !all_given; k++) {  // the larger batch's k-th allocation fails
        void* state = nullptr;
        if (run(&state, 3) != cudaSuccess) printf("a batch of three failed\n"), failed = 1;
        fake::null_copies = 0;
        fake::allocs = 0;
        fake::fail_alloc_at = k;
        const cudaError_t e = run(&state, 5);
        all_given = fake::allocs <= k;
        fake::fail_alloc_at = -1;
        if ((e == cudaSuccess) != all_given) printf("allocation %ld: status %d\n", k, (int)e), failed = 1;
        if (run(&state, 2) != cudaSuccess || run(&state, 5) != cudaSuccess) printf("a batch after it failed\n"), failed = 1;
        if (fake::null_copies)
          printf("lanes %d, field %d, allocation %ld: %d copies at a null pointer\n", lanes, (int)field, k,
                 fake::null_copies), failed = 1;
        gm::batch_release(state);
      }
    }
  return failed;
}
