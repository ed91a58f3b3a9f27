// A batch's captured graph is replayed only while the memory it names is the
// batch's: a batch that is captured, a larger one with a radius field (not
// captured) that moves that memory, and the first one again.
#include "fake_cudart.h"
#include "gm_internal.h"

static const int kMost = 3;  // grids

struct Batch {
  gm_batch_item items[kMost] = {};
  gm_mesh_view meshes[kMost] = {};
  int n;
  bool with_meshes;
  uint32_t occupied;  // cells per axis (and the radius bound of its fields)
  Batch(int res, bool field, bool with_meshes_, uint32_t occupied_, int n_ = 1)
      : n(n_), with_meshes(with_meshes_), occupied(occupied_) {
    static uint8_t grid[16];
    for (auto& it : items) {
      it.desc.res = res;
      for (int a = 0; a < 3; a++) it.desc.data_res[a] = res;
      it.desc.cell_size = 1.f / (float)res;
      it.d_input = it.d_closing = grid;
      it.d_scale = field ? reinterpret_cast<const int8_t*>(grid) : nullptr;
      it.uniform_radius = (int)occupied_;
    }
  }
};

static int failed = 0;

static void sequence(const char* what, int lanes, Batch first, Batch second) {
  void* state = nullptr;
  int k = 0;
  fake::stale_replays = fake::graphs = 0;
  // (the first batch twice: its second call replays)
  for (Batch* b : {&first, &first, &second, &first, &first}) {
    fake::read_back = b->occupied;
    const cudaError_t e = gm::batch_run(&state, b->n, b->items, 0, 0, b->with_meshes ? 3 : 0, lanes,
                                        b->with_meshes ? b->meshes : nullptr, 152, nullptr, nullptr);
    if (e != cudaSuccess) printf("%s: call %d: error %d\n", what, k, (int)e), failed = 1;
    if (++k == 2 && fake::graphs != 1) printf("%s: %d captures in two calls\n", what, fake::graphs), failed = 1;
  }
  if (fake::stale_replays) printf("%s: %d replays on freed memory\n", what, fake::stale_replays), failed = 1;
  if (fake::graphs > 2) printf("%s: %d captures\n", what, fake::graphs), failed = 1;
  gm::batch_release(state);
}

int main() {
  // the second batch's grids are larger, their occupied part is not
  sequence("meshes", 2, Batch(64, false, true, 10), Batch(128, true, true, 10));
  // the second batch's closings are larger: lane workspaces and crop buffers,
  // the grouped form's workspaces and its tables
  sequence("lanes", 2, Batch(64, false, false, 10), Batch(128, true, false, 40));
  sequence("lanes and meshes", 2, Batch(64, false, true, 10), Batch(64, true, true, 40));
  sequence("grouped", GM_BATCH_GROUPED, Batch(64, false, false, 10), Batch(128, true, false, 40));
  sequence("grouped, more grids", GM_BATCH_GROUPED, Batch(64, false, false, 10, 2), Batch(64, true, false, 10, 3));
  sequence("tuned", 0, Batch(64, false, false, 10), Batch(128, true, false, 40));
  return failed;
}
