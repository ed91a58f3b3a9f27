// An error that an earlier CUDA call of the program's own has left unread is not
// the library's: the calls after it do their work and answer for themselves.
#include <functional>

#include "fake_cudart.h"
#include "gm_internal.h"

int main() {
  int failed = 0;
  alignas(16) static uint8_t buffer[64];
  gm_grid_desc d = {};
  d.res = 64;
  d.cell_size = 1.f / 64;
  for (int a = 0; a < 3; a++) d.data_res[a] = 64, d.bbox_max[a] = 1.f;
  gm_box_desc b = {};
  b.cell_size = 1.f;
  for (int a = 0; a < 3; a++) b.dims[a] = b.data_res[a] = 32;
  fake::read_back = 10;
  gm_ctx* ctx = nullptr;
  if (gm_ctx_create(0, &ctx) != GM_OK) return 1;
  const int8_t* R = reinterpret_cast<const int8_t*>(buffer);
  gm_frame_field* ff = nullptr;
  const float lo[3] = {0, 0, 0}, hi[3] = {1, 1, 1}, at[3] = {.5f, .5f, .5f}, twist[3] = {0, 0, 1};
  if (gm_frame_field_create(ctx, lo, hi, 8, &ff) != GM_OK || gm_frame_field_add_point(ff, at, twist) != GM_OK) return 1;
  gm_server_opts opts = {};
  opts.slots = 1;
  opts.max_crop_res = 64;
  opts.rmax = 12;
  gm_server* srv = nullptr;
  static uint8_t grid[8 * 64 * 64 * 64];
  static int8_t scale[8 * 64 * 64 * 64];  // the server's field
  gm_mesh_view mesh;
  gm_batch_item item = {d, buffer, nullptr, 4, buffer};
  gm_edit edit = {};
  for (int a = 0; a < 3; a++) edit.center[a] = .5f;
  edit.scale = edit.support = 4.f / 128;
  edit.mode = GM_BRUSH_MAX;
  gm_edit_result done[4];
  int32_t count = 0;
  const struct {
    const char* name;
    std::function<int()> call;
  } calls[] = {
      {"gm_close", [&] { return gm_close(ctx, &d, buffer, nullptr, 4, GM_REF, GM_SE_SPHERE, buffer, nullptr, nullptr, nullptr); }},
      {"gm_close, field", [&] { return gm_close(ctx, &d, buffer, R, 0, GM_REF, GM_SE_CUBE, buffer, nullptr, nullptr, nullptr); }},
      {"gm_close_noalloc", [&] { return gm_close_noalloc(&d, buffer, nullptr, 4, GM_REF, GM_SE_SPHERE, buffer, nullptr, nullptr, nullptr); }},
      {"gm_close_box", [&] { return gm_close_box(ctx, &b, buffer, R, 0, GM_EXACT, GM_SE_SPHERE, buffer, nullptr); }},
      {"gm_mesh", [&] { return gm_mesh(ctx, &d, buffer, 3, &mesh, nullptr); }},
      {"gm_batch_close_mesh", [&] { return gm_batch_close_mesh(ctx, 1, &item, GM_REF, GM_SE_SPHERE, 3, 2, &mesh, nullptr); }},
      {"gm_frame_field_generate", [&] { return gm_frame_field_generate(ff, nullptr, nullptr); }},
      {"gm_server_create", [&] {
         if (srv) gm_server_destroy(srv);
         return gm_server_create(&d, buffer, scale, &opts, &srv);
       }},
      {"gm_server_submit", [&] { return gm_server_submit(srv, &edit, nullptr); }},
      {"gm_server_poll", [&] {
         const int s = gm_server_poll(srv, done, 4, &count);
         for (int i = 0; i < count; i++)
           if (done[i].status != GM_OK) return (int)done[i].status;
         return s;
       }},
      {"gm_server_restore", [&] { return gm_server_restore(srv, grid, reinterpret_cast<int8_t*>(grid)); }},
  };
  for (const auto& c : calls)
    for (int stale = 0; stale < 2; stale++) {
      c.call();  // (buffers and captures of a first call)
      fake::launches = 0;
      fake::last = stale ? cudaErrorInvalidDevice : cudaSuccess;
      const int s = c.call();
      static long whole;
      if (!stale) whole = fake::launches;
      if (s != GM_OK || fake::launches != whole)
        printf("%s: status %d, %ld of %ld launches\n", c.name, s, fake::launches, whole), failed = 1;
      fake::last = cudaSuccess;
    }
  return failed;
}
