// The closing's launch functions answer with the error of a pass that could
// not be launched, whichever it is (a fake runtime fails them in turn).
#include "fake_cudart.h"
#include "gm_internal.h"

int main() {
  int failed = 0;
  // `run` with each of its launches failing in turn
  auto each = [&](const char* what, auto run) {
    fake::fail_at = -1;
    fake::launches = 0;
    cudaError_t e = run();
    const long n = fake::launches;
    if (e != cudaSuccess || n == 0) printf("%s: %d after %ld launches\n", what, (int)e, n), failed = 1;
    for (long k = 0; k < n; k++) {
      fake::launches = 0;
      fake::fail_at = k;
      if (run() == cudaSuccess) printf("%s: launch %ld of %ld failed unseen\n", what, k, n), failed = 1;
    }
  };
  uint8_t* ws = static_cast<uint8_t*>(malloc(gm::close_workspace_bytes(16)));
  for (int mode = 0; mode < 2; mode++)
    for (int se = 0; se < 2; se++)
      for (int radius : {4, 100})  // (above 91 by the unpacked passes)
        for (int field = 0; field < 2; field++) {
          gm::CloseArgs a;
          a.res = 16;
          for (int k = 0; k < 3; k++) a.data_res[k] = 16;
          a.X = a.C_out = a.workspace = ws;
          a.R = field ? reinterpret_cast<const int8_t*>(ws) : nullptr;
          a.uniform_r = a.rmax = radius;
          a.mode = mode;
          a.se = se;
          char name[64];
          snprintf(name, sizeof(name), "closing mode %d se %d radius %d field %d", mode, se, radius, field);
          each(name, [&] { return gm::launch_close(a, nullptr, nullptr); });
        }
  each("distance field", [&] { return gm::launch_edt(ws, 16, 4, ws, reinterpret_cast<uint16_t*>(ws), nullptr, nullptr); });
  free(ws);
  return failed;
}
