// devices_host.cu -- renders on two devices of fake_cudart.cpp.  Prints, per
// device: the status of a render of an FP32 context, of a tensor-core context
// and of nes_render_view_noalloc, and the tensor-core march's shared-memory
// carveout there.
#include <cstdio>

#include "fake_cudart.h"
#include "nes_gb300.h"

namespace {
int tc_carveout = -1;
}

cudaError_t on_launch(const FakeLaunch& l) {
  if (l.is("march_tc_kernel")) tc_carveout = l.carveout;
  return cudaSuccess;
}

int main() {
  fake::devices = 2;
  fake::num_regs = 64;  // what the tensor-core march's launcher insists on
  static float rgb[16 * 16 * 3], depth[16 * 16], scene[16];
  static uint32_t occupancy[1];
  float* rgbs[1] = {rgb};
  float* depths[1] = {depth};
  nes_view view{};
  view.matrix[0] = view.matrix[5] = view.matrix[10] = 1.0f;
  view.width = view.height = 16;
  view.focal_px = 8.0f;
  for (int dev = 0; dev < 2; ++dev) {
    int rc[3] = {-1, -1, -1};
    for (int prec : {NES_PREC_FP32, NES_PREC_FP16_TC}) {
      nes_config cfg;
      nes_config_default(&cfg);
      cfg.device = dev;
      cfg.precision = prec;
      cfg.log2_table_size = 10;
      cfg.record_levels = 10;
      cfg.max_pixels = 256;
      nes_ctx* c = nullptr;
      if (nes_create(&cfg, &c) != NES_OK) return 2;
      rc[prec == NES_PREC_FP16_TC] = nes_render_views(c, &view, 1, rgbs, depths, nullptr);
      nes_destroy(c);
    }
    if (cudaSetDevice(dev) != cudaSuccess) return 3;
    rc[2] = nes_render_view_noalloc(scene, 10, scene, occupancy, &view, rgb, depth, nullptr);
    std::printf("%d %d %d %d\n", rc[0], rc[1], rc[2], tc_carveout);
    tc_carveout = -1;
  }
  return 0;
}
