// trainer_host.cu -- drives the trainer's host code over fake_cudart.cpp.
//   trainer_host failure <exact> <kernel> <part>
//     a batch that goes in several parts, <kernel> reporting a wait that ran
//     out in part <part> of a step; then a gradient without a failure.
//     Prints: the step's status, the parts of the gradient's batch, what its
//     table and weight gradients hold (each part adds one to their first
//     entries).
//   trainer_host memory <exact> <rays>
//     Prints the bytes of device memory that a trainer of so many rays takes
//     beyond gradient and moments of the table and the weights.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "ctx_internal.h"
#include "fake_cudart.h"

namespace nes {
bool view_ok(const nes_view&) { return true; }
}  // namespace nes

namespace {

constexpr uint32_t kTimeoutWord = 4u;  // the trainer's error word for a wait that ran out
int part = 0, failing_part = -1;
std::string failing_kernel;

}  // namespace

// Every step of every ray is occupied; a part has 1,000 records.
cudaError_t on_launch(const FakeLaunch& l) {
  uint32_t* err = nullptr;
  if (l.is("scan_kernel")) {
    uint32_t* first = l.arg<uint32_t*>(2);
    const int blocks = l.arg<int>(1);
    for (int b = 0; b <= blocks; ++b) first[b] = (uint32_t)b * 32u * 1024u;
  } else if (l.is("list_kernel")) {
    ++part;
  } else if (l.is("eval_tc_kernel")) {
    err = l.arg<uint32_t*>(6);
  } else if (l.is("adjoint_kernel")) {
    *l.arg<uint32_t*>(8) = 1000u;
    err = l.arg<uint32_t*>(9);
  } else if (l.is("backward_tc_kernel")) {
    err = l.arg<uint32_t*>(9);
  } else if (l.is("dw_tc_kernel")) {
    l.arg<float*>(3)[0] += 1.0f;
    err = l.arg<uint32_t*>(4);
  } else if (l.is("dw_kernel")) {  // strict: a launch per layer, the first layer's at the blob's start
    l.arg<float*>(3)[0] += 1.0f;
  } else if (l.is("scatter_kernel")) {
    l.arg<float2*>(5)[0].x += 1.0f;
  }
  if (err && part == failing_part && l.is(failing_kernel.c_str())) *err = kTimeoutWord;
  return cudaSuccess;
}

int main(int argc, char** argv) {
  const std::string mode = argc > 1 ? argv[1] : "";
  nes_ctx ctx;
  ctx.cfg.precision = NES_PREC_FP32;
  ctx.num_sms = 152;
  ctx.scene.T = 1u << 10;
  const size_t table_floats = (size_t)16 * ctx.scene.T * 2;
  if (cudaMalloc(reinterpret_cast<void**>(&ctx.d_table32), table_floats * sizeof(float)) != cudaSuccess ||
      cudaMalloc(reinterpret_cast<void**>(&ctx.d_weights), 65536) != cudaSuccess)
    return 2;
  nes_train_config cfg;
  nes_train_config_default(&cfg);
  nes_trainer* t = nullptr;
  if (mode == "failure" && argc == 5) {
    cfg.batch_rays = 1u << 18;
    cfg.exact_weight_grads = std::atoi(argv[2]);
    failing_kernel = argv[3];
    if (nes_trainer_create(&ctx, &cfg, &t) != NES_OK) return 3;
    nes_view view{};
    view.width = view.height = 512;
    view.focal_px = 500.0f;
    std::vector<float> target(4 * 512 * 512);
    if (nes_trainer_set_targets(t, &view, 1, target.data(), target.data()) != NES_OK) return 4;
    double loss = 0.0;
    failing_part = std::atoi(argv[4]);
    const int step = nes_trainer_step(t, 1, &loss);
    failing_part = -1;
    part = 0;
    std::vector<int32_t> pairs(2 * cfg.batch_rays);
    std::vector<float> table(table_floats), weights(65536);
    if (nes_trainer_grad(t, pairs.data(), (int)cfg.batch_rays, &loss, table.data(), weights.data()) != NES_OK)
      return 5;
    std::printf("%d %d %g %g\n", step, part, table[0], weights[0]);
    nes_trainer_destroy(t);
    return 0;
  }
  if (mode == "memory" && argc == 4) {
    cfg.exact_weight_grads = std::atoi(argv[2]);
    cfg.batch_rays = (uint32_t)std::atoi(argv[3]);
    const size_t before = fake::allocated;
    if (nes_trainer_create(&ctx, &cfg, &t) != NES_OK) return 3;
    std::printf("%zu\n", fake::allocated - before - 3 * (table_floats + nes::kWeightFloats) * sizeof(float));
    nes_trainer_destroy(t);
    return 0;
  }
  return 1;
}
