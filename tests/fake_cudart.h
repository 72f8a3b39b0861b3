// fake_cudart.h -- see fake_cudart.cpp: what a test program sees of it.
#pragma once
#include <cuda_runtime.h>

#include <string>

struct FakeLaunch {
  std::string name;  // mangled
  dim3 grid, block;
  size_t smem;
  int carveout;  // the kernel's preferred shared-memory carveout on the current device, or -1
  void** args;
  bool is(const char* kernel) const { return name.find(kernel) != std::string::npos; }
  template <class T>
  T arg(int i) const {
    return *static_cast<T*>(args[i]);
  }
};

// The program's: called in place of every kernel.
cudaError_t on_launch(const FakeLaunch& l);

namespace fake {
extern size_t allocated;  // bytes of the live device allocations
extern int devices;       // their number
extern int num_regs;      // registers per thread that every kernel reports
}
