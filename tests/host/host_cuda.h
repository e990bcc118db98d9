// A stand-in for the CUDA runtime on the host: device memory is host memory,
// copies happen at once, and a launch is written down instead of run.  Linked
// with the library's objects it shows what the host code asks of the GPU --
// which kernels, in which order, from which thread, with which shared memory.
#ifndef HOST_CUDA_H_
#define HOST_CUDA_H_

#include <cuda_runtime_api.h>

#include <cstddef>
#include <functional>
#include <string>
#include <thread>
#include <vector>

struct HostLaunch {
  std::string kernel;  // mangled name
  unsigned grid, block;
  size_t smem;
  void* const* args;   // valid inside on_launch only
  std::thread::id thread;
};
// every launch so far, in order
std::vector<HostLaunch> host_launches();
void host_launches_clear();
// called, outside any lock, after a launch is written down
void host_on_launch(std::function<void(const HostLaunch&)> f);

#endif
