// A short line's launch on two devices of one process, against a stand-in for the runtime that keeps
// the dynamic shared memory allowed for a kernel per device and refuses a launch beyond it, as CUDA
// does.  Host code: no GPU.
#include <cstdio>
#include <cuda_runtime.h>
#include <map>
#include <utility>

namespace fake {
int device = 0;
std::map<std::pair<int, const void*>, int> allowed;
template <class K> cudaError_t set(K* kernel, cudaFuncAttribute attr, int value) {
  if (attr == cudaFuncAttributeMaxDynamicSharedMemorySize) allowed[{device, (const void*)kernel}] = value;
  return cudaSuccess;
}
template <class K, class A> cudaError_t launch(const cudaLaunchConfig_t* cfg, K* kernel, const A&) {
  const auto it = allowed.find({device, (const void*)kernel});
  const size_t limit = it == allowed.end() ? 48 * 1024 : size_t(it->second);
  return cfg->dynamicSmemBytes > limit ? cudaErrorInvalidValue : cudaSuccess;
}
}  // namespace fake
#define cudaFuncSetAttribute fake::set
#define cudaLaunchKernelEx fake::launch
#include "../../hyperboliconvergence_gb300/csrc/hc_oned.cu"

using namespace hc;

template <class R> static int on(int device, int flux) {
  fake::device = device;
  if (prepare_line_run<R>(flux) != cudaSuccess) return 1;
  LineRunArgs<R> a{};
  a.nc = 100;
  a.nsteps = 1;
  const cudaError_t e = launch_line_run<R>(a, flux, nullptr);
  if (e != cudaSuccess) std::printf("device %d, flux %d: refused\n", device, flux);
  return e != cudaSuccess;
}

int main() {
  int bad = 0;
  for (int flux = 0; flux < FLUX_COUNT; ++flux)
    for (int device : {0, 1, 0, 3}) bad += on<double>(device, flux) + on<float>(device, flux);
  return bad ? 1 : 0;
}
