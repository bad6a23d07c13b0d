// hc_host.h -- host-side helpers shared by the C-ABI translation units.
#pragma once

#include "../../include/hc.h"
#include "hc_launch.h"

#include <algorithm>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

namespace hc {

// last error of the calling thread (defined in hc_api.cu)
void set_last_error(const std::string& msg);

inline int fail(int code, const std::string& msg) {
  set_last_error(msg);
  return code;
}

#define HC_CUDA(call)                                                                                       \
  do {                                                                                                      \
    cudaError_t e_ = (call);                                                                                \
    if (e_ != cudaSuccess) return ::hc::fail(HC_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// Device blocks an adjoint gives back, kept by its context or batch for the next one: a
// gradient takes about 40 blocks, and allocating and freeing them took 3 ms of the 24 ms of the
// 256 x 512 drag gradient and 4 ms of the 12 ms of an eight-instance batch.  At most kKeep bytes
// wait idle in a process, whatever the number of its contexts (beyond that, and for larger runs,
// blocks go back to the driver at once); a new recording frees those of its context that it did
// not take, hc_release_idle and any allocation of the library that fails free everyone's.  A block
// is used by one context or batch, on its stream: its next user is ordered behind its last one, and
// changing the stream waits for the old one.  The lists are behind one lock, as contexts may be
// used from several threads.
struct DevicePool {
  static constexpr size_t kKeep = size_t(2) << 30;
  DevicePool() {
    std::lock_guard<std::mutex> lock(all().m);
    all().pools.push_back(this);
  }
  ~DevicePool() {
    trim();
    std::lock_guard<std::mutex> lock(all().m);
    auto& v = all().pools;
    v.erase(std::find(v.begin(), v.end(), this));
  }
  DevicePool(const DevicePool&) = delete;
  DevicePool& operator=(const DevicePool&) = delete;
  cudaError_t take(void** p, size_t bytes);
  void give(void* p, size_t bytes) {
    {
      std::lock_guard<std::mutex> lock(all().m);
      if (all().bytes + bytes <= kKeep) {
        idle.push_back({p, bytes});
        all().bytes += bytes;
        return;
      }
    }
    cudaFree(p);
  }
  void trim() {
    std::vector<Block> blocks;
    {
      std::lock_guard<std::mutex> lock(all().m);
      drain(blocks);
    }
    for (auto& b : blocks) cudaFree(b.first);
  }
  // everyone's; whether there was anything to free
  static bool trim_all() {
    std::vector<Block> blocks;
    {
      std::lock_guard<std::mutex> lock(all().m);
      for (DevicePool* p : all().pools) p->drain(blocks);
    }
    for (auto& b : blocks) cudaFree(b.first);
    return !blocks.empty();
  }
  static size_t idle_bytes() {
    std::lock_guard<std::mutex> lock(all().m);
    return all().bytes;
  }

 private:
  using Block = std::pair<void*, size_t>;
  struct All {
    std::mutex m;
    std::vector<DevicePool*> pools;
    size_t bytes = 0;
  };
  static All& all() {
    static All* a = new All;  // outlives every context, also one freed at the process's end
    return *a;
  }
  void drain(std::vector<Block>& out) {
    for (auto& b : idle) {
      all().bytes -= b.second;
      out.push_back(b);
    }
    idle.clear();
  }
  std::vector<Block> idle;
};

// device memory; where there is none left, idle blocks are given back first
template <class T> cudaError_t device_alloc(T** p, size_t bytes) {
  cudaError_t e = cudaMalloc((void**)p, bytes);
  if (e == cudaErrorMemoryAllocation && DevicePool::trim_all()) {
    (void)cudaGetLastError();
    e = cudaMalloc((void**)p, bytes);
  }
  return e;
}
inline cudaError_t DevicePool::take(void** p, size_t bytes) {
  {
    std::lock_guard<std::mutex> lock(all().m);
    for (size_t k = 0; k < idle.size(); ++k)
      if (idle[k].second == bytes) {
        *p = idle[k].first;
        idle[k] = idle.back();
        idle.pop_back();
        all().bytes -= bytes;
        return cudaSuccess;
      }
  }
  return device_alloc(p, bytes);
}

// RK tables ssp11..ssp34 (ode.h:107-197)
struct RKTab {
  int nst;
  double alpha[4][4];
  double beta[4];
};
inline RKTab rk_table(int kind) {
  RKTab t{};
  if (kind == HC_RK_SSP11) {
    t.nst = 1; t.beta[0] = 1.0; t.alpha[0][0] = 1.0;
  } else if (kind == HC_RK_SSP22) {
    t.nst = 2; t.beta[0] = 1.0; t.beta[1] = 1.0;
    t.alpha[0][0] = 1.0; t.alpha[1][0] = 0.5; t.alpha[1][1] = 0.5;
  } else if (kind == HC_RK_SSP33) {
    t.nst = 3; t.beta[0] = 1.0; t.beta[1] = 0.5; t.beta[2] = 1.0;
    t.alpha[0][0] = 1.; t.alpha[1][0] = 0.5; t.alpha[1][1] = 0.5;
    t.alpha[2][0] = 1. / 6.; t.alpha[2][1] = 1. / 6.; t.alpha[2][2] = 2. / 3.;
  } else {
    t.nst = 4; t.beta[0] = 0.5; t.beta[1] = 1.0; t.beta[2] = 0.5; t.beta[3] = 1.0;
    t.alpha[0][0] = 1.0; t.alpha[1][0] = 0.5; t.alpha[1][1] = 0.5;
    t.alpha[2][0] = 1. / 3.; t.alpha[2][1] = 1. / 3.; t.alpha[2][2] = 1. / 3.;
    t.alpha[3][0] = 1. / 6.; t.alpha[3][1] = 1. / 6.; t.alpha[3][2] = 1. / 6.; t.alpha[3][3] = 1. / 2.;
  }
  return t;
}

template <class R> using StageFn = cudaError_t (*)(const StageArgs<R>&, int, cudaStream_t);
template <class R> using BatchFn = cudaError_t (*)(const BatchArgs<R>&, int tile, int grid, cudaStream_t);

template <class R> StageFn<R> stage_fn(int flux) {
  switch (flux) {
    case FLUX_ROE: return launch_stage<R, FLUX_ROE>;
    case FLUX_SLAU: return launch_stage<R, FLUX_SLAU>;
    case FLUX_SLAU_REF: return launch_stage<R, FLUX_SLAU_REF>;
    case FLUX_AUSMPUP: return launch_stage<R, FLUX_AUSMPUP>;
    case FLUX_RUSANOV: return launch_stage<R, FLUX_RUSANOV>;
    case FLUX_ROE_WS: return launch_stage<R, FLUX_ROE_WS>;
    case FLUX_ROE_FACE: return launch_stage<R, FLUX_ROE_FACE>;
    default: return launch_stage<R, FLUX_CENTRAL>;
  }
}
template <class R> BatchFn<R> batch_fn(int flux) {
  switch (flux) {
    case FLUX_ROE: return launch_batch_stage<R, FLUX_ROE>;
    case FLUX_SLAU: return launch_batch_stage<R, FLUX_SLAU>;
    case FLUX_SLAU_REF: return launch_batch_stage<R, FLUX_SLAU_REF>;
    case FLUX_AUSMPUP: return launch_batch_stage<R, FLUX_AUSMPUP>;
    case FLUX_RUSANOV: return launch_batch_stage<R, FLUX_RUSANOV>;
    case FLUX_ROE_WS: return launch_batch_stage<R, FLUX_ROE_WS>;
    case FLUX_ROE_FACE: return launch_batch_stage<R, FLUX_ROE_FACE>;
    default: return launch_batch_stage<R, FLUX_CENTRAL>;
  }
}
template <class R> cudaError_t prepare(int flux) {
  switch (flux) {
    case FLUX_ROE: return prepare_stage<R, FLUX_ROE>();
    case FLUX_SLAU: return prepare_stage<R, FLUX_SLAU>();
    case FLUX_SLAU_REF: return prepare_stage<R, FLUX_SLAU_REF>();
    case FLUX_AUSMPUP: return prepare_stage<R, FLUX_AUSMPUP>();
    case FLUX_RUSANOV: return prepare_stage<R, FLUX_RUSANOV>();
    case FLUX_ROE_WS: return prepare_stage<R, FLUX_ROE_WS>();
    case FLUX_ROE_FACE: return prepare_stage<R, FLUX_ROE_FACE>();
    default: return prepare_stage<R, FLUX_CENTRAL>();
  }
}

// geometry of one mesh (FP64 device buffers), built by hc_api.cu's kernels
struct GeomBuffers {
  double* nodes;   // (ni+1)*(nj+1)*2
  double* cx;
  double* cy;
  double* xm;      // 3 planes
  double* vol;     // ni*nj
  double* fi;      // FREC planes of (ni+1)*nj
  double* fj;      // FREC planes of ni*(nj+1)
};
// Enqueue the geometry kernels of one mesh on `s`; returns the number of launches.
int enqueue_geometry(const GeomBuffers& g, int ni, int nj, const int bc[4], cudaStream_t s);

}  // namespace hc
