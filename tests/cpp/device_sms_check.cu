// device_sms() with a thread that moves between devices, against a stand-in for the runtime's two
// queries.  Host code: no GPU.
#include <cuda_runtime.h>

namespace fake {
int device = 0, asked = 0;
inline cudaError_t get_device(int* d) {
  *d = device;
  return device < 0 ? cudaErrorNoDevice : cudaSuccess;
}
inline cudaError_t get_attribute(int* v, cudaDeviceAttr, int d) {
  ++asked;
  *v = 100 + d;
  return cudaSuccess;
}
}  // namespace fake
#define cudaGetDevice fake::get_device
#define cudaDeviceGetAttribute fake::get_attribute
#include "../../hyperboliconvergence_gb300/csrc/hc_launch.h"

int main() {
  int bad = 0;
  for (int pass = 0; pass < 3; ++pass)
    for (int d : {0, 1, 5, 0, 70, 1}) {
      fake::device = d;
      if (hc::device_sms() != 100 + d) ++bad;
    }
  if (fake::asked > 3 + 3) ++bad;  // once per device, except past the table
  fake::device = -1;
  if (hc::device_sms() != 152) ++bad;
  return bad ? 1 : 0;
}
