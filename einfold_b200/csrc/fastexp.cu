// The tables of exp_tang and exp_scaled, one per device.
#include <cmath>
#include <mutex>
#include <vector>

#include "common.h"
#include "fastexp.cuh"

namespace ef {

namespace {

constexpr int kDevices = 64;

// The table that fill() gives, made and copied to the current device once per
// device: a call that finds it there only looks it up.
template <class Fill>
const double* table_on(int device, std::once_flag* once, double** tables, Fill&& fill) {
  if (device < 0 || device >= kDevices) fail(EINFOLD_INVALID, "device %d out of range", device);
  std::call_once(once[device], [&] {
    const std::vector<double> host = fill();
    double* dev = nullptr;
    EF_CUDA(cudaMalloc(&dev, host.size() * sizeof(double)));
    EF_CUDA(cudaMemcpy(dev, host.data(), host.size() * sizeof(double), cudaMemcpyHostToDevice));
    tables[device] = dev;
  });
  if (!tables[device]) fail(EINFOLD_DEVICE, "the exp table of device %d could not be set up", device);
  return tables[device];
}

}  // namespace

const double* exp_table(int device) {
  static std::once_flag once[kDevices];
  static double* tables[kDevices] = {};
  return table_on(device, once, tables, [] {
    std::vector<double> host(64);
    for (int j = 0; j < 64; j++) host[j] = (double)std::exp2l((long double)j / 64.0L);
    return host;
  });
}

const double2* exp_scaled_table(int device) {
  static std::once_flag once[kDevices];
  static double* tables[kDevices] = {};
  return reinterpret_cast<const double2*>(table_on(device, once, tables, [] {
    std::vector<double> host(2 * kExpScaledEntries);
    for (int j = 0; j < kExpScaledEntries; j++) {
      const long double x = std::exp2l((long double)j / kExpScaledEntries);
      host[2 * j] = (double)x;
      host[2 * j + 1] = (double)(x - (long double)host[2 * j]);
    }
    return host;
  }));
}

}  // namespace ef
