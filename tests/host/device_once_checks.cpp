// RtDeviceOnce (device_once.cuh) over a fake cudaGetDevice: set once on every device, again after a failure, every time beyond 64.
#include "../../rusttensor_b200/csrc/device_once.cuh"

#include <cstdio>

static int current, failures;
extern "C" cudaError_t cudaGetDevice(int* d) {
  *d = current;
  return current < 0 ? cudaErrorNoDevice : cudaSuccess;
}
#define EXPECT(x) ((x) ? (void)0 : (void)(std::printf("line %d: %s\n", __LINE__, #x), ++failures))

int main() {
  RtDeviceOnce once, other;
  int calls[80] = {};
  auto ok = [&] { return ++calls[current], cudaSuccess; };
  for (int rep = 0; rep < 2; ++rep)
    for (current = 0; current < 80; ++current) EXPECT(once(ok) == cudaSuccess);
  for (int d = 0; d < 80; ++d) EXPECT(calls[d] == (d < 64 ? 1 : 2));
  current = 3;
  EXPECT(other([] { return cudaErrorInvalidValue; }) == cudaErrorInvalidValue);
  EXPECT(other(ok) == cudaSuccess && calls[3] == 2);
  EXPECT(other(ok) == cudaSuccess && calls[3] == 2);
  current = -1;
  EXPECT(other([] { return cudaSuccess; }) == cudaErrorNoDevice);
  return failures ? 1 : 0;
}
