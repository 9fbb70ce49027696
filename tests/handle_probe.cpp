// Test access to a handle's internals: the force pass and the device status word.
#include "sc_host.hpp"

extern "C" int probe_set_pass(sc_handle* H, int kind, int target, double pad) {
  sc::Handle& h = H->h;
  return h.set_pass(kind, target, std::vector<double>(h.nsys, pad)) ? 0 : h.last_status;
}

extern "C" int probe_or_status(sc_handle* H, int bits) {
  sc::Handle& h = H->h;
  int st = 0;
  if (cudaStreamSynchronize(h.stream) != cudaSuccess ||
      cudaMemcpy(&st, h.d.status, sizeof st, cudaMemcpyDeviceToHost) != cudaSuccess)
    return -1;
  st |= bits;
  return cudaMemcpy(h.d.status, &st, sizeof st, cudaMemcpyHostToDevice) == cudaSuccess ? 0 : -1;
}
