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

// whether the FP64 form has its pair results (2), its reciprocals alone (1), or neither
extern "C" int probe_extras(sc_handle* H) { return H->h.d.pr_win > 0 ? 2 : H->h.d.iaa != nullptr; }
extern "C" int probe_give_back(sc_handle* H) { return H->h.give_back() ? 0 : -1; }

// all device memory but `left` bytes; null when it cannot be had
extern "C" void* probe_fill(size_t left) {
  size_t free_bytes = 0, total = 0;
  void* p = nullptr;
  if (cudaMemGetInfo(&free_bytes, &total) != cudaSuccess || free_bytes <= left) return nullptr;
  if (cudaMalloc(&p, free_bytes - left) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return p;
}
extern "C" int probe_free(void* p) { return cudaFree(p) == cudaSuccess ? 0 : -1; }

// what is left of the handle's memory pool after probe_fill, in pieces of down to 4 KB
static std::vector<void*> g_pieces;
extern "C" int probe_exhaust(sc_handle* H) {
  sc::Handle& h = H->h;
  if (!h.use_pool) return -1;
  for (size_t n = size_t(1) << 30; n >= 4096; n /= 2)
    for (;;) {
      void* p = nullptr;
      if (cudaMallocFromPoolAsync(&p, n, sc::device_pool(h.device), h.stream) != cudaSuccess) {
        cudaGetLastError();
        break;
      }
      g_pieces.push_back(p);
    }
  return cudaStreamSynchronize(h.stream) == cudaSuccess ? (int)g_pieces.size() : -1;
}
extern "C" int probe_release(sc_handle* H) {
  for (void* p : g_pieces) cudaFreeAsync(p, H->h.stream);
  g_pieces.clear();
  return cudaStreamSynchronize(H->h.stream) == cudaSuccess ? 0 : -1;
}
