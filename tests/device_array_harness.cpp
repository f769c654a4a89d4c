// How fv2d_set_prim_device and fv2d_get_prim_device reach the caller's array,
// with the runtime of fake_cudart.hpp: kernels use it themselves only where it is
// binary64 words in one allocation of the context's device; everything else is
// copied through the context's staging buffer.  Exit code 0: as expected.
#include "../include/fv2d_gpu.h"
#include "fake_cudart.hpp"

constexpr int NX = 20, NY = 12;
constexpr size_t BYTES = sizeof(double) * 4 * NX * NY;

int main() {
  fv2d_params p;
  fv2d_params_default(&p);
  p.Nx = NX;
  p.Ny = NY;
  fv2d_ctx *c = nullptr;
  if (fv2d_create(&p, 0, &c) != FV2D_OK) return 2;

  static double memory[4 * NX * NY + 8];
  char *const start = reinterpret_cast<char *>(memory);
  struct Case {
    const char *name;
    cudaMemoryType type;
    int device;
    size_t offset;       // of the array in its allocation
    size_t size;         // of the allocation; 0: unknown to the driver
    cudaError_t known;   // of the pointer query
    bool in_place;
  };
  const cudaMemoryType dev = cudaMemoryTypeDevice;
  for (const Case &k : {
           Case{"own device", dev, 0, 0, BYTES, cudaSuccess, true},
           Case{"inside a larger allocation", dev, 0, 24, BYTES + 24, cudaSuccess, true},
           Case{"another device", dev, 1, 0, BYTES, cudaSuccess, false},
           Case{"managed", cudaMemoryTypeManaged, 0, 0, BYTES, cudaSuccess, false},
           Case{"page-locked host", cudaMemoryTypeHost, 0, 0, BYTES, cudaSuccess, false},
           Case{"pageable host", cudaMemoryTypeUnregistered, 0, 0, 0, cudaSuccess, false},
           Case{"query fails", dev, 0, 0, BYTES, cudaErrorInvalidValue, false},
           Case{"not a binary64 address", dev, 0, 4, BYTES + 8, cudaSuccess, false},
           Case{"one word short", dev, 0, 8, BYTES, cudaSuccess, false},
           Case{"no known allocation", dev, 0, 0, 0, cudaSuccess, false},
       }) {
    double *const q = reinterpret_cast<double *>(start + k.offset);
    fake::Runtime &r = fake::rt();
    r.attributes = [&](const void *) {
      cudaPointerAttributes a = {};
      a.type = k.type;
      a.device = k.device;
      return a;
    };
    if (k.known != cudaSuccess) r.attributes = nullptr;
    r.range = [&](CUdeviceptr *base, size_t *size, CUdeviceptr) {
      *base = reinterpret_cast<CUdeviceptr>(start);
      *size = k.size;
      return k.size ? CUDA_SUCCESS : CUDA_ERROR_NOT_FOUND;
    };
    r.launches.clear();
    r.copies.clear();
    if (fv2d_set_prim_device(c, q) != FV2D_OK) return 3;
    void *source = nullptr;
    for (const fake::Launch &l : r.launches)
      if (l.kernel.find("prepare") != std::string::npos) source = l.word;
    const fake::Copy *copy = nullptr;
    for (const fake::Copy &x : r.copies)
      if (x.src == q) copy = &x;
    const bool set_ok = k.in_place ? source == q && !copy
                                   : source && copy && copy->bytes == BYTES && copy->dst == source && source != q;
    r.copies.clear();
    r.launches.clear();
    if (fv2d_get_prim_device(c, q) != FV2D_OK) return 4;
    bool packed = false, copied = false;
    for (const fake::Launch &l : r.launches) packed |= l.kernel.find("pack") != std::string::npos;
    for (const fake::Copy &x : r.copies) copied |= x.dst == q && x.bytes == BYTES;
    if (!set_ok || !packed || copied == k.in_place || cudaGetLastError() != cudaSuccess) {
      std::printf("%s\n", k.name);
      return 1;
    }
  }
  fv2d_destroy(c);
  return 0;
}
