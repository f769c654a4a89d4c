// fake_cudart.hpp -- a CUDA runtime without a GPU, for host tests of the code
// that drives one: the library's objects are linked with this file instead of
// the CUDA runtime.  "Device" memory is host memory, copies and memsets run at
// once, kernels do not run at all.
//
// What it keeps is the order: every stream, and the host, has a clock; a
// stream's operation comes after everything the host had seen when it queued
// it, an event carries a stream's clock to the streams that wait for it, and a
// synchronisation carries it to the host.  Copies record the bytes they read and
// write; two that touch the same bytes, at least one of them writing, with
// nothing between them to order them, are a race (races()).  Host threads share
// one clock.  launches() holds the queued kernels with the first word of their
// first argument, attributes() sets what cudaPointerGetAttributes says.
#pragma once

#include <cuda.h>
#include <cuda_runtime_api.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>
#include <string>
#include <vector>

namespace fake {

using VectorClock = std::map<int, long>;  // per stream: its operations seen

struct Access {
  uintptr_t lo, hi;
  bool write;
  int stream;
  long when;
  std::string what;
};
struct Launch {
  std::string kernel;
  cudaStream_t stream;
  void *word;        // first word of the first argument
  bool programmatic;  // may start before the previous launch has ended
};
struct Copy {
  const void *dst, *src;
  size_t bytes;
};

struct Runtime {
  std::mutex mu;
  std::map<int, VectorClock> streams, events;
  VectorClock host;
  int next_id = 1;
  std::vector<Access> live;  // not yet known complete to the host
  std::vector<std::string> races;
  std::map<const void *, std::string> names;  // kernels by host function
  std::map<void *, size_t> device;            // allocations
  std::vector<Launch> launches;
  std::vector<Copy> copies;
  std::function<cudaPointerAttributes(const void *)> attributes;
  std::function<CUresult(CUdeviceptr *, size_t *, CUdeviceptr)> range;
  cudaError_t last = cudaSuccess;
  int sms = 152;

  static void merge(VectorClock &a, const VectorClock &b) {
    for (auto &[s, t] : b) a[s] = std::max(a[s], t);
  }
  // A new operation of stream s.
  long tick(int s) {
    merge(streams[s], host);
    return ++streams[s][s];
  }
  void access(int s, long when, const void *p, size_t n, bool write, const char *what) {
    const uintptr_t lo = reinterpret_cast<uintptr_t>(p), hi = lo + n;
    const VectorClock &seen = streams[s];
    for (const Access &x : live) {
      if (x.hi <= lo || hi <= x.lo || !(x.write || write)) continue;
      auto it = seen.find(x.stream);
      if (it == seen.end() || it->second < x.when)
        races.push_back(std::string(what) + " of stream " + std::to_string(s) + " against " + x.what + " of stream " +
                        std::to_string(x.stream) + ", " + std::to_string(n) + " bytes");
    }
    live.push_back({lo, hi, write, s, when, what});
  }
  void host_waits(const VectorClock &c) {
    merge(host, c);
    live.erase(std::remove_if(live.begin(), live.end(), [&](const Access &x) { return host[x.stream] >= x.when; }),
               live.end());
  }
};
inline Runtime &rt() {
  static Runtime *r = new Runtime;  // objects register their kernels before main
  return *r;
}
inline int id(const void *handle) { return (int)reinterpret_cast<uintptr_t>(handle); }

inline void launch(const void *fn, void **args, cudaStream_t st, bool programmatic = false) {
  std::lock_guard<std::mutex> lock(rt().mu);
  rt().tick(id(st));
  void *word = nullptr;
  if (args && args[0]) std::memcpy(&word, args[0], sizeof word);
  rt().launches.push_back({rt().names[fn], st, word, programmatic});
}
inline CUresult encode_tiled(CUtensorMap *map, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                             const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                             CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  std::memset(map, 0, sizeof *map);
  return CUDA_SUCCESS;
}
inline CUresult address_range(CUdeviceptr *base, size_t *size, CUdeviceptr p) {
  return rt().range ? rt().range(base, size, p) : CUDA_ERROR_NOT_FOUND;
}
inline cudaError_t new_handle(void **h) {
  std::lock_guard<std::mutex> lock(rt().mu);
  *h = reinterpret_cast<void *>((uintptr_t)rt().next_id++);
  return cudaSuccess;
}
inline cudaError_t allocate(void **p, size_t n, bool device) {
  *p = std::calloc(1, n + 256);  // large blocks: pages on first use
  if (!*p) return cudaErrorMemoryAllocation;
  std::lock_guard<std::mutex> lock(rt().mu);
  if (device) rt().device[*p] = n;
  return cudaSuccess;
}
inline cudaError_t deallocate(void *p) {
  {
    std::lock_guard<std::mutex> lock(rt().mu);
    for (auto &[s, c] : rt().streams) rt().host_waits(VectorClock(c));
    rt().device.erase(p);
  }
  std::free(p);
  return cudaSuccess;
}

}  // namespace fake

extern "C" {
// kernels of the objects
void **__cudaRegisterFatBinary(void *) {
  static void *handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
  fake::rt().names[host] = name;
}
static thread_local struct {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} g_config;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, CUstream_st *stream) {
  g_config = {grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
  *grid = g_config.grid;
  *block = g_config.block;
  *smem = g_config.smem;
  *static_cast<cudaStream_t *>(stream) = g_config.stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *fn) {
  *k = (cudaKernel_t) const_cast<void *>(fn);
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void **args, size_t, cudaStream_t st) {
  fake::launch((const void *)k, args, st);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *fn, dim3, dim3, void **args, size_t, cudaStream_t st) {
  fake::launch(fn, args, st);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *fn, void **args) {
  bool programmatic = false;
  for (unsigned k = 0; k < c->numAttrs; ++k)
    programmatic |= c->attrs[k].id == cudaLaunchAttributeProgrammaticStreamSerialization &&
                    c->attrs[k].val.programmaticStreamSerializationAllowed;
  fake::launch(fn, args, c->stream, programmatic);
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) {
  *n = 8;
  return cudaSuccess;
}

// device
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? fake::rt().sms : 1 << 20;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = fake::rt().last;
  fake::rt().last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetDriverEntryPointByVersion(const char *name, void **fn, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *q) {
  *fn = !std::strcmp(name, "cuTensorMapEncodeTiled") ? (void *)fake::encode_tiled
        : !std::strcmp(name, "cuMemGetAddressRange") ? (void *)fake::address_range
                                                     : nullptr;
  if (q) *q = *fn ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
  if (!fake::rt().attributes) return fake::rt().last = cudaErrorInvalidValue;
  *a = fake::rt().attributes(p);
  return cudaSuccess;
}

// memory
cudaError_t cudaMalloc(void **p, size_t n) { return fake::allocate(p, n, true); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return fake::allocate(p, n, false); }
cudaError_t cudaFree(void *p) { return fake::deallocate(p); }
cudaError_t cudaFreeHost(void *p) { return fake::deallocate(p); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }  // of zeros, on fresh memory
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  fake::Runtime &r = fake::rt();
  std::lock_guard<std::mutex> lock(r.mu);
  const long when = r.tick(fake::id(st));
  r.access(fake::id(st), when, s, n, false, "a copy's read");
  r.access(fake::id(st), when, d, n, true, "a copy's write");
  r.copies.push_back({d, s, n});
  std::memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *, size_t, const void *, size_t, size_t, size_t, cudaMemcpyKind, cudaStream_t) {
  return cudaSuccess;
}

// streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return fake::new_handle((void **)s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  std::lock_guard<std::mutex> lock(fake::rt().mu);
  fake::rt().host_waits(fake::VectorClock(fake::rt().streams[fake::id(s)]));
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  std::lock_guard<std::mutex> lock(fake::rt().mu);
  fake::rt().tick(fake::id(s));
  fake::Runtime::merge(fake::rt().streams[fake::id(s)], fake::rt().events[fake::id(e)]);
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return fake::new_handle((void **)g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *g, cudaGraph_t, unsigned long long) {
  return fake::new_handle((void **)g);
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) {
  std::lock_guard<std::mutex> lock(fake::rt().mu);
  fake::rt().tick(fake::id(s));
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return fake::new_handle((void **)e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return fake::new_handle((void **)e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  std::lock_guard<std::mutex> lock(fake::rt().mu);
  fake::rt().tick(fake::id(s));
  fake::rt().events[fake::id(e)] = fake::rt().streams[fake::id(s)];
  return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}
}
