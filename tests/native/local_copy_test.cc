// Self test of the one-rank copy: which calls go to the kernel and which to the runtime's copy.  The driver's answers about
// a pointer, the kernel's launch and the runtime's copy are fakes, so it runs without a GPU.
#include "core/enqueue.h"
#include "core/cuda_driver.h"
#include "kernels/collectives.cuh"

#include <string>

namespace uccl {
namespace {

struct World {
  unsigned type = CU_MEMORYTYPE_DEVICE, managed = 0, access = CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READWRITE;
  int device = 3;
  uintptr_t owner = 7, current = 7;  // contexts
  uintptr_t start = 0x10000;  // of the one allocation that there is
  size_t size = 4096;
  cudaError_t launch = cudaSuccess, copy = cudaSuccess;
  int launches = 0, copies = 0;
};
World world;

CUresult fakePointerGetAttributes(unsigned n, CUpointer_attribute* what, void** to, CUdeviceptr) {
  for (unsigned i = 0; i < n; ++i) {
    switch (what[i]) {
      case CU_POINTER_ATTRIBUTE_MEMORY_TYPE: *static_cast<unsigned*>(to[i]) = world.type; break;
      case CU_POINTER_ATTRIBUTE_IS_MANAGED: *static_cast<unsigned*>(to[i]) = world.managed; break;
      case CU_POINTER_ATTRIBUTE_DEVICE_ORDINAL: *static_cast<int*>(to[i]) = world.device; break;
      case CU_POINTER_ATTRIBUTE_RANGE_START_ADDR: *static_cast<CUdeviceptr*>(to[i]) = world.start; break;
      case CU_POINTER_ATTRIBUTE_RANGE_SIZE: *static_cast<size_t*>(to[i]) = world.size; break;
      case CU_POINTER_ATTRIBUTE_ACCESS_FLAGS: *static_cast<unsigned*>(to[i]) = world.access; break;
      case CU_POINTER_ATTRIBUTE_CONTEXT: *static_cast<CUcontext*>(to[i]) = reinterpret_cast<CUcontext>(world.owner); break;
      default: return CUDA_ERROR_INVALID_VALUE;
    }
  }
  return CUDA_SUCCESS;
}
CUresult fakeCtxGetCurrent(CUcontext* c) {
  *c = reinterpret_cast<CUcontext>(world.current);
  return CUDA_SUCCESS;
}
const DriverApi& fakeDriverApi() {
  static DriverApi api;
  api.ok = true;
  api.pointerGetAttributes = fakePointerGetAttributes;
  api.ctxGetCurrent = fakeCtxGetCurrent;
  return api;
}
cudaError_t fakeLaunch(const void*, void*, size_t, cudaStream_t) { return ++world.launches, world.launch; }
cudaError_t fakeMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return ++world.copies, world.copy; }

}  // namespace
}  // namespace uccl

#define driverApi fakeDriverApi
#define launchLocalCopy fakeLaunch
#define cudaMemcpyAsync fakeMemcpyAsync
#define localCopy localCopyTested
#include "core/local_copy.cc"

namespace uccl {

// "" or what is wrong
std::string testLocalCopy() {
  const char* from = reinterpret_cast<const char*>(0x10000);
  char* to = reinterpret_cast<char*>(0x10800);
  std::string wrong;
  auto expect = [&](const char* what, int launches, int copies, ucclResult_t result, auto change, int srcOff = 0, size_t bytes = 256) {
    Comm c;
    c.nRanks = 1;
    c.cudaDev = 3;
    world = World();
    change(c);
    const ucclResult_t r = localCopyTested(&c, from + srcOff, to, bytes, nullptr);
    if (r != result || world.launches != launches || world.copies != copies) wrong += std::string(what) + "; ";
  };
  expect("kernel", 1, 0, ucclSuccess, [](Comm&) {});
  expect("nothing to copy", 0, 0, ucclSuccess, [](Comm&) {}, 0, 0);
  expect("in place", 0, 0, ucclSuccess, [](Comm&) {}, 0x800);
  expect("source not aligned", 0, 1, ucclSuccess, [](Comm&) {}, 8);
  expect("beyond the allocation", 0, 1, ucclSuccess, [](Comm&) {}, 0, 4097);
  expect("destination ends beyond it", 0, 1, ucclSuccess, [](Comm&) {}, 0, 2049);
  expect("host memory", 0, 1, ucclSuccess, [](Comm&) { world.type = CU_MEMORYTYPE_HOST; });
  expect("managed memory", 0, 1, ucclSuccess, [](Comm&) { world.managed = 1; });
  expect("another GPU's memory", 0, 1, ucclSuccess, [](Comm&) { world.device = 2, world.owner = 8; });
  expect("another GPU's memory of no context", 0, 1, ucclSuccess, [](Comm&) { world.device = 2, world.owner = 0; });
  expect("another context's memory", 0, 1, ucclSuccess, [](Comm&) { world.owner = 8; });
  expect("memory of no context", 1, 0, ucclSuccess, [](Comm&) { world.owner = 0; });
  expect("read-only memory", 0, 1, ucclSuccess, [](Comm&) { world.access = CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READ; });
  expect("limited CTAs", 0, 1, ucclSuccess, [](Comm& c) { c.forcedBlocks = 2; });
  expect("limited CTAs of the configuration", 0, 1, ucclSuccess, [](Comm& c) { c.cfg.maxCtas = 2; });
  expect("copy engines", 0, 1, ucclSuccess, [](Comm& c) { c.cfg.execMode = EXEC_COPY_ENGINE; });
  // a stream of another GPU takes copies and refuses kernels
  expect("refused launch", 1, 1, ucclSuccess, [](Comm&) { world.launch = cudaErrorInvalidResourceHandle; });
  expect("both refused", 1, 1, ucclSystemError, [](Comm&) { world.launch = world.copy = cudaErrorStreamCaptureInvalidated; });
  return wrong;
}

}  // namespace uccl
