// The collectives of a one-rank communicator and a send to oneself: a copy in stream order.
#include "../kernels/collectives.cuh"
#include "cuda_driver.h"
#include "enqueue.h"

namespace uccl {

namespace {

// Whether [p, p + bytes) is memory that a kernel of the current context may read and write: in one allocation of its own.
// Another context's memory is mapped for that one alone; the runtime's copy looks contexts up by the address.  Memory that is
// mapped by address belongs to no context, and its GPU is asked for: each attribute costs a small copy some 30 ns.
bool ownMemory(const Comm* c, CUcontext current, const void* p, size_t bytes) {
  const DriverApi& d = driverApi();
  unsigned type = 0, managed = 1, flags = 0;
  int device = -1;
  CUcontext owner = nullptr;
  CUdeviceptr start = 0;
  size_t size = 0;
  CUpointer_attribute what[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE,      CU_POINTER_ATTRIBUTE_IS_MANAGED, CU_POINTER_ATTRIBUTE_CONTEXT,
                                CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE, CU_POINTER_ATTRIBUTE_ACCESS_FLAGS};
  void* to[] = {&type, &managed, &owner, &start, &size, &flags};
  const CUdeviceptr at = reinterpret_cast<CUdeviceptr>(p);
  if (d.pointerGetAttributes(6, what, to, at) != CUDA_SUCCESS) return false;
  if (type != CU_MEMORYTYPE_DEVICE || managed != 0 || flags != CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READWRITE) return false;
  if (at < start || size < bytes || at - start > size - bytes) return false;
  if (owner != nullptr) return owner == current;
  CUpointer_attribute where[] = {CU_POINTER_ATTRIBUTE_DEVICE_ORDINAL};
  void* toDevice[] = {&device};
  return d.pointerGetAttributes(1, where, toDevice, at) == CUDA_SUCCESS && device == c->cudaDev;
}
bool ownMemory(const Comm* c, const void* src, const void* dst, size_t bytes) {
  const DriverApi& d = driverApi();
  CUcontext current = nullptr;  // of the communicator's GPU, which the caller has made current
  return d.ok && d.ctxGetCurrent(&current) == CUDA_SUCCESS && ownMemory(c, current, src, bytes) && ownMemory(c, current, dst, bytes);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

// A kernel where nothing speaks against it: it costs the host less than cudaMemcpyAsync and comes up while the launch
// before ends.  The runtime's copy takes what is not 16-byte aligned, other memory than this GPU's (which it may refuse), and
// all of it where the communicator's CTAs are limited or its data are to go by copy engines.  It also takes over when the launch
// is refused: a copy may be put into a stream of another GPU, a kernel may not.
ucclResult_t localCopy(Comm* c, const void* src, void* dst, size_t bytes, cudaStream_t s) {
  if (src == dst || bytes == 0) return ucclSuccess;
  const bool free = c->nRanks == 1 && c->forcedBlocks <= 0 && c->cfg.maxCtas <= 0 && c->cfg.execMode == EXEC_SM_ONLY;
  if (free && aligned16(src) && aligned16(dst) && ownMemory(c, src, dst, bytes) && launchLocalCopy(src, dst, bytes, s) == cudaSuccess)
    return ucclSuccess;
  if (cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, s) != cudaSuccess) {
    commSetError(c, "cudaMemcpyAsync failed: %s", cudaGetErrorString(cudaGetLastError()));
    return ucclSystemError;
  }
  return ucclSuccess;
}

}  // namespace uccl
