"""The library's host code against a CUDA runtime that runs nothing.

The objects of ``libshmt.so`` are linked with the runtime below instead of CUDA's: memory is host memory, copies
and fills happen at once, launches are counted and do nothing.  What kernels would write (the words a mini-batch
hands to the host) a test writes itself, a failure's status among them, so no GPU has to fail for it.
"""
import ctypes as C
import subprocess

SOURCE = r"""
#include <cuda_runtime.h>
#include <stdlib.h>
#include <string.h>
#include <map>
#include <vector>

namespace {
struct Fill { void* at; long value, bytes; };
std::map<void*, size_t> blocks;
std::vector<Fill> fills;
void* host_words;
long launches, frees;
int capturing, failing;
cudaError_t last_error = cudaSuccess;
const void* last_kernel;
}  // namespace

extern "C" {
void fake_reset() { fills.clear(); launches = frees = 0; }
long fake_launches() { return launches; }
long fake_frees() { return frees; }
void fake_capture(int on) { capturing = on; }
void fake_fail_launches(int on) { failing = on; }
int fake_last_error() { return last_error; }
const void* fake_last_kernel() { return last_kernel; }
void* fake_host_words() { return host_words; }
// fills with `value` since the reset: the largest, and how many of at least so many bytes
long fake_largest_fill(int value) {
  long most = 0;
  for (auto& f : fills)
    if (f.value == value && f.bytes > most) most = f.bytes;
  return most;
}
long fake_fills(int value, long least) {
  long n = 0;
  for (auto& f : fills) n += f.value == value && f.bytes >= least;
  return n;
}

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last_error;
  last_error = cudaSuccess;
  return e;
}
cudaError_t cudaMalloc(void** p, size_t n) { *p = aligned_alloc(256, (n + 255) / 256 * 256); blocks[*p] = n; return cudaSuccess; }
cudaError_t cudaFree(void* p) { ++frees; blocks.erase(p); free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { host_words = *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaHostRegister(void*, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaHostUnregister(void*) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { fills.push_back({p, v, (long)n}); memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemset2DAsync(void*, size_t, int, size_t, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyFromSymbol(void* d, const void*, size_t n, size_t, cudaMemcpyKind) { memset(d, 0, n); return cudaSuccess; }
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void**, const void*) { return cudaErrorNotSupported; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  memset(a, 0, sizeof(*a));
  a->type = blocks.count((void*)p) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)2; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamGetId(cudaStream_t s, unsigned long long* id) { *id = (unsigned long long)s; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  *s = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 1; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { *n = 1; return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { ++launches; return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* kernel, void**) {
  ++launches;
  last_kernel = kernel;
  if (failing) last_error = cudaErrorLaunchOutOfResources;
  return failing ? cudaErrorLaunchOutOfResources : cudaSuccess;
}
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t*, void*) { return cudaErrorNotSupported; }
cudaError_t cudaIpcOpenMemHandle(void**, cudaIpcMemHandle_t, unsigned) { return cudaErrorNotSupported; }
cudaError_t cudaIpcCloseMemHandle(void*) { return cudaErrorNotSupported; }
void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
cudaError_t __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return cudaSuccess; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
  *g = *b = dim3(1, 1, 1);
  *m = 0;
  *(cudaStream_t*)s = nullptr;
  return cudaSuccess;
}
}
"""


def load(tmp_path):
    """The library over the runtime above, with ctypes signatures."""
    from shmtensor_b200 import _lib, build
    build.build()                                # the objects, where they are older than the sources
    cuda = build.Path(build._nvcc()).resolve().parent.parent / "include"
    src, lib = tmp_path / "fake_runtime.cc", tmp_path / "libshmt_fake.so"
    src.write_text(SOURCE)
    objs = [str(build.BUILD_DIR / (build.Path(s).stem + ".o")) for s in build.SOURCES]
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", str(cuda), str(src), *objs, "-o",
                    str(lib), "-lrt", "-lpthread"], check=True)
    out = C.CDLL(str(lib))
    for name, (res, args) in _lib.SIGNATURES.items():
        fn = getattr(out, name)
        fn.restype, fn.argtypes = res, args
    for name, res, args in (("fake_launches", C.c_long, []), ("fake_frees", C.c_long, []), ("fake_reset", None, []),
                            ("fake_capture", None, [C.c_int]), ("fake_host_words", C.POINTER(C.c_int64), []),
                            ("fake_fail_launches", None, [C.c_int]), ("fake_last_error", C.c_int, []),
                            ("fake_last_kernel", C.c_void_p, []), ("fake_largest_fill", C.c_long, [C.c_int]),
                            ("fake_fills", C.c_long, [C.c_int, C.c_long])):
        fn = getattr(out, name)
        fn.restype, fn.argtypes = res, args
    return out
