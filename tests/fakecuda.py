"""The library linked a second time from the same objects, with chosen CUDA runtime calls going through fakes that can be
told to return an error: what the host code does with the error is tested without making the GPU fail.

``fake.library(tmp)`` builds and loads it; ``use(monkeypatch, lib)`` makes the package call it."""
import ctypes as C
import os
import subprocess

from mrhyde_gb300 import _lib, buildlib

SRC = r"""
#include <cuda_runtime.h>
extern "C" {
long fake_launch_at = 0;      // the launch (counted from 1 on) that is refused
long fake_launches = 0;       // cudaLaunchKernelExC calls so far
size_t fake_pool_most = ~(size_t)0;  // larger workspace requests find no memory
long fake_pool_refused = 0, fake_pool_taken = 0;
size_t fake_pool_largest = 0;  // largest request that was granted
cudaError_t __real_cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**);
cudaError_t __wrap_cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a) {
  if (++fake_launches == fake_launch_at) return cudaErrorInvalidValue;
  return __real_cudaLaunchKernelExC(c, f, a);
}
cudaError_t __real_cudaMallocFromPoolAsync(void**, size_t, cudaMemPool_t, cudaStream_t);
cudaError_t __wrap_cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t m, cudaStream_t s) {
  if (n > fake_pool_most) {
    ++fake_pool_refused;
    return cudaErrorMemoryAllocation;
  }
  ++fake_pool_taken;
  if (n > fake_pool_largest) fake_pool_largest = n;
  return __real_cudaMallocFromPoolAsync(p, n, m, s);
}
}
"""
WRAPPED = ["cudaLaunchKernelExC", "cudaMallocFromPoolAsync"]


def library(tmp):
    buildlib.build()
    objs = [os.path.join(buildlib.BUILD_DIR, os.path.basename(f)[:-3] + ".o") for f in buildlib.sources()]
    if not all(map(os.path.exists, objs)):
        buildlib.build(force=True)
    src, out = os.path.join(tmp, "fake.cu"), os.path.join(tmp, "libmrhyde_fake.so")
    with open(src, "w") as fh:
        fh.write(SRC)
    wrap = [a for w in WRAPPED for a in ("-Xlinker", f"--wrap={w}")]
    subprocess.run([buildlib._nvcc(), *buildlib.ARCH, "-shared", "-Xcompiler", "-fPIC", *wrap, "-o", out, src, *objs],
                   check=True)
    lib = C.CDLL(out)
    for name, (res, args) in _lib.SIGNATURES.items():
        getattr(lib, name).restype, getattr(lib, name).argtypes = res, args
    return lib


class Fake:
    def __init__(self, lib):
        self.lib = lib

    def __getattr__(self, name):
        kind = C.c_size_t if name in ("pool_most", "pool_largest") else C.c_long
        return kind.in_dll(self.lib, "fake_" + name)
