"""A stand-in CUDA runtime for host-side tests without a GPU: the built library runs on it in a child
process.  Memory is the host's, kernels do not run (buffers keep what the host put there, zeros
otherwise), there are two devices, every launch is noted by its kernel's name, and a launch with
more dynamic shared memory than a kernel gets unasked is refused unless the limit was raised for
that kernel on the launch's own device."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUNTIME = r"""
#include <cuda_runtime_api.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#define MAX 4096
static struct { const void *f; int dev; size_t bytes; } limit[MAX];
static int n_limit, device;
static cudaError_t last = cudaSuccess;
/* the kernels' names, as the library registers them, and those launched since test_launched() */
static struct { const void *f; const char *name; } kernel[MAX];
static int n_kernel;
static char launched[1 << 20];
static size_t n_launched;
const char *test_launched(void) {
  static char out[1 << 20];
  memcpy(out, launched, n_launched);
  out[n_launched] = 0;
  n_launched = 0;
  return out;
}
void __cudaRegisterFunction(void **h, const char *f, char *df, const char *name, int limit_, uint3 *t, uint3 *b, dim3 *bd,
                            dim3 *gd, int *w) {
  if (n_kernel < MAX) { kernel[n_kernel].f = f; kernel[n_kernel++].name = name; }
}

static int refuse_limits;  // a test's switch: the limit cannot be raised
void test_refuse_limits(int on) { refuse_limits = on; }

cudaError_t cudaGetDeviceCount(int *n) { *n = 2; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrComputeCapabilityMajor ? 10
     : a == cudaDevAttrWarpSize ? 32 : a == cudaDevAttrMaxGridDimX ? 2147483647
     : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 0;
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes *a, const void *f) {
  memset(a, 0, sizeof *a);
  a->ptxVersion = a->binaryVersion = 100;
  a->maxThreadsPerBlock = 1024;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) {
  if (refuse_limits) return last = cudaErrorInvalidValue;
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize && n_limit < MAX) {
    limit[n_limit].f = f; limit[n_limit].dev = device; limit[n_limit++].bytes = (size_t)v;
  }
  return cudaSuccess;
}
static cudaError_t launch(const void *f, size_t shared) {
  for (int k = 0; k < n_kernel; ++k)
    if (kernel[k].f == f && n_launched + strlen(kernel[k].name) + 2 < sizeof launched)
      n_launched += (size_t)sprintf(launched + n_launched, "%s\n", kernel[k].name);
  size_t room = 40960;  /* 48 KB less room for static shared memory */
  for (int k = 0; k < n_limit; ++k)
    if (limit[k].f == f && limit[k].dev == device && limit[k].bytes > room) room = limit[k].bytes;
  return shared <= room ? cudaSuccess : (last = cudaErrorInvalidValue);
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **args, size_t shared, cudaStream_t st) {
  return launch(f, shared);
}
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3 g, dim3 b, void **args, size_t shared, cudaStream_t st) {
  return launch(f, shared);
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int b, size_t s, unsigned fl) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { return (*p = calloc(n ? n : 1, 1)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t s) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t s) { free(p); return cudaSuccess; }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t s) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError(void) { return last; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "invalid argument"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { *s = (cudaStream_t)calloc(1, 1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus *c) {
  *c = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)calloc(1, 1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t e, cudaStream_t s, unsigned f) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return cudaSuccess; }
"""

PROLOGUE = r"""
import ctypes, sys
sys.path.insert(0, sys.argv[1])
runtime = ctypes.CDLL(sys.argv[2])
runtime.test_launched.restype = ctypes.c_char_p
def launched():
    "the kernels launched since the last call (mangled names)"
    return runtime.test_launched().decode().split()
"""


def run(tmp_path, program):
    """Runs the program (PROLOGUE before it) on the stand-in; returns what it printed."""
    from nuvort_b200 import api
    if not os.path.exists(api.LIB_PATH):
        pytest.skip("the CUDA library is not built")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    source, library, main = tmp_path / "runtime.c", tmp_path / "runtime.so", tmp_path / "program.py"
    source.write_text(RUNTIME)
    main.write_text(PROLOGUE + program)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-w", "-I", os.path.join(cuda, "include"), str(source), "-o", str(library)],
                   check=True)
    env = dict(os.environ, LD_PRELOAD=str(library), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, str(main), os.path.join(ROOT, "tests"), str(library)], env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
