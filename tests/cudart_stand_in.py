"""A stand-in for the CUDA runtime, for tests of the library's host code on
machines without a GPU: a subprocess preloads it, device memory is host
memory, kernels do not run.  It refuses the n-th allocation, counts kernel
launches and keeps their grids, and counts launches that come after a copy
from pageable host memory (which may return early, and which other streams do
not wait for) and before a synchronisation.  On the stream that a test names as
capturing, copies are recorded only and a synchronisation fails."""
import os
import subprocess
import sys
import textwrap

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "cheddar-fhe_b200")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

RUNTIME = r'''
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>
static long mallocs, live, fail_at = -1, launches, copying, early;
static cudaError_t last;
static struct { int x, y, threads; } grids[1024];
int fake_grid(long i, int what) { return what == 0 ? grids[i].x : what == 1 ? grids[i].y : grids[i].threads; }
static void launch(dim3 g, dim3 b) {
  if (launches < 1024) grids[launches].x = g.x, grids[launches].y = g.y, grids[launches].threads = b.x;
  launches++;
  early += copying;
}
long fake_mallocs(void) { return mallocs; }
long fake_live(void) { return live; }
long fake_launches(void) { return launches; }
long fake_early(void) { return early; }
int fake_last(void) { return last; }
void fake_reset(long n) { mallocs = launches = early = 0; fail_at = n; }
static cudaError_t ok(void) { return cudaSuccess; }
static cudaStream_t capturing;
void fake_capture(void *s) { capturing = s; }
cudaError_t cudaMalloc(void **p, size_t n) {
  if (mallocs++ == fail_at) return last = cudaErrorMemoryAllocation;
  *p = calloc(1, n);
  live++;
  return ok();
}
cudaError_t cudaFree(void *p) { if (p) live--; free(p); return ok(); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) {
  memcpy(d, s, n);
  copying |= k == cudaMemcpyHostToDevice;
  return ok();
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t t) {
  if (!capturing || t != capturing) memmove(d, s, n);
  return ok();
}
cudaError_t cudaMemset(void *d, int v, size_t n) { memset(d, v, n); return ok(); }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t s) { memset(d, v, n); return ok(); }
cudaError_t cudaSetDevice(int d) { return ok(); }
cudaError_t cudaGetDevice(int *d) { *d = 0; return ok(); }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d) { *v = 148; return ok(); }
cudaError_t cudaDeviceSynchronize(void) { copying = 0; return ok(); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { *s = (cudaStream_t)malloc(1); return ok(); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return ok(); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  return capturing && s == capturing ? (last = cudaErrorStreamCaptureUnsupported) : ok();
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { return ok(); }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus *c) { *c = 0; return ok(); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { *e = (cudaEvent_t)malloc(1); return ok(); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return ok(); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return ok(); }
cudaError_t cudaGetLastError(void) { cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) { return ok(); }
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **a, size_t m, cudaStream_t s) {
  launch(g, b);
  return ok();
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **a) {
  launch(c->gridDim, c->blockDim);
  return ok();
}
'''

PRELUDE = f"""
import ctypes as C, json, os, sys
import numpy as np
sys.path.insert(0, {PKG!r})
import cheddar_b200 as chd
rt = C.CDLL(None)
for f in ("fake_mallocs", "fake_live", "fake_launches", "fake_early"):
    getattr(rt, f).restype = C.c_long
rt.fake_reset.argtypes = [C.c_long]
rt.fake_grid.argtypes = [C.c_long, C.c_int]
rt.fake_capture.argtypes = [C.c_void_p]

def refused(make):
    try:
        return None, make()
    except chd.CheddarError as e:
        return str(e), None
"""


@pytest.fixture(scope="module")
def runtime(tmp_path_factory):
    d = tmp_path_factory.mktemp("runtime")
    src, so = d / "runtime.c", d / "runtime.so"
    src.write_text(RUNTIME)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-w", f"-I{CUDA}/include", "-o", str(so), str(src)], check=True)

    def run(body):
        r = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(body)], capture_output=True, text=True,
                           timeout=600, env=dict(os.environ, LD_PRELOAD=str(so)))
        assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-3000:]

    return run
