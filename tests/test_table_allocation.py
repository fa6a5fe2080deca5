"""Device memory that runs out while a context builds its constant tables.

Runs without a GPU: the library's process gets a stand-in for the CUDA runtime
(preloaded, host memory for device memory) that refuses the n-th allocation
and counts kernel launches.  A context must be refused whichever allocation
fails, never come up with a table missing, and give back what it had taken;
whatever is refused must also leave the next call, with memory again, intact.
The stand-in also counts launches that come after a copy from pageable host
memory (which may return early, and which other streams do not wait for) and
before a synchronisation.
"""
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
long fake_mallocs(void) { return mallocs; }
long fake_live(void) { return live; }
long fake_launches(void) { return launches; }
long fake_early(void) { return early; }
int fake_last(void) { return last; }
void fake_reset(long n) { mallocs = launches = early = 0; fail_at = n; }
static cudaError_t ok(void) { return cudaSuccess; }
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
  memmove(d, s, n);
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
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return ok(); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { return ok(); }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus *c) { *c = 0; return ok(); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { *e = (cudaEvent_t)malloc(1); return ok(); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return ok(); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return ok(); }
cudaError_t cudaGetLastError(void) { cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaFuncSetAttribute(const void *f, enum cudaFuncAttribute a, int v) { return ok(); }
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **a, size_t m, cudaStream_t s) {
  launches++;
  early += copying;
  return ok();
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **a) {
  launches++;
  early += copying;
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


def test_context_is_refused_whichever_allocation_fails(runtime):
    # three primes of digits 1 wide: every table kind of N = 2^16 and of a
    # smaller degree, over three levels and a rescale
    runtime("""
        p = json.load(open(os.path.join(chd.PARAM_DIR, "keyswitch_l8_a3.json")))
        p.update(main_primes=p["main_primes"][:3], auxiliary_primes=p["auxiliary_primes"][:1],
                 level_config=[[i, 0] for i in range(1, 4)], default_encryption_level=0)
        for log_n in (16, 12):
            text = json.dumps(dict(p, log_degree=log_n))
            rt.fake_reset(-1)
            ctx = chd.Context(text)
            total = rt.fake_mallocs()
            assert total >= 15 and rt.fake_live() == total
            ctx.close()
            assert rt.fake_live() == 0
            for n in range(total):
                rt.fake_reset(n)
                err, ctx = refused(lambda: chd.Context(text))
                assert err and "allocation" in err, (log_n, n, err)
                assert rt.fake_live() == 0 and rt.fake_last() == 0, (log_n, n)
    """)


def test_level_constants_of_the_64_bit_path(runtime):
    # built on first use: ModUp and ModDown + Rescale fail with the
    # allocation, launch nothing, and work once there is memory
    runtime("""
        p = json.load(open(os.path.join(chd.PARAM_DIR, "bootparam_40_64bit.json")))
        p.update(main_primes=p["main_primes"][:3], auxiliary_primes=p["auxiliary_primes"][:2],
                 level_config=[[i, 0] for i in range(1, 4)], default_encryption_level=0)
        src, ext = np.zeros((5, 65536), np.uint64), np.zeros((2, 5, 65536), np.uint64)
        calls = [lambda c: c.modup_raw(2, src.ctypes.data, ext.ctypes.data),
                 lambda c: c.moddown_raw(2, chd.CHD_MODDOWN_RESCALE, src.ctypes.data, ext.ctypes.data)]
        for call in calls:
            total = 1
            n = -1
            while n < total:
                rt.fake_reset(-1)
                ctx = chd.Context64(json.dumps(p))
                rt.fake_reset(n)
                err, _ = refused(lambda: call(ctx))
                if n < 0:
                    total = rt.fake_mallocs()
                    assert total >= 5 and err is None
                elif n < total:
                    assert err and "failed" in err and rt.fake_launches() == 0, (n, err)
                    rt.fake_reset(-1)
                    call(ctx)
                assert rt.fake_launches() > 0 and rt.fake_early() == 0
                del ctx
                n += 1
    """)


def test_tables_of_the_encoder(runtime):
    # built on first use; a call that had memory for one of the two tables
    # only must not leave the next one without the other
    runtime("""
        p = json.load(open(os.path.join(chd.PARAM_DIR, "keyswitch_l8_a3.json")))
        p.update(log_degree=12)
        re, im, pt, slots = np.ones(4), np.zeros(4), np.zeros((8, 4096), np.uint32), C.c_int()

        def encode(ctx):
            chd._check(chd.lib().chd_encode(ctx.ptr, 2, 2.0 ** 30, re.ctypes.data, im.ctypes.data, 4, 0, pt.ctypes.data,
                                            C.byref(slots)))

        total, n = 1, -1
        while n < total:
            rt.fake_reset(-1)
            ctx = chd.Context(json.dumps(p))
            rt.fake_reset(n)
            err, _ = refused(lambda: encode(ctx))
            if n < 0:
                total, held = rt.fake_mallocs(), rt.fake_live()
                assert total >= 3 and err is None
            elif n < total:
                assert err and "failed" in err and rt.fake_launches() == 0, (n, err)
                rt.fake_reset(-1)
                encode(ctx)
            assert rt.fake_launches() > 0 and rt.fake_early() == 0 and rt.fake_live() == held, n
            ctx.close()
            n += 1
    """)


def test_64_bit_modup_refuses_digits_of_more_than_16_primes(runtime):
    # as the 32-bit path does; the conversion holds 16 sources
    runtime("""
        p = json.load(open(os.path.join(chd.PARAM_DIR, "bootparam_40.json")))
        q = p["main_primes"]
        buf = np.zeros((2, 40, 65536), np.uint64)
        for alpha, fits in ((16, True), (17, False)):
            spec = dict(p, log_degree=16, main_primes=q[:alpha + 1], auxiliary_primes=q[20:20 + alpha], terminal_primes=[],
                        level_config=[[alpha, 0], [alpha + 1, 0]], default_encryption_level=0, additional_base=[1, 0])
            ctx = chd.Context64(json.dumps(spec))
            rt.fake_reset(-1)
            err, _ = refused(lambda: ctx.modup_raw(1, buf[0].ctypes.data, buf.ctypes.data))
            assert (err is None) == fits and (rt.fake_launches() > 0) == fits, (alpha, err)
    """)
