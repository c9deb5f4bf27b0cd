"""An out-of-memory while the learned correction's arrays are allocated, followed by a retry: the
library runs on the host against a fake of the CUDA runtime whose cudaMalloc fails at a chosen call
(memory is host memory, kernels are not run), so nothing here touches a GPU."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#include <stdlib.h>
#include <string.h>
static int fail_in = -1, error = 0, allocated = 0;
void fake_fail_in(int calls) { fail_in = calls; }
int fake_allocated(void) { return allocated; }
int cudaMalloc(void** p, size_t n)
{
    if (fail_in >= 0 && fail_in-- == 0)
        return error = 2; /* cudaErrorMemoryAllocation; p keeps its value */
    *p = calloc(1, n);
    ++allocated;
    return 0;
}
int cudaFree(void* p) { free(p); return 0; }
int cudaHostAlloc(void** p, size_t n, unsigned f) { *p = calloc(1, n); return 0; }
int cudaFreeHost(void* p) { free(p); return 0; }
int cudaGetLastError(void) { int e = error; error = 0; return e; }
int cudaMemcpy(void* d, const void* s, size_t n, int k) { memcpy(d, s, n); return 0; }
int cudaMemcpyAsync(void* d, const void* s, size_t n, int k, void* st) { memcpy(d, s, n); return 0; }
int cudaMemset(void* d, int v, size_t n) { return 0; }
int cudaMemsetAsync(void* d, int v, size_t n, void* st) { return 0; }
int cudaLaunchKernel(const void* f, ...) { return 0; }
int cudaSetDevice(int d) { return 0; }
int cudaGetDevice(int* d) { *d = 0; return 0; }
int cudaDeviceGetAttribute(int* v, int a, int d) { *v = 148; return 0; }
int cudaFuncSetAttribute(const void* f, int a, int v) { return 0; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* b, const void* f, int t, size_t s, unsigned g) { *b = 1; return 0; }
int cudaStreamCreateWithFlags(void** s, unsigned f) { *s = calloc(1, 8); return 0; }
int cudaStreamDestroy(void* s) { free(s); return 0; }
int cudaStreamSynchronize(void* s) { return 0; }
int cudaEventCreate(void** e) { *e = calloc(1, 8); return 0; }
int cudaEventCreateWithFlags(void** e, unsigned f) { *e = calloc(1, 8); return 0; }
int cudaEventDestroy(void* e) { free(e); return 0; }
int cufftPlan3d(int* p, int a, int b, int c, int t) { *p = 1; return 0; }
int cufftSetStream(int p, void* s) { return 0; }
int cufftGetSize(int p, size_t* n) { *n = 0; return 0; }
int cufftDestroy(int p) { return 0; }
"""

PROGRAM = r"""
import ctypes, sys
import numpy as np
from blitzar_b200._lib import BZ_OUT_OF_MEMORY, BzError, Engine

fake = ctypes.CDLL(sys.argv[1])
params = np.linspace(-1, 1, Engine.MLP_PARAMS).astype(np.float32)

def engine():
    return Engine(1000, solver=1, box_length=1.0, treepm_grid_size=32, treepm_assignment=2, treepm_gradient=1)

with engine() as e:
    before = fake.fake_allocated()
    e.learn_set(params, 1.0)
    arrays = fake.fake_allocated() - before
assert arrays == 8, arrays  # five of the network, three of the pairs
for k in range(arrays):
    with engine() as e:
        before = fake.fake_allocated()
        fake.fake_fail_in(k)
        try:
            e.learn_set(params, 1.0)
            raise AssertionError(f"allocation {k} failed unnoticed")
        except BzError as x:
            assert x.status == BZ_OUT_OF_MEMORY, (k, x)
        try:
            e.learn_enable(True)
            raise AssertionError("enabled without its arrays")
        except BzError:
            pass
        e.learn_set(params, 1.0)  # memory is there again
        got = fake.fake_allocated() - before
        assert got == arrays, (k, got)
        assert np.array_equal(e.learn_get()[0], params)
        e.learn_enable(True)
print("ok")
"""


def test_retry_after_out_of_memory_allocates_every_array(tmp_path):
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        pytest.skip("no C compiler")
    src, so = tmp_path / "fake.c", tmp_path / "libfake.so"
    src.write_text(FAKE)
    subprocess.run([cc, "-shared", "-fPIC", "-O1", "-w", "-o", str(so), str(src)], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", PROGRAM, str(so)], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
