"""Results reach the caller's arrays where page-locked memory is refused: staging.cu built against stand-ins
for the CUDA calls that it makes (copies are memcpy, page-locking fails after a set number of allocations)."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "jues.jl_gb300", "csrc")

STAND_INS = r"""
#include "staging.cuh"
#include <cstdlib>
#include <cstring>
using namespace jues;
namespace jues { void copy_out(Ctx *, double *, const double *, size_t); }
static int allocs_left = 0, locked_now = 0;
extern "C" {
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    if (allocs_left-- <= 0) return cudaErrorMemoryAllocation;
    *p = std::malloc(n);
    ++locked_now;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { std::free(p); --locked_now; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
// one context: an upload of `up` doubles (0: none) with `first` allocations granted, then a copy back of n doubles
// with `second` granted; 0, or what the library reports
int run(double *dst, const double *src, long long n, double *up_dst, long long up, int first, int second) {
    Ctx *c = static_cast<Ctx *>(std::calloc(1, sizeof(Ctx)));
    int rc = 0;
    try {
        allocs_left = first;
        if (up) staged_h2d(c, {HostSeg{up_dst, src, (size_t)up * sizeof(double)}});
        allocs_left = second;
        copy_out(c, dst, src, (size_t)n);
    } catch (const Error &e) {
        rc = e.code;
    }
    if (c->staging) staging_destroy(c->staging);
    std::free(c);
    return rc + 1000 * locked_now;
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include")
    if not shutil.which("g++") or not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("no g++ or no CUDA headers")
    d = tmp_path_factory.mktemp("staging")
    src, so = d / "stand_ins.cpp", d / "libstaging.so"
    src.write_text(STAND_INS)
    # -Bsymbolic: its own stand-ins, also where the process has loaded the CUDA runtime
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-pthread", "-I", CSRC, "-I", inc, str(src), "-x",
                    "c++", os.path.join(CSRC, "staging.cu"), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.run.argtypes = [C.c_void_p, C.c_void_p, C.c_longlong, C.c_void_p, C.c_longlong, C.c_int, C.c_int]
    return lib


# doubles: one 16 MB buffer and a little (two fills), and nine buffers' worth
@pytest.mark.parametrize("n", [(2 << 20) + 77, 18 << 20])
@pytest.mark.parametrize("up,first,second", [
    (0, 0, 0),       # no page-locked memory at all
    (0, 0, 1),       # one buffer, where two take turns
    (0, 0, 9),
    (1000, 1, 0),    # an upload's slot and no more
    (1000, 1, 1),
    (1000, 1, 9),
])
def test_results_arrive(lib, n, up, first, second):
    src, dst, updst = np.random.default_rng(n).random(n), np.zeros(n), np.zeros(max(up, 1))
    rc = lib.run(dst.ctypes.data, src.ctypes.data, n, updst.ctypes.data, up, first, second)
    assert rc == 0
    assert np.array_equal(dst, src) and np.array_equal(updst[:up], src[:up])


def test_refused_upload_slot_is_an_error(lib):
    src, dst = np.arange(1000.0), np.zeros(1000)
    assert lib.run(dst.ctypes.data, src.ctypes.data, 1000, dst.ctypes.data, 1000, 0, 0) == 3   # JUES_ECUDA
