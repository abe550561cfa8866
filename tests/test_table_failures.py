"""A transform plan whose tables cannot be allocated or uploaded: the failure is reported, it does not count as an axis that
the transforms do not take, and the next call plans again.  On the CPU: a host program with the library's objects and a
CUDA runtime of its own that fails on request."""
import os
import subprocess

import pytest

RUNTIME = r"""
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

int fail_malloc, fail_copy, freed;
extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
    if (fail_malloc) return cudaErrorMemoryAllocation;
    *p = malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) { free(p); ++freed; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)1; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (fail_copy) return cudaErrorUnknown;
    memcpy(d, s, n);
    return cudaSuccess;
}
}
"""

PROGRAM = r"""
#include <stdio.h>
#include <string.h>
#include "dffft.cuh"
#include "fft64.cuh"

extern int fail_malloc, fail_copy, freed;
#define EXPECT(c) if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; }

template <class Plan, class F>
int check(F &&plan, int bad_length) {
    mps::GridParams gp;
    memset(&gp, 0, sizeof(gp));
    gp.N[0] = gp.N[1] = 24;
    gp.N[2] = 30;
    Plan p;
    fail_malloc = 1;
    EXPECT(plan(gp, &p) == MPS_NO_MEMORY && !p.ok);
    fail_malloc = 0, fail_copy = 1, freed = 0;
    EXPECT(plan(gp, &p) == MPS_CUDA_ERR && !p.ok && freed == 1);
    fail_copy = 0;
    EXPECT(plan(gp, &p) == MPS_OK && p.ok && p.ax[2].N == 30 && p.ax[2].tw);
    gp.N[1] = bad_length;   // not taken: no failure
    EXPECT(plan(gp, &p) == MPS_OK && !p.ok);
    return 0;
}

int main() {
    return check<mps::F64Plan3>(mps::f64_plan, 131) || check<mps::DfPlan3>(mps::df_plan, 7);
}
"""


def test_failures_are_reported(tmp_path):
    from mutual_polarization_slab_gb300 import _build
    objects = [os.path.join(_build.BUILD, f) for f in ("common.o", "fft64.o", "dffft.o")]
    if not all(map(os.path.exists, objects)) or _build.is_stale():
        pytest.skip("the library has not been built here")
    src, runtime, exe = tmp_path / "plans.cu", tmp_path / "runtime.cpp", tmp_path / "plans"
    src.write_text(PROGRAM)
    runtime.write_text(RUNTIME)
    subprocess.run([_build.nvcc_path(), *_build.ARCH, *_build.NVCC_FLAGS, "-I", _build.CSRC, "-o", str(exe), str(src),
                    str(runtime), *objects, "-cudart", "shared"], check=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
