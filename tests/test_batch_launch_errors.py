"""A batch step that a launch error cuts short, on the CPU: the batch's object
code linked against a stand-in for the CUDA runtime that records the calls made
to it, runs nothing, and fails one launch on request."""
import ctypes as C
import importlib
import os
import subprocess

import pytest

from conftest import ROOT, dg

FAKE = r"""
#include <cuda_runtime_api.h>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include "solver_internal.h"

namespace dg {
int fail(int code, const std::string&) { return code; }
}

static std::string calls;
static std::map<const void*, std::string> names;
static int fail_in = 0;       // fails the n-th launch from here
static cudaError_t last = cudaSuccess;
static unsigned long long handles = 1;

static cudaError_t launch(const void* fun)
{
    const std::string& n = names[fun];
    calls += (n.find("batch_stage_kernel") != std::string::npos  ? "stage "
              : n.find("batch_step_end") != std::string::npos    ? "end "
                                                                  : "other ");
    if (fail_in && --fail_in == 0) return last = cudaErrorLaunchOutOfResources;
    return cudaSuccess;
}

extern "C" {
const char* fake_calls() { return calls.c_str(); }
void fake_reset(int n) { calls.clear(); fail_in = n; }

void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*)
{
    names[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* fun) { *k = (cudaKernel_t)fun; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t, cudaStream_t) { return launch((const void*)k); }
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t) { return launch(f); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* f, void**) { return launch(f); }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "stand-in"; }

cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int)
{
    std::memset(p, 0, sizeof *p);
    p->multiProcessorCount = 2;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned)
{
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)(handles++); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { calls += "sync "; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
// no capture: the step is launched directly
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = nullptr; return cudaErrorStreamCaptureUnsupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t, cudaGraph_t, cudaGraphExecUpdateResultInfo*) { return cudaErrorUnknown; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorUnknown; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)(handles++); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)(handles++); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) { *t = 1; return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = (cudaMemPool_t)(handles++); return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t)
{
    *p = std::calloc(n, 1);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t)
{
    calls += "zero ";
    std::memset(d, v, n);
    return cudaSuccess;
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    build = importlib.import_module("3ddg_gb300.build")
    objs = [os.path.join(build.OBJ, n + ".o") for n in ("batch.cu", "basis.cpp", "mesh.cpp", "params.cpp")]
    if not all(os.path.exists(o) for o in objs):
        pytest.skip("no object files of the build")
    d = tmp_path_factory.mktemp("fake")
    src, so = d / "fake.cpp", d / "libfake.so"
    src.write_text(FAKE)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-w", "-shared", "-fPIC", "-I" + os.path.join(build._cuda_home(), "include"),
                           "-I" + build.INCLUDE, "-I" + build.CSRC, str(src)] + objs +
                          ["-Wl,-Bsymbolic", "-Wl,--no-undefined", "-lpthread", "-o", str(so)])
    L = C.CDLL(str(so))
    L.fake_calls.restype = C.c_char_p
    L.dg_batch_step.argtypes = [C.c_void_p, C.c_int]
    L.dg_batch_destroy.argtypes = [C.c_void_p]
    return L


def problem(order, n):
    return dg().params_from_dict(dict(ORDER=order, NUM_ELEMENTS=[n] * 3, NUM_BLOCKS=[1, 1, 1], ELEMENT_WIDTH=[0.5] * 3,
                                      STARTING_CORNER=[0.0] * 3, EVALUATE_ADVECTION=1, EVALUATE_DIFFUSION=1,
                                      PRECISION=32, C0=1.5, RHO0=1000.0))


@pytest.mark.parametrize("orders", [(3,), (2, 3, 4)])
@pytest.mark.parametrize("nth", [1, 2, 6])
def test_step_after_a_failed_launch_starts_from_clear_counters(orders, nth, lib):
    """The launches before the failed one took tiles from the counters, which
    the step's last launch did not get to clear: the next step waits for them
    and clears the counters before its first stage kernel."""
    n = len(orders)
    params = (type(problem(3, 2)) * n)(*[problem(o, 6) for o in orders])
    h = C.c_void_p()
    assert lib.dg_batch_create(n, params, (C.c_double * n)(*[1e-3] * n), (C.c_int * n)(*[100] * n), None, None,
                               C.byref(h)) == 0
    try:
        lib.fake_reset(0)
        assert lib.dg_batch_step(h, 1) == 0
        lib.fake_reset(0)
        assert lib.dg_batch_step(h, 2) == 0
        done = lib.fake_calls().split()  # steps that end leave clear counters behind
        assert done == ([b"stage"] * (6 * n) + [b"end"]) * 2
        lib.fake_reset(nth)
        assert lib.dg_batch_step(h, 3) != 0
        cut = lib.fake_calls().split()
        assert cut.count(b"stage") == nth and b"end" not in cut
        assert b"sync" in cut[nth:]
        lib.fake_reset(0)
        assert lib.dg_batch_step(h, 1) == 0
        again = lib.fake_calls().split()
        assert b"zero" in again[:again.index(b"stage")]
        assert again.count(b"stage") == 6 * n and again.count(b"end") == 1
    finally:
        lib.dg_batch_destroy(h)
