"""The FP32 kernels' 64-bit-offset forms, which fields of 4 GiB and more (a
batch: states of 2^32 values) take, against their 32-bit forms bit for bit.

The kernels take the distance of two elements in memory as an argument: a few
elements that lie far enough apart reach the offsets of a large problem, with
all fields interleaved in the room between them.  The shim instantiates the
forms of each kernel from its header; the single-problem kernels also as a
dependent launch."""
import ctypes as C
import importlib
import os
import subprocess

import numpy as np
import pytest

from conftest import dg

pytestmark = pytest.mark.gpu

SHIM = r"""
#include <cstring>
#include "incr_kernels.cuh"
#include "batch_kernels.cuh"
using namespace dg;

extern "C" int narrow_rules(unsigned long long fs) { return incr_narrow(fs) | batch_narrow(fs) << 1; }

template <int K, bool PDL, typename Off>
static void single(float* b, long long fs, int np, int n, const int* nbr, const float* sigma, const int* bnd_src,
                   const float* bnd_ap, const double* D, const double* L0, const double* LN)
{
    const double w[3] = {0.5, 0.4, 0.6};
    const OpConst<float, K> S = make_stage_const<float, K>(0.01, D, L0, LN, w, 1000.0, 1.5, 5.0, 4.3e-6);
    const OpConst<float, K> G = make_grad_const<float, K>(D, L0, LN, w, 1000.0, 1.5, 4.3e-6);
    StageIO<float> io;
    std::memset(&io, 0, sizeof io);
    io.src = b;
    io.inc = b + 4 * fs;
    io.dst = b + 8 * fs;
    io.comp = b + 12 * fs;
    io.q = io.q_out = b + 16 * fs;
    io.fs = fs;
    io.np = np;
    io.ca = 0.01f;
    io.cb = 0.667f;
    io.eps = 1e-8f;
    io.final_stage = 1;
    MeshDev<float> m;
    std::memset(&m, 0, sizeof m);
    m.nbr = nbr;
    m.sigma = sigma;
    m.bnd_src = bnd_src;
    m.bnd_ap = bnd_ap;
    m.n_elem = n;
    m.src_p = 0.3f;
    const int grid = (n + incr_epb(K) - 1) / incr_epb(K), threads = incr_threads(K);
    if (PDL) launch_pdl(incr_gradient_kernel<K, PDL, Off>, grid, threads, 0, io, m, G);
    else incr_gradient_kernel<K, PDL, Off><<<grid, threads>>>(io, m, G);
    void (*stage)(StageIO<float>, MeshDev<float>, const OpConst<float, K>, int, int);
    if constexpr (incr_epb(K) > 1) stage = incr_packed_stage_kernel<K, true, PDL, Off>;
    else stage = incr_stage_kernel<K, true, PDL, Off>;
    if (PDL) launch_pdl(stage, grid, threads, 0, io, m, S, 1, 1);
    else stage<<<grid, threads>>>(io, m, S, 1, 1);
}

template <int K, typename Off>
static void batch(float* b, long long fs, int np, int n, const int* nbr, const float* sigma, BatchProblem* dP,
                  BatchTile* dT, int* counters, const double* D, const double* L0, const double* LN)
{
    const double w[3] = {1.0, 1.0, 1.0};
    const OpConst<double, K> S = make_stage_const<double, K>(1.0, D, L0, LN, w, 1000.0, 1.5, 5.0, 4.3e-6);
    BatchProblem P;
    std::memset(&P, 0, sizeof P);
    P.K = K;
    P.np = np;
    P.n_elem = n;
    P.src_face = 4;
    P.active = 1;
    P.u[0] = b;
    P.u[1] = b + 4 * fs;
    P.comp = b + 8 * fs;
    P.d[0] = b + 12 * fs;
    P.d[1] = b + 16 * fs;
    P.q = b + 20 * fs;
    P.nbr = nbr;
    P.sigma = sigma;
    P.fs = fs;
    BatchOps ops;
    std::memset(&ops, 0, sizeof ops);
    for (int i = 0; i < K; i++) {
        for (int j = 0; j < K; j++) ops.rows[i][j] = (float)D[i * K + j];
        ops.rows[i][K] = (float)L0[i];
        ops.rows[i][K + 1] = (float)LN[i];
    }
    std::memcpy(P.rows, ops.rows, sizeof P.rows);
    for (int a = 0; a < 3; a++) {
        P.invw[a] = 2.f;
        P.gscale[a] = 8.6e-6f;
        P.ca[a] = 0.01f / (a + 1);
        P.cb[a] = 0.3f * a;
        P.src_p[a] = 0.3f;
    }
    for (int s = 0; s < 2; s++)
        for (int i = 0; i < 4; i++) {
            P.cM[s][i] = (float)S.cM[0][s][i];
            P.cA[s][i] = (float)S.cA[0][s][i];
        }
    P.k1 = (float)S.k1;
    P.k2 = (float)S.k2;
    P.r0 = (float)S.r0;
    P.inv_c2 = 0.44f;
    P.inv_z = 6.7e-4f;
    const BatchTile T = {0, 0, n, K};
    cudaMemcpy(dP, &P, sizeof P, cudaMemcpyHostToDevice);
    cudaMemcpy(dT, &T, sizeof T, cudaMemcpyHostToDevice);
    for (int s = 0; s < 3; s++) {
        const BatchArgs A = {dP, dT, 0, 1, counters, s};
        batch_stage_kernel<K, 0, false, Off><<<1, bthreads_of(K)>>>(A, ops);
        batch_stage_kernel<K, 1, false, Off><<<1, bthreads_of(K)>>>(A, ops);
    }
}

extern "C" int run(int form, int K, int wide, float* b, long long fs, int np, int n, const int* nbr, const float* sigma,
                   const int* bnd_src, const float* bnd_ap, void* dP, void* dT, int* counters, const double* D,
                   const double* L0, const double* LN)
{
#define SINGLE(k)                                                                                          \
    if (form == 0 && K == k) {                                                                            \
        if (wide == 2) single<k, true, unsigned>(b, fs, np, n, nbr, sigma, bnd_src, bnd_ap, D, L0, LN);  \
        else if (wide) single<k, false, size_t>(b, fs, np, n, nbr, sigma, bnd_src, bnd_ap, D, L0, LN);   \
        else single<k, false, unsigned>(b, fs, np, n, nbr, sigma, bnd_src, bnd_ap, D, L0, LN);           \
    }
#define BATCH(k)                                                                                           \
    if (form == 1 && K == k) {                                                                            \
        if (wide) batch<k, size_t>(b, fs, np, n, nbr, sigma, (BatchProblem*)dP, (BatchTile*)dT, counters, D, L0, LN); \
        else batch<k, unsigned>(b, fs, np, n, nbr, sigma, (BatchProblem*)dP, (BatchTile*)dT, counters, D, L0, LN);    \
    }
    SINGLE(2) SINGLE(3) SINGLE(4) SINGLE(5) SINGLE(6) SINGLE(7) SINGLE(8) BATCH(3) BATCH(5) BATCH(6)
    const cudaError_t e = cudaGetLastError();
    return (int)(e == cudaSuccess ? cudaDeviceSynchronize() : e);
}
extern "C" int problem_bytes() { return (int)sizeof(BatchProblem); }
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    build = importlib.import_module("3ddg_gb300.build")
    d = tmp_path_factory.mktemp("wide")
    src, so = d / "shim.cu", d / "libshim.so"
    src.write_text(SHIM)
    subprocess.check_call([os.path.join(build._cuda_home(), "bin", "nvcc")] + build.NVCC_FLAGS +
                          ["-w", "-shared", str(src), "-o", str(so)])
    lib = C.CDLL(str(so))
    vp, i = C.c_void_p, C.c_int
    lib.run.argtypes = [i, i, i, vp, C.c_longlong, i, i] + [vp] * 10
    lib.narrow_rules.argtypes = [C.c_ulonglong]
    return lib


def test_rules(shim):
    """Fields below 4 GiB; states of fewer than 2^32 values."""
    for fs, want in [(1, 3), (2 ** 30 - 1, 3), (2 ** 30, 0), (2 ** 32, 0)]:
        assert shim.narrow_rules(fs) == want


# 9 elements: the last of them at 2^30 values and more (a field's 4 GiB), 2^32 in a batch
@pytest.mark.parametrize("form,K,far", [(0, 2, 2 ** 27), (0, 4, 2 ** 27), (0, 5, 2 ** 27), (0, 8, 2 ** 27),
                                        (1, 3, 2 ** 29), (1, 5, 2 ** 29), (1, 6, 2 ** 29)])
def test_far_elements_bitwise_as_near_ones(form, K, far, shim):
    near = 23 * 1024
    n = 9
    assert K ** 3 <= 1024 and far >= near and (n - 1) * far * 4 >= 2 ** 32 and (form == 0 or (n - 1) * far >= 2 ** 32)
    compare(form, K, ((0, near), (1, far)), shim)


@pytest.mark.parametrize("K", range(2, 9))
def test_dependent_launches_bitwise_as_waiting_ones(K, shim):
    compare(0, K, ((0, 23 * 1024), (2, 23 * 1024)), shim)


def compare(form, K, forms, shim):
    """The outputs of the given (form, distance) pairs are the same bits."""
    import torch
    n, fs, n_fields = 9, 1024, 23
    near = n_fields * fs
    far = max(d for _, d in forms)
    if torch.cuda.mem_get_info()[0] < (n * far * 4 + (4 << 30)):
        pytest.skip("not enough free device memory")
    rng = np.random.default_rng(10 * K + form)
    values = torch.from_numpy((rng.standard_normal((n, n_fields, K ** 3)) * 1e-3).astype(np.float32)).cuda()
    nbr = rng.integers(0, n, (n, 6)).astype(np.int32)
    nbr[rng.random((n, 6)) < 0.2] = -1 - 2
    nbr[4, 4] = -1 - 4
    cuda = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    d_nbr, sigma = cuda(nbr), cuda(rng.random(n).astype(np.float32))
    bnd_src = cuda(np.array([0, 0, 0, 0, 1, 0], dtype=np.int32))
    bnd_ap = cuda(rng.random(6 * K * K).astype(np.float32))
    d_prob = torch.zeros(shim.problem_bytes() + 64, dtype=torch.uint8, device="cuda")
    tiles, counters = (torch.zeros(16, dtype=torch.int32, device="cuda") for _ in range(2))
    ops = dg().line_operators(K - 1)
    host = [np.ascontiguousarray(ops[k]) for k in ("deriv", "lift0", "liftN")]
    out = []
    for wide, np_slots in forms:
        buf = torch.empty(n * np_slots, dtype=torch.float32, device="cuda")
        view = buf.view(n, np_slots)[:, :near].view(n, n_fields, fs)[:, :, :K ** 3]
        view.copy_(values)
        torch.cuda.synchronize()
        p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
        rc = shim.run(form, K, wide, p(buf), fs, np_slots, n, p(d_nbr), p(sigma), p(bnd_src), p(bnd_ap), p(d_prob),
                      p(tiles), p(counters), *[a.ctypes.data_as(C.c_void_p) for a in host])
        assert rc == 0
        out.append(view.cpu().numpy().copy())
        del view, buf
    changed = (out[0] != values.cpu().numpy()).reshape(n, n_fields, -1).any(axis=2)
    assert changed[:, 16 if form == 0 else 20].all() and np.isfinite(out[0]).all()
    assert np.array_equal(out[0], out[1])
