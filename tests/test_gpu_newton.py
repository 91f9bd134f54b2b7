"""rcp and root (csrc/surface_fluxes.cuh) against the division and the square root that
numpy rounds correctly, over the range their comment states and at its ends, and states
on which they meet 0.

Tolerance: one unit in the last place of the result.  The last Newton step leaves a
relative error of the square of the step before (FP64 2^-78, FP32 2^-42) and one rounding
of a sum whose correction is itself rounded: below one unit.
"""

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle as O
from gpu_util import initial_state, oracle_law, product_scheme, rel_err, wrap_oracle_grid

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = """
#include "surface_fluxes.cuh"
template <typename T>
__global__ void both(const T* x, T* r, T* s, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        r[i] = rb200::rcp(x[i]);
        s[i] = rb200::root(x[i]);
    }
}
template <typename T>
int run(const T* x, T* r, T* s, int n) {
    both<T><<<64, 256>>>(x, r, s, n);
    cudaError_t e = cudaGetLastError();
    return e != cudaSuccess ? (int)e : (int)cudaDeviceSynchronize();
}
extern "C" int run64(const double* x, double* r, double* s, int n) { return run(x, r, s, n); }
extern "C" int run32(const float* x, float* r, float* s, int n) { return run(x, r, s, n); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    d = tmp_path_factory.mktemp("newton")
    (d / "newton.cu").write_text(SOURCE)
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared",
                           "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I",
                           os.path.join(ROOT, "raven.jl_b200", "csrc"), "-o", str(d / "newton.so"),
                           str(d / "newton.cu")])
    return ctypes.CDLL(str(d / "newton.so"))


def _both(lib, x):
    import torch

    t = torch.from_numpy(x).cuda()
    r, s = torch.empty_like(t), torch.empty_like(t)
    torch.cuda.synchronize()
    f = lib.run64 if x.dtype == np.float64 else lib.run32
    assert f(*(ctypes.c_void_p(v.data_ptr()) for v in (t, r, s)), ctypes.c_int(x.size)) == 0
    return r.cpu().numpy(), s.cpu().numpy()


@pytest.mark.parametrize("dtype,rcp_lo,root_lo,hi", [(np.float64, -1022, -960, 1022), (np.float32, -126, -100, 126)])
def test_within_one_unit(lib, cuda_ok, dtype, rcp_lo, root_lo, hi):
    rng = np.random.default_rng(1)
    n = 1 << 20
    for lo, which in ((rcp_lo, 0), (root_lo, 1), (-4, 0), (-4, 1)):
        top = hi if lo < -4 else 4
        x = np.ldexp(rng.uniform(1, 2, n), rng.integers(lo, top, n)).astype(dtype)
        x[:2] = np.ldexp(1.0, lo), np.ldexp(1.0, top)
        want = (dtype(1) / x, np.sqrt(x))[which]
        got = _both(lib, x)[which]
        assert (np.abs(got - want) <= np.spacing(want)).all()
        if which == 0:
            assert np.array_equal(_both(lib, -x)[0], -got)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_ends_of_the_range(lib, cuda_ok, dtype):
    tiny = np.finfo(dtype).smallest_subnormal
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, tiny, -1.0, np.finfo(dtype).max], dtype=dtype)
    r, s = _both(lib, x)
    with np.errstate(all="ignore"):
        want_r, want_s = dtype(1) / x, np.sqrt(x)
    want_r[7] = 0  # a subnormal reciprocal
    want_s[5] = tiny  # a subnormal argument counts as 0
    assert np.array_equal(r, want_r, equal_nan=True) and np.array_equal(np.signbit(r[:4]), np.signbit(want_r[:4]))
    keep = [0, 1, 2, 3, 4, 5, 6]
    assert np.array_equal(s[keep], want_s[keep], equal_nan=True) and np.signbit(s[1])


@pytest.mark.parametrize("dim,nq", [(2, 5), (3, 4), (3, 5), (3, 8)])
def test_node_without_pressure(rb, cuda_ok, dim, nq):
    """One node at rest with p = 0 exactly, entropy-conservative form: rho / p is infinite there
    and its logarithmic mean has no value, so the energy of its lines is NaN; densities and
    momenta stay finite, as in the oracle, which divides."""
    og = O.Grid(dim, nq, (2,) * dim, [0.0] * dim, [10.0] * dim, (1,) * dim)
    law, form = product_scheme(rb, "eul_ec", dim)
    dg = rb.DGSEM(law=law, grid=wrap_oracle_grid(og), volume_form=form, surface_numericalflux=rb.RusanovFlux())
    assert (dg.pipelined_ctas > 0) == (dim == 3)
    olaw = oracle_law("eul_ec", dim)
    q = initial_state(og, olaw, "eul_ec", seed=11, amp=0.01)
    node = 1 + nq + (nq * nq if dim == 3 else 0)  # interior
    q[node, 1:, 0] = 0.0
    ref = og.tendency(olaw, q)
    assert np.isfinite(ref[:, :-1]).all() and not np.isfinite(ref[node, -1, 0])
    qg = rb.GridArray.from_numpy(q)
    dq = qg.similar()
    dg(dq, qg, 0.0, increment=False)
    got = dq.numpy()
    assert np.array_equal(np.isfinite(got), np.isfinite(ref))
    assert rel_err(got[:, :-1], ref[:, :-1]) <= 1e-12
