"""The reciprocal of the FP32 kernels' canopy solve (``rcp_nr``, ibis_pair.cuh) against the
correctly rounded one.

The approximation it starts from has an error of at most 2**-20; two Newton-Raphson steps
square it to 2**-40 and 2**-80.  The last step is one fma whose correction is known to
2**-53 of itself, so its result is the rounding of a number within 2**-80 of 1 / x: the
correctly rounded reciprocal or, where 1 / x lies next to the middle of two doubles, the
other of the two.
"""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

from ibis_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = """
#include "ibis_pair.cuh"
__global__ void k(const double* x, double* y, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = ibis::rcp_nr(x[i]);
}
extern "C" int rcp_of(const double* x, double* y, int n) {
    k<<<(n + 255) / 256, 256>>>(x, y, n);
    return cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def rcp_of(cuda_lib, tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("pair")
    (d / "rcp.cu").write_text(SOURCE)
    subprocess.run([nvcc, *build.ARCH, *build.COMMON, *build.F32_FLAGS, "-I", build.CSRC, "-shared", "-o",
                    str(d / "rcp.so"), str(d / "rcp.cu")], check=True, capture_output=True)
    fn = ctypes.CDLL(str(d / "rcp.so")).rcp_of
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int]

    def call(x):
        xd = torch.from_numpy(x).cuda()
        y = torch.zeros_like(xd)
        torch.cuda.synchronize()
        assert fn(xd.data_ptr(), y.data_ptr(), x.size) == 0
        return y.cpu().numpy()

    return call


@pytest.mark.parametrize("span", [1, 12, 30, 250])
def test_reciprocals_are_within_one_unit(rcp_of, span):
    rng = np.random.default_rng(span)
    x = 10.0 ** rng.uniform(-span, span, 1 << 20) * rng.choice([-1.0, 1.0], 1 << 20)
    two = 2.0 ** np.arange(-int(span * 3.3), int(span * 3.3) + 1)
    x = np.concatenate([x, two, -two, np.nextafter(two, 0), np.nextafter(two, np.inf)])
    got, want = rcp_of(x), 1.0 / x
    assert np.isfinite(want).all() and (np.abs(want) > np.finfo(np.float64).tiny).all()
    assert (np.abs(got - want) <= np.spacing(np.abs(want))).all()
