"""The plasma push's reciprocal and square root against 64-bit mantissas, over
the exponents that momenta and their squares can take."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs CUDA", allow_module_level=True)

from lcodepy_b200 import build  # noqa: E402

SOURCE = """
#include "common.cuh"
__global__ void k(int n, const double *x, double *r, double *s)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { r[i] = lcb::rcp_nr(x[i]); s[i] = lcb::sqrt_nr(fabs(x[i])); }
}
extern "C" int run(int n, const double *x, double *r, double *s)
{
    k<<<(n + 127) / 128, 128>>>(n, x, r, s);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def newton(tmp_path_factory):
    if shutil.which(build.NVCC) is None:
        pytest.skip("needs nvcc")
    d = tmp_path_factory.mktemp("newton")
    src, lib = d / "newton.cu", d / "newton.so"
    src.write_text(SOURCE)
    subprocess.check_call([build.NVCC, *build.ARCH, *build.FLAGS, "-I" + build.CSRC, "-shared", "-o", os.fspath(lib),
                           os.fspath(src), "-lcudart"])
    so = C.CDLL(os.fspath(lib))

    def call(x):
        t = [torch.tensor(x, device="cuda"), *(torch.zeros(len(x), dtype=torch.float64, device="cuda") for _ in "rs")]
        torch.cuda.synchronize()
        assert so.run(len(x), *(C.c_void_p(v.data_ptr()) for v in t)) == 0
        return t[1].cpu().numpy(), t[2].cpu().numpy()
    return call


def test_within_their_bound(newton):
    rng = np.random.default_rng(3)
    n = 400_000
    x = np.ldexp(rng.uniform(1, 2, n), rng.integers(-1000, 1000, n))
    x[: n // 2] = rng.uniform(1, 4, n // 2)          # every mantissa of both parities
    x[::2] = -x[::2]
    r, s = newton(x)
    one, xl = np.longdouble(1), x.astype(np.longdouble)
    for got, want in ((r, one / xl), (s, np.sqrt(np.abs(xl)))):
        ulp = np.spacing(np.abs(want).astype(np.float64)).astype(np.longdouble)
        assert float((np.abs(got - want) / ulp).max()) <= 0.51
