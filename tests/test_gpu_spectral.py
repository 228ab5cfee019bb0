"""Field solves on either side of the choice between the fast transforms
(N - 1 a product of primes up to 13) and the dense tensor-core products:
every radix, the lengths with their own kernels and the smallest grids,
against the oracle.  The fast transforms run in FP64 in both precisions, so
both are held to the FP64 bound: two transforms and back of at most 2 N
points with a spectral factor lose a few tens of 2^-53 of the field's
largest value; the factor's spread (a condition of at most N^2) multiplies
the right-hand side's own rounding, which both sides share."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs CUDA", allow_module_level=True)

from lcodepy_b200 import _lib  # noqa: E402
from test_gpu_kernels import test_compute_fields_sizes_vs_oracle as check  # noqa: E402

BOTH = (_lib.LCB_PREC_FP64, _lib.LCB_PREC_MIXED)


@pytest.mark.parametrize("precision", BOTH)
@pytest.mark.parametrize("N", [9, 11, 15, 19, 23, 27, 51, 65, 79, 91, 111, 155, 193, 321, 331, 385])
def test_fast_transforms_vs_oracle(N, precision):
    check(N, precision, 1e-11)
    assert _lib.load().lcb_wave_kernel_choice(N, precision) == 3


@pytest.mark.parametrize("precision,rel", [(_lib.LCB_PREC_FP64, 1e-11), (_lib.LCB_PREC_MIXED, 3e-5)])
@pytest.mark.parametrize("N", [39, 95, 259])
def test_dense_transforms_vs_oracle(N, precision, rel):
    """Grids with a larger prime factor in N - 1 (19, 47, 43)."""
    check(N, precision, rel)
    assert _lib.load().lcb_wave_kernel_choice(N, precision) in (1, 2)
