"""Field solves on either side of the choice between the fast transforms
(N - 1 a product of primes up to 13) and the dense tensor-core products:
every radix, the lengths with their own kernels, both kernels of the columns
(two columns a block below 1,100 points a line, one above) and the smallest
grids, against the oracle.  The fast transforms run in FP64 in both
precisions, so both are held to the FP64 bound: two transforms and back of at
most 2 N points with a spectral factor lose a few tens of 2^-53 of the field's
largest value; the factor's spread (a condition of at most N^2) multiplies
the right-hand side's own rounding, which both sides share."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs CUDA", allow_module_level=True)

import ctypes as C  # noqa: E402
import os  # noqa: E402
import subprocess  # noqa: E402
import sys  # noqa: E402

import numpy as np  # noqa: E402

from lcodepy_b200 import _lib  # noqa: E402
from lcodepy_b200.plasma3d import FieldOperators  # noqa: E402
from oracle import oracle as O  # noqa: E402
from test_gpu_kernels import DEV, _fields_args  # noqa: E402
from test_gpu_kernels import test_compute_fields_sizes_vs_oracle as check  # noqa: E402

BOTH = (_lib.LCB_PREC_FP64, _lib.LCB_PREC_MIXED)


@pytest.mark.parametrize("precision", BOTH)
@pytest.mark.parametrize("N", [9, 11, 15, 19, 23, 27, 51, 55, 65, 79, 91, 111, 133, 155, 193, 321, 331, 385, 551, 577, 641])
def test_fast_transforms_vs_oracle(N, precision):
    check(N, precision, 1e-11)
    assert _lib.load().lcb_wave_kernel_choice(N, precision) == 3


@pytest.mark.parametrize("precision,rel", [(_lib.LCB_PREC_FP64, 1e-11), (_lib.LCB_PREC_MIXED, 3e-5)])
@pytest.mark.parametrize("N", [35, 39, 95, 139, 259, 495, 519])
def test_dense_transforms_vs_oracle(N, precision, rel):
    """Grids with a larger prime factor in N - 1 (17, 19, 47, 23, 43, 19, 37):
    32- and 64-wide tiles, eight and four slices, full and ragged ones."""
    check(N, precision, rel)
    assert _lib.load().lcb_wave_kernel_choice(N, precision) in (1, 2)


@pytest.mark.parametrize("kernel", ["tiled", "persistent"])
def test_either_wave_kernel_on_grids_with_fast_transforms(kernel):
    """LCB_WAVE_KERNEL, read once per process, takes the dense products for
    every grid."""
    code = ("import sys; sys.path[:0] = sys.argv[1:]\n"
            "from test_gpu_kernels import _lib, test_compute_fields_sizes_vs_oracle as check\n"
            "for N in (33, 129, 257, 513):\n"
            "    check(N, _lib.LCB_PREC_FP64, 1e-11)\n"
            "    check(N, _lib.LCB_PREC_MIXED, 3e-5)\n"
            "    assert _lib.load().lcb_wave_kernel_choice(N, _lib.LCB_PREC_FP64) != 3\n")
    here = os.path.dirname(os.path.abspath(__file__))
    subprocess.run([sys.executable, "-c", code, os.path.dirname(here), here], check=True, timeout=300,
                   env={**os.environ, "LCB_WAVE_KERNEL": kernel})


@pytest.mark.parametrize("small", ["transverse currents", "charge"])
@pytest.mark.parametrize("N", [51, 65, 129, 769])
def test_a_small_field_keeps_its_precision(N, small):
    """Fields that share a transform and differ by a factor of a million: each
    to the rounding of its own size.  The right-hand sides are sums of a few
    terms of their own field's size, so that the oracle's rounding and the
    kernel's are some 2^-53 of it, times sqrt(N) or so of the transforms.  (769:
    several patches per block of the right-hand sides.)"""
    rng = np.random.default_rng(N)
    h = dxi = 0.05
    p = O.Params(N=N, h=h, dxi=dxi, sub_coeff=1 + dxi, boundary=0)
    consts = O.Consts(None, O.dirichlet_matrix(N, h), O.mixed_matrix(N, h, 1 + dxi), O.neumann_matrix(N, h))
    a, b = (1.0, 1e-6) if small == "transverse currents" else (1e-6, 1.0)

    def cur():
        v = np.zeros((4, 2, N, N))
        v[:, :, 3:-3, 3:-3] = rng.normal(0, 1, (4, 2, N - 6, N - 6))
        return O.Currents(a * v[0], b * v[1], b * v[2], b * v[3])
    cp, cf = cur(), cur()
    zero = np.zeros((N, N))
    F, Fp = (O.Fields(*(np.zeros((N, N)) for _ in range(7))) for _ in range(2))
    full, half = O.compute_fields(p, F, Fp, consts, zero, zero, cp, cf)
    d = {"N": N, "h": h, "dxi": dxi, "sub": 1 + dxi, "rb_full": zero, "rb_prev": zero}
    for k in ("ro", "jx", "jy", "jz"):
        d["cp_" + k], d["cf_" + k] = getattr(cp, k), getattr(cf, k)
    names = ("Ex", "Ey", "Ez", "Bx", "By", "Bz", "Phi")
    for k in names:
        d["in_" + k], d["prev_" + k] = getattr(F, k), getattr(Fp, k)
    prec = _lib.LCB_PREC_FP64
    ops = FieldOperators(N, h, 1 + dxi, DEV, False)
    outs = [torch.zeros((7, N, N), dtype=torch.float64, device=DEV) for _ in range(2)]
    ws = torch.empty(_lib.load().lcb_compute_fields_workspace_bytes(N, prec), dtype=torch.uint8, device=DEV)
    args, keep = _fields_args(d, prec, ops, outs, ws)
    _lib.check(_lib.load().lcb_compute_fields(C.byref(args), _lib.stream_handle()), "compute_fields")
    got = outs[0].cpu().numpy()
    for i, k in enumerate(names):
        want = getattr(full, k)
        assert np.abs(got[i] - want).max() <= 1e-13 * np.abs(want).max(), k
