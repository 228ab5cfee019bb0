"""The fused particle stage against the three kernels run separately, where its
tiles and rules can go wrong: one to four particles per cell along an axis
(tiles of 16 x 32 particles cover 4 to 16 cells, odd sides leave remainders),
one and two sorts, first and later stages, lattices that are not where the
kernel expects the package's own (shifted by a cell and by half a cell), a
lattice smaller than one tile, and a particle that is not a number.

FP64: a node's sum has at most a few hundred terms of the same magnitude, so
its rounding stays below 1e-13 of the largest; mixed: the gather's FP32
weights and fields (6e-8 each) move the particles' momenta by at most that
share of the fields' kick, far below 1e-5 of the currents."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs CUDA", allow_module_level=True)

from lcodepy_b200 import _lib  # noqa: E402
from lcodepy_b200.config import Config  # noqa: E402
from lcodepy_b200.solver import CurrentSet, Plane2d3vPlasmaSolver  # noqa: E402

DEV = torch.device("cuda")
NAMES = ("x_offt", "y_offt", "px", "py", "pz", "q")


def _solver(N, ppc, ion_model, precision, shift=0.0, seed=5):
    h = 0.1
    cfg = Config({'geometry': '3d', 'window-width': (N + 0.5) * h / 2, 'transverse-step': h, 'xi-step': h,
                  'window-length': 1.0, 'ion-model': ion_model, 'plasma-particles-per-cell': ppc,
                  'precision': precision, 'print-every': 0})
    cfg._adjust_config_values_3d()
    ps = Plane2d3vPlasmaSolver(cfg, DEV)
    ps.init_state(0.0)
    prev, full = ps.states
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)

    def rnd(scale):
        return (torch.rand(prev.q.numel(), generator=g, device=DEV, dtype=torch.float64) - 0.5) * 2 * scale
    for s in (prev, full):
        s.x_init += shift * h
        s.y_init += shift * h
    prev.x_offt.copy_(rnd(0.8 * h))
    prev.y_offt.copy_(rnd(0.8 * h))
    for k in ("px", "py", "pz"):
        getattr(prev, k).copy_(rnd(0.3) * prev.m)
    prev.q[::37] = 0        # absorbed earlier
    for k in NAMES:
        getattr(full, k).copy_(getattr(prev, k))
    full.x_offt += rnd(0.05 * h)
    full.y_offt += rnd(0.05 * h)
    ps.fields[0].buf.copy_((torch.rand(7, ps.N, ps.N, generator=g, device=DEV, dtype=torch.float64) - 0.5) * 0.1)
    return ps


def _close(got, ref, rel, what):
    scale = float(ref.abs().max())
    assert float((got - ref).abs().max()) <= rel * max(scale, 1e-300), what


@pytest.mark.parametrize("precision,rel", [("fp64", 1e-12), ("mixed", 1e-5)])
@pytest.mark.parametrize("N,ppc,ions,first,shift", [
    (65, 1, "background", True, 0.0), (65, 4, "background", False, 0.0), (67, 9, "mobile", False, 0.0),
    (55, 16, "background", True, 0.0), (65, 4, "mobile", True, 1.0), (65, 4, "background", True, 0.5),
    (65, 1, "background", False, -2.25), (33, 4, "background", True, 0.0)])
def test_stage_against_separate_kernels(N, ppc, ions, first, shift, precision, rel):
    ps = _solver(N, ppc, ions, precision, shift)
    prev, full = ps.states
    F = ps.fields[0]
    start = {k: getattr(full, k).clone() for k in NAMES}
    if first:
        ps._move_wo_fields(prev, full)
    ps._move_smart(F, prev, full)
    want = CurrentSet(ps.N, DEV)
    ps._deposit(full, want)
    sep = {k: getattr(full, k).clone() for k in NAMES}
    got = []
    for _ in range(2):
        for k, v in start.items():
            getattr(full, k).copy_(v)
        out = CurrentSet(ps.N, DEV)
        out.buf.fill_(7.0)
        ps._move_deposit(F, prev, full, out, first)
        got.append(out.buf)
    torch.cuda.synchronize()
    assert int(ps.err.item()) == 0
    for k in NAMES:
        _close(getattr(full, k), sep[k], rel, k)
    for i, k in enumerate(("ro", "jx", "jy", "jz")):
        _close(got[0][i], want.buf[i], rel, k)
    if precision == "mixed":
        assert torch.equal(got[0], got[1])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_stage_drops_a_particle_that_is_not_a_number(precision):
    ps = _solver(65, 4, "background", precision)
    prev, full = ps.states
    k = prev.n_per_sort // 2 + 11
    prev.px[k] = float("nan")
    out = CurrentSet(ps.N, DEV)
    ps._move_deposit(ps.fields[0], prev, full, out, True)
    torch.cuda.synchronize()
    assert int(ps.err.item()) & _lib.DEVERR_PLASMA_STENCIL
    assert np.isfinite(out.buf.cpu().numpy()).all()


@pytest.mark.parametrize("N,ppc", [(129, 1), (129, 4), (129, 9)])
def test_background_cancels_the_electrons_at_rest(N, ppc):
    """Electrons that have not moved, deposited by the fused stage, against
    the background charge: what is left is the rounding of single nodes (some
    1.5 of 2^-53 rms), whose mean over n nodes is 1.5 / sqrt(n) of it, and no
    common part."""
    h = 0.05
    cfg = Config({'geometry': '3d', 'window-width': (N + 0.5) * h / 2, 'transverse-step': h, 'xi-step': h,
                  'window-length': 1.0, 'ion-model': 'background', 'plasma-particles-per-cell': ppc,
                  'precision': 'fp64', 'print-every': 0})
    cfg._adjust_config_values_3d()
    ps = Plane2d3vPlasmaSolver(cfg, DEV)
    ps.init_state(0.0)
    prev, full = ps.states
    assert all(float(getattr(s, k).abs().max()) == 0 for s in (prev, full) for k in ("x_offt", "y_offt", "px", "py", "pz"))
    out = CurrentSet(N, DEV)
    ps._move_deposit(ps.fields[0], prev, full, out, True)
    left = (out.buf[0][0] + ps.ro_initial).cpu().numpy()[24:-24, 24:-24]
    np.testing.assert_array_equal(out.buf[0][1].cpu().numpy(), ps.ro_initial.cpu().numpy())
    assert abs(left.mean()) <= 4 * 1.5 * 2.0 ** -53 / left.size ** 0.5
    assert (left ** 2).mean() ** 0.5 <= 2.5 * 2.0 ** -53


def _compare_with_separate(ps, rel):
    prev, full = ps.states
    F = ps.fields[0]
    start = {k: getattr(full, k).clone() for k in NAMES}
    ps._move_smart(F, prev, full)
    want, out = CurrentSet(ps.N, DEV), CurrentSet(ps.N, DEV)
    ps._deposit(full, want)
    for k, v in start.items():
        getattr(full, k).copy_(v)
    ps._move_deposit(F, prev, full, out, False)
    torch.cuda.synchronize()
    assert int(ps.err.item()) == 0
    for i, k in enumerate(("ro", "jx", "jy", "jz")):
        _close(out.buf[i], want.buf[i], rel, k)
    return want.buf[0][0]


@pytest.mark.parametrize("precision,rel", [("fp64", 1e-12), ("mixed", 1e-5)])
@pytest.mark.parametrize("ppc,share", [(1, 0.98), (4, 0.98), (4, 0.7), (9, 0.98)])
def test_stage_where_a_tile_meets_in_few_cells(ppc, share, precision, rel):
    """A density spike: the particles of every 16 x 32 of the lattice drawn
    together to a point, so that one cell holds hundreds."""
    ps = _solver(97, ppc, "background", precision)
    prev, full = ps.states
    Ns = prev.Ns
    i = torch.arange(Ns, device=DEV)
    for k, tile in (("x", 16), ("y", 32)):
        at = getattr(prev, k + "_init").view(Ns, Ns)
        u = at[:, 0] if k == "x" else at[0]
        to = u[(i // tile * tile + tile // 2).clamp(max=Ns - 1)]
        d = (to - u) * share
        for s in (prev, full):
            getattr(s, k + "_offt").copy_((d[:, None] if k == "x" else d[None]).expand(Ns, Ns).reshape(-1))
    for s in (prev, full):
        for k in ("px", "py", "pz"):
            getattr(s, k).mul_(0.1)
    # (512 particles of 1 / ppc each in a cell, weights up to 0.6^2)
    assert float(_compare_with_separate(ps, rel).abs().max()) > (0.5 * 512 / ppc * 0.36 if share > 0.9 else 3)


@pytest.mark.parametrize("ppc", [1, 4])
@pytest.mark.parametrize("precision,big,rel", [("fp64", 1e201, 1e-12), ("fp64", 1e199, 1e-12), ("mixed", 4096.0, 1e-8)])
def test_stage_with_values_out_of_a_blocks_range(ppc, precision, big, rel):
    """Particles whose density reaches what a block does not sum (FP64 1e200,
    mixed 2^10) go to HBM by themselves; the others stay as they are."""
    ps = _solver(65, ppc, "background", precision)
    prev, full = ps.states
    n = prev.n_per_sort
    ps.fields[0].buf.zero_()
    k = n // 2 + 11
    for s in (prev, full):
        s.q[k] = big * ps.h ** 2
        s.x_offt[k] = s.y_offt[k] = s.px[k] = s.py[k] = s.pz[k] = 0
    top = _compare_with_separate(ps, rel)
    assert 0.1 * big < float(top.abs().max()) < big
    far = torch.ones(ps.N, ps.N, dtype=torch.bool, device=DEV)
    at = int(top.abs().argmax())
    far[at // ps.N - 5:at // ps.N + 6, at % ps.N - 5:at % ps.N + 6] = False
    got, want = CurrentSet(ps.N, DEV), CurrentSet(ps.N, DEV)
    ps._deposit(full, want)
    ps._move_deposit(ps.fields[0], prev, full, got, False)
    for a, b in zip(got.buf, want.buf):
        _close(a[0][far], b[0][far], 1e-12 if precision == "fp64" else 1e-5, "elsewhere")
