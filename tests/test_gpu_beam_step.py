"""One layer step of the beam against its parts: the push by lcb_beam_move and
the ordered selection of moved, fallen and lost particles by boolean masks, at
the edges of the compaction's tiles (256 particles), with fresh and fallen
particles and either alone, in both forms of the push (a group of lanes per
particle up to 16384, a thread each above) and with the fallen particles'
counter updated in place.  Both forms of the push against the oracle."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs CUDA", allow_module_level=True)

from lcodepy_b200 import _lib  # noqa: E402
from lcodepy_b200.beam3d import BeamCalculator, BeamParticles, BeamSource  # noqa: E402
from lcodepy_b200.config import Config  # noqa: E402
from oracle import oracle as O  # noqa: E402

DEV = torch.device("cuda")
STATE = ("xi", "x", "y", "px", "py", "pz")


class Planes:
    def __init__(self, buf):
        self.buf = buf
        self.struct = _lib.Fields7()
        for i in range(7):
            self.struct.f[i] = buf[i].data_ptr()


def _beam(n, layer, dxi, g):
    """Particles of one layer: fast ones, slow ones that fall behind, and some
    near the radius where they are lost."""
    def rnd():
        return torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    b = BeamParticles(DEV)
    b.xi = torch.sort(-dxi * (layer + rnd().clamp(1e-3, 1 - 1e-3)), descending=True).values
    b.x, b.y = rnd() * 2.3 - 1.15, rnd() * 2.3 - 1.15
    b.px, b.py = rnd() - 0.5, rnd() - 0.5
    b.pz = torch.where(rnd() < 0.4, 0.8 + 2 * rnd(), 1000 + rnd())
    b.q_m = -torch.ones_like(b.xi)
    b.q_norm = rnd()
    b.id = torch.arange(1, n + 1, device=DEV, dtype=torch.int64)
    b.dt = torch.zeros_like(b.xi)
    b.remaining_steps = torch.zeros_like(b.id)
    return b


@pytest.mark.parametrize("fresh,fallen,in_place", [
    (1, 0, False), (255, 0, False), (256, 0, False), (257, 0, False), (5000, 0, False), (5000, 0, True),
    (20000, 0, False), (0, 1, False), (255, 2, False), (300, 4000, False), (300, 4000, True), (0, 9000, True),
    (200, 20000, False), (0, 80000, True)])
def test_layer_step_against_its_parts(fresh, fallen, in_place):
    n = fresh + fallen
    L = _lib.load()
    N, dxi = 65, 0.05
    cfg = Config({'geometry': '3d', 'window-width': 1.63, 'transverse-step': 0.05, 'window-length': 1.0,
                  'xi-step': dxi, 'time-step': 1.0})
    cfg._adjust_config_values_3d()
    assert cfg.getint('window-width-steps') == N
    g = torch.Generator(device=DEV)
    g.manual_seed(n)
    layer = 3
    b = _beam(n, layer, dxi, g)
    F = [Planes((torch.rand(7, N, N, generator=g, device=DEV, dtype=torch.float64) - 0.5) * 0.4) for _ in range(2)]
    bc = BeamCalculator(cfg, DEV)
    bc.start_time_step(BeamSource(cfg, b, DEV))
    dt, rs = torch.zeros_like(b.xi), torch.zeros_like(b.id)
    if fallen:   # two substeps of half a time step left
        dt[fresh:], rs[fresh:] = 0.5, 2
        b.dt, b.remaining_steps = dt.clone(), rs.clone()
        for k in b._all():
            getattr(bc.fell[0], k)[:fallen] = getattr(b, k)[fresh:]
        bc.counts[0] = fallen
    a = bc._args(layer + 1, (0, 0), (0, fresh), F[0], F[1])
    if in_place:
        a.fell_out_count = a.fell_in_count
    bc.drain.id[:] = -7
    _lib.check(L.lcb_beam_step(C.byref(a), _lib.stream_handle()), "lcb_beam_step")

    st = _lib.stream_handle()
    _lib.check(L.lcb_beam_substepping(fresh, b.q_m.data_ptr(), b.pz.data_ptr(), 2.0, 1.0, dt.data_ptr(), rs.data_ptr(),
                                      st), "substepping")
    p = {k: getattr(b, k).clone() for k in STATE}
    ids = b.id.clone()
    flags = torch.zeros(n, dtype=torch.uint8, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    _lib.check(L.lcb_beam_move(n, dxi, bc.r_max, layer, bc.h, N, b.q_m.data_ptr(), dt.data_ptr(),
                               C.byref(F[0].struct), C.byref(F[1].struct), rs.data_ptr(), ids.data_ptr(),
                               *(p[k].data_ptr() for k in ("x", "y", "xi", "px", "py", "pz")), flags.data_ptr(),
                               err.data_ptr(), st), "lcb_beam_move")
    torch.cuda.synchronize()
    f = flags.cpu().numpy()
    counts = bc.counts.cpu().numpy()
    fell_slot = bc.fell_cur if in_place else 1 - bc.fell_cur
    moved, fell = (f & 2) > 0, (f & 4) > 0
    assert n < 200 or (moved.any() and fell.any() and (f & 1).any())
    assert counts[2] == moved.sum() and counts[fell_slot] == fell.sum() and counts[3] == ((f & 1) > 0).sum()
    for buf, mask in ((bc.drain, moved), (bc.fell[1 - bc.fell_cur], fell)):
        k = int(mask.sum())
        np.testing.assert_array_equal(buf.id[:k].cpu().numpy(), ids.cpu().numpy()[mask])
        np.testing.assert_array_equal(buf.remaining_steps[:k].cpu().numpy(), rs.cpu().numpy()[mask])
        for name in STATE:
            np.testing.assert_array_equal(getattr(buf, name)[:k].cpu().numpy(), p[name].cpu().numpy()[mask])
    # every lost particle, those that fell as well among them, without a gap
    lost = (f & 1) > 0
    assert n < 5000 or (lost & fell).any()
    k = int(lost.sum())
    np.testing.assert_array_equal(bc.lost.id[:k].cpu().numpy(), ids.cpu().numpy()[lost])
    for name in STATE:
        np.testing.assert_array_equal(getattr(bc.lost, name)[:k].cpu().numpy(), p[name].cpu().numpy()[lost])
    if n > 1:
        assert (bc.drain.id[int(moved.sum()):] == -7).all()


@pytest.mark.parametrize("n", [3000, 20000])
def test_push_of_any_mass_against_the_oracle(n):
    """Both forms of the push against the oracle, a third of the particles
    without charge over mass (infinitely heavy: they do not move, their
    momenta grow).  A step of 0.8 layers leaves some in the layer and lets
    others fall.  As many substeps, gathers and square roots as for any beam:
    the bound is that of the push's other test."""
    N, h, dxi, layer = 65, 0.05, 0.05, 9
    rng = np.random.default_rng(n)
    p = O.Params(N=N, h=h, dxi=dxi, sub_coeff=1, boundary=0)
    b = O.Beam(xi=rng.uniform(-layer * dxi, -(layer - 1) * dxi, n), x=rng.normal(0, 0.4, n), y=rng.normal(0, 0.4, n),
               px=rng.normal(0, 1, n), py=rng.normal(0, 1, n), pz=rng.choice([0.3, 20.0, 1000.0], n),
               q_m=rng.choice([-1.0, 1 / 1836.0, 0.0], n), q_norm=np.ones(n), id=np.arange(1, n + 1, dtype=np.int64),
               dt=np.zeros(n), remaining_steps=np.zeros(n, np.int64))
    X, Y = np.meshgrid(np.arange(N), np.arange(N), indexing="ij")
    F = [O.Fields(*(0.3 * np.sin(0.2 * (i + 1 + s) * X + 0.1 * Y) for i in range(6)), np.zeros((N, N)))
         for s in (0, 0.3)]
    planes = [Planes(torch.stack([torch.tensor(getattr(f, k), device=DEV) for k in
                                  ("Ex", "Ey", "Ez", "Bx", "By", "Bz", "Phi")])) for f in F]
    g = {k: torch.tensor(getattr(b, k), device=DEV) for k in STATE + ("q_m", "id", "dt", "remaining_steps")}
    heavy = b.q_m == 0
    lost, moved, fell = O.move_beam_layer(p, b, 0, layer, *F, 0.04, 2.0)
    L, st = _lib.load(), _lib.stream_handle()
    _lib.check(L.lcb_beam_substepping(n, g["q_m"].data_ptr(), g["pz"].data_ptr(), 2.0, 0.04, g["dt"].data_ptr(),
                                      g["remaining_steps"].data_ptr(), st), "substepping")
    flags = torch.zeros(n, dtype=torch.uint8, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    R = h * N / 2
    _lib.check(L.lcb_beam_move(n, dxi, max(0.9 * R, R - 1), layer - 1, h, N, g["q_m"].data_ptr(), g["dt"].data_ptr(),
                               C.byref(planes[0].struct), C.byref(planes[1].struct), g["remaining_steps"].data_ptr(),
                               g["id"].data_ptr(), *(g[k].data_ptr() for k in ("x", "y", "xi", "px", "py", "pz")),
                               flags.data_ptr(), err.data_ptr(), st), "lcb_beam_move")
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    f = flags.cpu().numpy()
    assert (heavy & ((f & 2) > 0)).any() and (heavy & ((f & 4) > 0)).any()
    for bit, ref in ((1, lost), (2, moved), (4, fell)):
        sel = (f & bit) > 0
        np.testing.assert_array_equal(g["id"].cpu().numpy()[sel], ref.id)
        for k in STATE:
            want = getattr(ref, k)
            assert np.abs(g[k].cpu().numpy()[sel] - want).max(initial=0) <= 1e-11 * np.abs(want).max(initial=1e-300), k
