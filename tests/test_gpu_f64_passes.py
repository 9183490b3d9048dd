"""The FP64 step as passes over z slabs against the tile march, which evaluates the same expressions in
the same order: equal bit for bit, whichever of the two a call takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _pair(n, **kw):
    """The same forced state in a context that runs the passes and in one whose tile the caller chose."""
    from glmmhdturb_b200 import Solver
    kw = dict(dtype="f64", gamma=5 / 3, turb_amp=2.0, turb_T=0.5, **kw)
    a, b = Solver(n, **kw), Solver(n, tile=(16, 16, 0), **kw)
    u = a.alloc()
    a.ic_turbulent(u, mach=1.5, seed=3)
    a.forcing_reset()
    a.forcing_advance()
    b.set_modes(a.get_modes())
    return a, b, u


def _step(s, u, out):
    s.step(u, out, 0.02 * s.dx, t=0.1, ch=3.0, glm_fac=0.99, do_turb=True, want_cfl=True)


@pytest.mark.parametrize("recon,riem", [("mc", "hlld"), ("mc", "hll"), ("mc", "llf"), ("mc", "llf_bound"), ("minmod", "hlld"),
                                        ("ppm", "hlld"), ("ppm", "hll")])
@pytest.mark.parametrize("iflo", [True, False])
def test_schemes(recon, riem, iflo):
    a, b, u = _pair((48, 32, 13), recon=recon, riemann=riem, iflo=iflo, llf_dmin=0.5 if riem == "hlld" else 0.0)
    x, y = torch.full_like(u, float("nan")), torch.empty_like(u)
    _step(a, u, x)
    _step(b, u, y)
    assert torch.equal(x, y)
    assert a.cfl_result() == b.cfl_result()


def test_slabs():
    """A box whose scratch is more than one slab (18 planes of it exceed 1 GB)."""
    a, b, u = _pair((512, 512, 44))
    x, y = torch.full_like(u, float("nan")), torch.empty_like(u)
    _step(a, u, x)
    _step(b, u, y)
    assert torch.equal(x, y)


def test_more_planes_than_a_launch_takes():
    """A narrow box whose planes exceed gridDim.y (65535) in one slab, though their scratch would fit one."""
    from glmmhdturb_b200 import Solver
    n = (8, 4, 70000)
    a, b = Solver(n, dtype="f64", gamma=5 / 3), Solver(n, dtype="f64", gamma=5 / 3, tile=(8, 4, 0))
    u = a.alloc()
    a.ic_turbulent(u, mach=1.0, seed=3)
    x, y = torch.full_like(u, float("nan")), torch.empty_like(u)
    for s, o in ((a, x), (b, y)):
        s.step(u, o, 0.02 * s.dx, ch=3.0, glm_fac=0.99, want_cfl=True)
    assert torch.equal(x, y)
    assert a.cfl_result() == b.cfl_result()


def test_kernel_info_reports_the_route():
    """The flux pass of a context that runs the passes (16x8 columns, 128 registers for four blocks per SM, its
    shared memory below the 48 KB of a launch without attributes); the march of one whose tile was chosen."""
    from glmmhdturb_b200 import Solver
    a = Solver((48, 32, 13), dtype="f64").kernel_info()
    b = Solver((48, 32, 13), dtype="f64", tile=(16, 16, 0)).kernel_info()
    assert a["tile"][:2] == (16, 8) and 1 <= a["tile"][2] <= 13 and 0 < a["regs"] <= 128 and 0 < a["smem"] <= 48 * 1024
    assert b["tile"][:2] == (16, 16) and b["regs"] > 128 and b["smem"] > 48 * 1024


def test_under_capture_and_after():
    """A captured step takes the tile march (it must not be ordered against work outside its graph)."""
    from glmmhdturb_b200 import Solver
    s = Solver((33, 20, 9), dtype="f64", gamma=5 / 3)
    u = s.alloc()
    s.ic_turbulent(u, mach=1.0, seed=1)
    x, y = torch.empty_like(u), torch.full_like(u, float("nan"))
    s.step(u, x, 0.02 * s.dx, ch=3.0, glm_fac=0.99)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        s.step(u, y, 0.02 * s.dx, ch=3.0, glm_fac=0.99)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(x, y)


@pytest.mark.parametrize("n", [(24, 24, 24), (33, 20, 9)])
def test_small_boxes_on_several_streams(n):
    """Steps of small boxes that change the stream take the march, which overlaps, instead of turns at the
    scratch; the values are the same in any order of streams, and a stream that stays takes the passes again."""
    from glmmhdturb_b200 import Solver
    s = Solver(n, dtype="f64", gamma=5 / 3)
    us, ref = [], []
    for seed in range(4):
        u = s.alloc()
        s.ic_turbulent(u, mach=1.0, seed=seed + 1)
        o = torch.empty_like(u)
        s.step(u, o, 0.02 * s.dx, ch=3.0, glm_fac=0.99)
        us.append(u)
        ref.append(o)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in us]
    outs = [torch.full_like(u, float("nan")) for u in us]
    torch.cuda.synchronize()
    for i in (0, 1, 2, 3, 3, 3, 0, 2, 1, 1, 0):
        s.step(us[i], outs[i], 0.02 * s.dx, ch=3.0, glm_fac=0.99, stream=streams[i])
    torch.cuda.synchronize()
    for o, r in zip(outs, ref):
        assert torch.equal(o, r)


def test_two_streams_share_a_context():
    """Steps of one context on two streams take its scratch in turn."""
    from glmmhdturb_b200 import Solver
    s = Solver(48, dtype="f64", gamma=5 / 3)
    us, ref = [], []
    for seed in (1, 2):
        u = s.alloc()
        s.ic_turbulent(u, mach=1.0, seed=seed)
        o = torch.empty_like(u)
        s.step(u, o, 0.02 * s.dx, ch=3.0, glm_fac=0.99)
        us.append(u)
        ref.append(o)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [torch.full_like(u, float("nan")) for u in us]
    torch.cuda.synchronize()
    for _ in range(5):
        for st, u, o in zip(streams, us, outs):
            s.step(u, o, 0.02 * s.dx, ch=3.0, glm_fac=0.99, stream=st)
    torch.cuda.synchronize()
    for o, r in zip(outs, ref):
        assert torch.equal(o, r)
