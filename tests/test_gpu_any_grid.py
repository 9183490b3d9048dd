"""Steps on grids that no tile divides (the last tiles overhang the box), on rows that are no whole
16-byte quads, on boxes smaller than a tile, and with z chunks that do not divide the box."""
import math

import numpy as np
import pytest
import torch

from tests.gpu_util import max_rel_err, perturbed_glm_state, to_dev

pytestmark = pytest.mark.gpu

TOL_F32 = 3e-5   # one FP32 step against the FP64 oracle, as the other FP32 parity tests
# below a tile; one column or row over it; one short of it; quads but no whole tile; a tile in one axis
GRIDS = [(1, 1, 1), (5, 3, 4), (33, 17, 6), (31, 15, 20), (36, 20, 9), (64, 21, 7), (97, 48, 5)]


def _dtype(name):
    return torch.float64 if name == "f64" else torch.float32


def _check(got, ref, dtype):
    if dtype == "f64":
        np.testing.assert_array_equal(got, ref)
    else:
        err, errs = max_rel_err(got.astype(np.float64), ref)
        assert err <= TOL_F32, errs


@pytest.mark.parametrize("n", GRIDS)
@pytest.mark.parametrize("recon,riem", [("mc", "hlld"), ("ppm", "hll"), ("minmod", "llf")])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_unsplit_step(oracle, n, recon, riem, dtype):
    from glmmhdturb_b200 import Solver
    u0 = perturbed_glm_state(oracle, n, seed=sum(n))
    cfg = oracle.Config(n=n, gamma=5 / 3, recon=recon, riemann=riem, iflo=True)
    f = oracle.OUForcing(amp=2.0, seed=5)
    f.advance()
    dt = 0.1 * cfg.dx
    s = Solver(n, dtype=dtype, recon=recon, riemann=riem, gamma=5 / 3, turb_T=1.0)
    s.set_modes(f.modes)
    u = to_dev(u0, _dtype(dtype))
    out = torch.full_like(u, float("nan"))
    s.step(u, out, dt, t=0.4, ch=2.0, glm_fac=0.99, do_turb=True, want_cfl=True)
    ref = oracle.step_unsplit(cfg, u0, dt, 2.0, 0.99, ramp=0.4, modes=f.modes)
    _check(out.cpu().numpy(), ref, dtype)
    cfl = s.cfl_result()
    assert np.allclose(cfl, oracle.cfl(cfg, ref), rtol=0 if dtype == "f64" else TOL_F32)


@pytest.mark.parametrize("n", GRIDS)
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_march_step(oracle, n, dtype):
    from glmmhdturb_b200 import Solver
    u0 = perturbed_glm_state(oracle, n, seed=sum(n) + 1)
    cfg = oracle.Config(n=n, gamma=5 / 3, recon="mc", riemann="hll")
    dt = 0.1 * cfg.dx
    s = Solver(n, dtype=dtype, scheme="march1d", riemann="hll", gamma=5 / 3, smallp=cfg.smallp)
    u = to_dev(u0, _dtype(dtype))
    out = torch.full_like(u, float("nan"))
    s.step(u, out, dt, ch=2.0, glm_fac=0.99)
    _check(out.cpu().numpy(), oracle.step_march1d(cfg, u0, dt, 2.0, 0.99), dtype)


@pytest.mark.parametrize("n", GRIDS)
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_ct_step(oracle, n, dtype):
    from glmmhdturb_b200 import Solver
    cfg = oracle.Config(n=n, gamma=5 / 3, riemann="hlld", emf="contact")
    q0 = oracle.ct_ic_ot(cfg)
    rng = np.random.default_rng(sum(n))
    q0[1:4] += 0.05 * rng.standard_normal(q0[1:4].shape)
    dt = 0.1 * cfg.dx
    s = Solver(n, dtype=dtype, scheme="ct", riemann="hlld", emf="contact", gamma=5 / 3)
    q = to_dev(q0, _dtype(dtype))
    out = torch.full_like(q, float("nan"))
    s.step(q, out, dt)
    ref = oracle.ct_step(cfg, q0, dt)
    if dtype == "f64":
        err, errs = max_rel_err(out.cpu().numpy(), ref)
        assert err <= 1e-12, errs
    else:
        _check(out.cpu().numpy(), ref, dtype)


@pytest.mark.parametrize("n", [(33, 17, 6), (36, 20, 9), (17, 33, 10)])
def test_fp32_record_tile_matches_cell_passes(n):
    """The FP32 adjoint's record tile on grids it overhangs against its per-cell passes."""
    from glmmhdturb_b200 import Solver
    s = Solver(n, dtype="f32", gamma=5 / 3, turb_amp=2.0, turb_T=0.5)
    u = s.alloc()
    s.ic_turbulent(u, mach=0.7, seed=2)
    s.forcing_reset()
    s.forcing_advance()
    g = torch.randn(u.shape, generator=torch.Generator().manual_seed(4)).cuda()
    got = []
    for percell in (False, True):
        s.adjoint_set_passes(percell)
        gb = torch.full_like(u, float("nan"))
        s.adjoint_step(u, g, gb, 0.02 * s.dx, t=0.1, ch=3.0, glm_fac=0.99, do_turb=True)
        got.append((gb, s.adjoint_amp_grad()))
    # the two forms round differently; a cell at a limiter kink may take either branch
    assert float((got[0][0] - got[1][0]).norm() / got[1][0].norm()) <= 3e-3
    assert math.isclose(got[0][1], got[1][1], rel_tol=1e-3)


def test_chunks_of_a_box_round_alike():
    """The z chunk is chosen by the box's size; the step does not depend on it."""
    from glmmhdturb_b200 import Solver
    a = Solver(48, dtype="f32", gamma=5 / 3)
    u = a.alloc()
    a.ic_turbulent(u, mach=1.0, seed=6)
    out = []
    for lz in (0, 1, 7, 48):
        s = a if lz == 0 else Solver(48, dtype="f32", gamma=5 / 3, tile=(16, 16, lz))
        o = torch.empty_like(u)
        s.step(u, o, 0.02 * s.dx, ch=3.0, glm_fac=0.99)
        out.append(o)
    assert torch.equal(out[1], out[2]) and torch.equal(out[1], out[3])
    assert float((out[0] - out[1]).norm() / out[1].norm()) <= 1e-6   # another tile, another kernel
