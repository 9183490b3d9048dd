"""Ensembles whose boxes share a stream (more boxes than lanes: 64 in FP32, 4 or 2 in FP64, where a lane's boxes also
take its scratch in turn) or a launch (small boxes of one size), runs without and with the replayed pair of
steps, odd and even numbers of steps, and a box of several slabs.  Every box must equal its own single-box run."""
import pytest
import torch

from tests.gpu_util import max_rel_err

pytestmark = pytest.mark.gpu

COURANT, CP, T = 0.3, 0.18, 0.5


def _runs(sizes, dtype, steps, graph=True, **scheme):
    """The ensemble's states and times after two runs of `steps` steps on the same buffers (the second one is
    replayed where that pays), and each box's from two single-box runs."""
    from glmmhdturb_b200 import Ensemble, Solver
    amps, seeds = [1.0 + 0.25 * (b % 7) for b in range(len(sizes))], [11 + b for b in range(len(sizes))]
    ens = Ensemble(sizes, amps=amps, seeds=seeds, dtype=dtype, courant=COURANT, turb_T=T, glm_cp_coef=CP, **scheme)
    u, w = ens.alloc(), ens.alloc()
    singles = []
    for b, n in enumerate(sizes):
        s = Solver(n, dtype=dtype, gamma=5 / 3, courant=COURANT, turb_amp=amps[b], turb_T=T, turb_ndt=100, turb_seed=seeds[b],
                   glm_cp_coef=CP, **scheme)
        s.ic_turbulent(u[b], mach=0.5 + 0.1 * (b % 6), seed=seeds[b])
        x, y = u[b].clone(), torch.empty_like(u[b])
        s.forcing_reset()
        t, r = s.run(x, y, steps, forcing=True)
        singles.append(s.run(r, y if r is x else x, steps, t0=t, forcing=True))
        s.close()
    ens.run(u, w, steps, forcing=True, graph=graph)
    if steps % 2:
        for a, b in zip(u, w):
            a.copy_(b)
    t = ens.run(u, w, steps, forcing=True, graph=graph)
    return t, (w if steps % 2 else u), singles


@pytest.mark.parametrize("steps", [3, 6])
def test_fp64_boxes_share_lanes_and_their_scratch(steps):
    """Eight uneven boxes on four lanes; the mean box is below the size from which steps are not replayed."""
    t, got, singles = _runs([32, 48, 16, 64, 32, 16, 48, 32], "f64", steps)
    for b, (ts, ref) in enumerate(singles):
        assert t[b] == ts and torch.equal(got[b], ref), b


def test_fp64_box_of_several_slabs_beside_others():
    """With four lanes a 160^3 box has three slabs; the mean box is above 48^3, so no steps are replayed."""
    t, got, singles = _runs([160, 64, 80, 96, 32], "f64", 3)
    for b, (ts, ref) in enumerate(singles):
        assert t[b] == ts and torch.equal(got[b], ref), b


def _check_f32(t, got, singles):
    for b, (ts, ref) in enumerate(singles):
        assert abs(t[b] - ts) <= 1e-6 * ts
        # other tiles than the single box's: FP32 round-off (1e-7..6e-7 after nine steps; psi, small, up to 6e-5)
        err, errs = max_rel_err(got[b].cpu().numpy(), ref.cpu().numpy())
        assert max(errs[:8]) <= 1e-5 and errs[8] <= 1e-3, (b, errs)


@pytest.mark.parametrize("steps", [4, 5])
def test_fp32_steps_that_are_not_replayed(steps):
    """A mean box above 48^3 takes plain launches, whether or not a graph is asked for."""
    _check_f32(*_runs([64, 48, 96, 64], "f32", steps))


@pytest.mark.parametrize("steps,graph", [(4, True), (5, True), (5, False)])
def test_fp32_more_boxes_than_lanes(steps, graph):
    _check_f32(*_runs([16, 32, 16, 48, 16] * 14, "f32", steps, graph))


# small boxes of one size in one launch: fewer and more than a launch takes (64), beside others; each scheme
@pytest.mark.parametrize("sizes,steps", [([16] * 5, 3), ([16] * 70 + [32], 4), ([32, 16] * 6, 5)])
def test_fp64_small_boxes_share_launches(sizes, steps):
    t, got, singles = _runs(sizes, "f64", steps)
    for b, (ts, ref) in enumerate(singles):
        assert t[b] == ts and torch.equal(got[b], ref), b


@pytest.mark.parametrize("dtype", ["f64", "f32"])
@pytest.mark.parametrize("recon,riemann", [("mc", "hll"), ("mc", "llf"), ("ppm", "hll")])
def test_schemes_of_boxes_that_share_launches(dtype, recon, riemann):
    t, got, singles = _runs([16] * 6 + [32] * 2, dtype, 3, recon=recon, riemann=riemann)
    if dtype == "f32":
        _check_f32(t, got, singles)
    else:
        for b, (ts, ref) in enumerate(singles):
            assert t[b] == ts and torch.equal(got[b], ref), b


@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_states_off_a_16_byte_boundary(dtype):
    """One box of a shared launch whose planes allow no 16-byte copies: the same values as with aligned ones."""
    from glmmhdturb_b200 import Ensemble, Solver
    sizes = [16] * 6 + [32] * 3
    out = []
    for shift in (0, 1):
        ens = Ensemble(sizes, amps=[2.0] * len(sizes), dtype=dtype, courant=COURANT, turb_T=T, glm_cp_coef=CP)
        u, w = ens.alloc(), ens.alloc()
        for b, n in enumerate(sizes):
            s = Solver(n, dtype=dtype, gamma=5 / 3)
            s.ic_turbulent(u[b], mach=0.8, seed=b)
            s.close()
        if shift:
            for b in (2, 7):
                flat = torch.empty(u[b].numel() + shift, dtype=u[b].dtype, device="cuda")[shift:].view(u[b].shape)
                u[b] = flat.copy_(u[b])
        t = ens.run(u, w, 3)
        out.append((t, w))
    assert out[0][0] == out[1][0]
    assert all(torch.equal(a, b) for a, b in zip(out[0][1], out[1][1]))


@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_buffers_exchanged_between_runs(dtype):
    """Odd runs whose result buffer is the next run's input, against one longer run: the same values, bound anew
    each time and replayed only when the same buffers come again."""
    from glmmhdturb_b200 import Ensemble, Solver
    sizes = [32, 16, 48, 32]
    out = []
    for runs in ((3, 3, 3, 3), (12,)):
        ens = Ensemble(sizes, amps=[2.0] * 4, dtype=dtype, courant=COURANT, turb_T=T, glm_cp_coef=CP)
        u, w = ens.alloc(), ens.alloc()
        for b, n in enumerate(sizes):
            s = Solver(n, dtype=dtype, gamma=5 / 3)
            s.ic_turbulent(u[b], mach=0.8, seed=b)
            s.close()
        for k in runs:
            t = ens.run(u, w, k)
            if k % 2:
                u, w = w, u
        out.append((t, u))
    # A run reduces the CFL maxima of its first state in a pass of its own: in FP64 the maxima that the step before
    # fused, in FP32 (IEEE there, approximate roots in the step) within a few 2^-24 of them, and so dt.
    (t, got), (ts, ref) = out
    if dtype == "f32":
        _check_f32(t, got, list(zip(ts, ref)))
    else:
        assert t == ts and all(torch.equal(a, b) for a, b in zip(got, ref))
