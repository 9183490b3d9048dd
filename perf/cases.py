"""The work that a program built on this library has it do, as cases that can be timed and checked.

A case is a dict of plain values.  prepare() makes its inputs on the GPU from a seed and the solver a
program would keep, run() is one pass through the public entry points, exact() the same pass in plain
torch in 64 bits.  Grids, schemes and parameters are those of the repository's benchmark, tests and
configurations, or generic sizes beside them (odd and uneven boxes).
"""
import math

import numpy as np
import torch

from glmmhdturb_b200 import Ensemble, Solver, adjoint

GAMMA, COURANT, CP, TURB_T, NDT = 5.0 / 3.0, 0.3, 0.18, 0.5, 100
SMALLR, SMALLC, SMALLP = 1e-6, 1e-4, 1e-6
PFL = SMALLR * SMALLC ** 2 / GAMMA
MIN_RHO = 1e-5
CH, SIGNAL = 5.0, 12.0      # cleaning speed and summed signal speed of the prepared states (dt = C dx / SIGNAL)
TIME = 0.1                   # time of a single step: the forcing ramp is TIME / TURB_T

# the 61 +- pairs of forcing modes, 1 <= |k|^2 <= 9, in the order the library documents
MODES = [(kx, ky, kz) for kx in range(4) for ky in range(-3, 4) for kz in range(-3, 4)
         if 1 <= kx * kx + ky * ky + kz * kz <= 9 and (kx > 0 or (kx == 0 and (ky > 0 or (ky == 0 and kz > 0))))]


# --------------------------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------------------------
def _glm(nx, ny, nz, dtype="f32", recon="mc", riemann="hlld"):
    return {"kind": "glm", "nx": nx, "ny": ny, "nz": nz, "dtype": dtype, "recon": recon, "riemann": riemann}


def _ct(nx, ny, nz, dtype="f32", recon="mc", riemann="hlld", emf="contact"):
    return {"kind": "ct", "nx": nx, "ny": ny, "nz": nz, "dtype": dtype, "recon": recon, "riemann": riemann, "emf": emf}


def _march(nx, ny, nz, dtype="f32", recon="mc", nsp=0):
    return {"kind": "march", "nx": nx, "ny": ny, "nz": nz, "dtype": dtype, "recon": recon, "nsp": nsp}


def _adjoint(nx, ny, nz, dtype="f32", recon="mc", riemann="hlld"):
    return {"kind": "adjoint", "nx": nx, "ny": ny, "nz": nz, "dtype": dtype, "recon": recon, "riemann": riemann}


def _gradient(n, steps, every, dtype="f64"):
    return {"kind": "gradient", "nx": n, "ny": n, "nz": n, "dtype": dtype, "steps": steps, "every": every}


def _loop(n, steps, dtype="f32"):
    return {"kind": "loop", "nx": n, "ny": n, "nz": n, "dtype": dtype, "steps": steps}


def _ensemble(boxes, pick, steps, largest=128, dtype="f32"):
    return {"kind": "ensemble", "boxes": boxes, "pick": pick, "steps": steps, "largest": largest, "dtype": dtype}


def _stats(nx, ny, nz, dtype="f32", kmax=8, nbins=64):
    return {"kind": "stats", "nx": nx, "ny": ny, "nz": nz, "dtype": dtype, "kmax": kmax, "nbins": nbins}


def listed():
    return [
        # the headline: a forced step of a 512^3 production box and the CFL read-back that sets the next dt
        {"name": "glm_f32_512", **_glm(512, 512, 512)},
        # the same host loop on a small box, where launches, the read-back and filling the chip count
        {"name": "glm_f32_64", **_glm(64, 64, 64)},
        # a box no tile divides
        {"name": "glm_f32_odd", **_glm(201, 135, 99)},
        # the shock-robust scheme of the Orszag-Tang runs (PPM + HLL), on an uneven box
        {"name": "ppm_f32_240", **_glm(240, 120, 120, recon="ppm", riemann="hll")},
        # double precision, as the parity runs use it
        {"name": "glm_f64_192", **_glm(192, 192, 192, dtype="f64")},
        # constrained transport with the upwind EMF
        {"name": "ct_f32_256", **_ct(256, 256, 256)},
        # the march scheme behind the bridge, with two passive species
        {"name": "march_f32_240", **_march(240, 240, 240, nsp=2)},
        # one reverse step of a gradient run
        {"name": "adjoint_f32_128", **_adjoint(128, 128, 128)},
        # a whole gradient: checkpointed forward run, band loss, reverse sweep
        {"name": "gradient_f64_64", **_gradient(64, 6, 3)},
        # the device-resident loop: many small steps in one call
        {"name": "loop_f32_64", **_loop(64, 20)},
        # an ensemble of 64 uneven boxes advanced together
        {"name": "ensemble_64", **_ensemble(64, 2024, 4)},
        # the analysis of a snapshot: diagnostics, kinetic-energy spectrum, density PDF
        {"name": "stats_f32_256", **_stats(256, 256, 256)},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi):
    """Three sizes around a base spread over its logarithm: a cube of whole tiles, an uneven box of
    whole quads, or any sizes."""
    base, shape = _log(rng, lo, hi), rng.choice(("cube", "quads", "any"))
    if shape == "cube":
        n = max(16, 16 * round(base / 16))
        return n, n, n
    axes = [max(lo, min(hi, int(base * rng.uniform(0.6, 1.25)))) for _ in range(3)]
    return tuple(4 * max(1, n // 4) for n in axes) if shape == "quads" else tuple(axes)


def draw(rng):
    kind = rng.choice(("glm", "glm", "glm64", "ct", "march", "adjoint", "gradient", "loop", "ensemble", "stats"))
    dtype = rng.choice(("f32", "f32", "f64"))
    if kind == "glm":
        return _glm(*_grid(rng, 16, 400), recon=rng.choice(("mc", "mc", "minmod", "ppm")),
                    riemann=rng.choice(("hlld", "hlld", "hll", "llf")))
    if kind == "glm64":
        return _glm(*_grid(rng, 16, 200), dtype="f64", recon=rng.choice(("mc", "mc", "ppm")),
                    riemann=rng.choice(("hlld", "hll")))
    if kind == "ct":
        return _ct(*_grid(rng, 16, 160 if dtype == "f64" else 288), dtype=dtype, recon=rng.choice(("mc", "ppm")),
                   riemann=rng.choice(("hlld", "hll")), emf=rng.choice(("contact", "average")))
    if kind == "march":
        return _march(*_grid(rng, 16, 160 if dtype == "f64" else 320), dtype=dtype, recon=rng.choice(("mc", "ppm")),
                      nsp=rng.choice((0, 0, 1, 2, 3)))
    if kind == "adjoint":
        return _adjoint(*_grid(rng, 16, 96 if dtype == "f64" else 160), dtype=dtype, recon=rng.choice(("mc", "minmod")),
                        riemann=rng.choice(("hlld", "hlld", "hll")))
    if kind == "gradient":
        return _gradient(rng.randrange(20, 65), rng.randrange(2, 7), rng.randrange(2, 4))
    if kind == "loop":
        return _loop(rng.randrange(16, 129), rng.randrange(4, 33), dtype=rng.choice(("f32", "f64")))
    if kind == "ensemble":
        return _ensemble(_log(rng, 4, 64), rng.randrange(1 << 20), rng.randrange(2, 5), largest=rng.choice((64, 96)),
                         dtype=rng.choice(("f32", "f32", "f64")))
    return _stats(*_grid(rng, 24, 288), dtype=dtype, kmax=rng.choice((4, 8, 8)), nbins=rng.choice((32, 64, 200)))


def _sizes(case):
    """Box sizes, Mach numbers and plasma betas of an ensemble."""
    r = np.random.default_rng(case["pick"])
    sizes = r.choice([s for s in (32, 48, 64, 96, 128) if s <= case["largest"]], size=case["boxes"])
    return [int(n) for n in sizes], r.uniform(0.3, 3.0, size=case["boxes"]), r.uniform(0.1, 10.0, size=case["boxes"])


# --------------------------------------------------------------------------------------------
# inputs: a turbulent state as a run meets it (broad-band velocity, density and field, rms Mach 1,
# a little grid-scale structure)
# --------------------------------------------------------------------------------------------
def _dtype(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _fields(count, n, gen, waves=24):
    """`count` unit-rms random fields (float32): plane waves with |k| up to a sixth of the grid, power
    falling with k, plus 1 % noise."""
    nx, ny, nz = n
    top = max(2.0, min(n) / 6.0)
    out = torch.empty((count, nz, ny, nx), device="cuda")
    for f in out:
        k = torch.exp(torch.rand(waves, generator=gen, device="cuda") * math.log(top))
        d = torch.randn((3, waves), generator=gen, device="cuda")
        d = torch.round(k * d / d.norm(dim=0))
        amp = torch.randn(waves, generator=gen, device="cuda") * k ** -0.8
        ph = torch.rand(waves, generator=gen, device="cuda") * (2 * math.pi)
        ax = [2 * math.pi * (torch.arange(m, device="cuda") + 0.5) / m for m in n]
        a = d[0][:, None] * ax[0]
        b = d[1][:, None] * ax[1] + ph[:, None]
        ab = b[:, :, None] + a[:, None, :]
        c = d[2][:, None] * ax[2]
        f.copy_(((amp[:, None] * torch.cos(c)).T @ torch.cos(ab).reshape(waves, -1)
                 - (amp[:, None] * torch.sin(c)).T @ torch.sin(ab).reshape(waves, -1)).reshape(nz, ny, nx))
        f.div_(f.std() + 1e-6)
        f.add_(torch.randn(f.shape, generator=gen, device="cuda"), alpha=0.01)
    return out


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _state(n, seed, dtype, mach=1.0, b0=0.775, species=0, out=None):
    """9 conserved planes of the GLM state, then rho*X of each species."""
    nx, ny, nz = n
    g = _gen(seed)
    u = torch.empty((9 + species, nz, ny, nx), dtype=dtype, device="cuda") if out is None else out
    f = _fields(9, n, g)
    rho = torch.exp(0.3 * f[0])
    v = f[1:4] * (mach / math.sqrt(3.0))
    b = f[4:7] * 0.15
    b[0] += b0
    p = 0.6 * torch.exp(0.2 * f[7])
    u[0].copy_(rho)
    for i in range(3):
        u[1 + i].copy_(rho * v[i])
        u[5 + i].copy_(b[i])
    u[4].copy_(p / (GAMMA - 1.0) + 0.5 * rho * (v * v).sum(0) + 0.5 * (b * b).sum(0))
    u[8].copy_(0.02 * f[8])
    if species:
        for i, x in enumerate(_fields(species, n, g)):
            u[9 + i].copy_(rho * (0.5 + 0.15 * x).clamp(0.0, 1.0))
    return u


def _ct_state(n, seed, dtype):
    """[rho, m, E, bxf, byf, bzf]: the face field is the curl of an edge potential."""
    nx, ny, nz = n
    u = _state(n, seed, dtype)
    a = _fields(3, n, _gen(seed + 1)).to(dtype) * (0.15 / (2 * math.pi * 3))
    q = torch.empty((8, nz, ny, nx), dtype=dtype, device="cuda")
    fwd = lambda f, d: torch.roll(f, -1, (2, 1, 0)[d]) - f  # noqa: E731
    b = [fwd(a[2], 1) * ny - fwd(a[1], 2) * nz, fwd(a[0], 2) * nz - fwd(a[2], 0) * nx, fwd(a[1], 0) * nx - fwd(a[0], 1) * ny]
    b[0] = b[0] + 0.775
    m = u[5:8]
    ek = u[4] - 0.5 * (m * m).sum(0)
    q[:4].copy_(u[:4])
    q[4].copy_(ek)
    for d in range(3):
        q[5 + d].copy_(b[d])
        c = 0.5 * (b[d] + torch.roll(b[d], -1, (2, 1, 0)[d]))
        q[4].add_(0.5 * c * c)
    return q


def _modes(seed):
    """Solenoidal forcing modes of unit rms acceleration, [61][3][2]."""
    r = np.random.default_rng(int(seed) + 99)
    k = np.array(MODES, dtype=float)
    kk = np.sqrt((k * k).sum(1))
    z = r.standard_normal((61, 3, 2))
    z -= (k / kk[:, None])[:, :, None] * np.einsum("mi,mic->mc", k / kk[:, None], z)[:, None, :]
    z /= kk[:, None, None]
    return z / math.sqrt(2.0 * (z * z).sum())


def _solver(case, seed, **kw):
    n = (case["nx"], case["ny"], case["nz"])
    return Solver(n, dtype=case["dtype"], gamma=GAMMA, courant=COURANT, smallr=SMALLR, smallc=SMALLC, smallp=SMALLP,
                  glm_cp_coef=CP, turb_T=TURB_T, turb_ndt=NDT, turb_amp=2.0, turb_seed=1 + int(seed) % 1000003, **kw)


def _dt(case):
    return COURANT / case["nx"] / SIGNAL


def prepare(case, seed):
    kind, dtype = case["kind"], _dtype(case)
    st = {"case": case}
    if kind == "ensemble":
        sizes, mach, beta = _sizes(case)
        ens = Ensemble(sizes, amps=[2.0 * m for m in mach], seeds=[int(seed) % 1000003 + i for i in range(len(sizes))],
                       dtype=case["dtype"], gamma=GAMMA, courant=COURANT, turb_T=TURB_T, turb_ndt=NDT, glm_cp_coef=CP,
                       smallr=SMALLR, smallc=SMALLC)
        flat = [torch.empty(9 * sum(n ** 3 for n in sizes), dtype=dtype, device="cuda") for _ in range(3)]
        views, at = [[], [], []], 0
        for b, n in enumerate(sizes):
            for f, v in zip(flat, views):
                v.append(f[at:at + 9 * n ** 3].view(9, n, n, n))
            at += 9 * n ** 3
            _state((n, n, n), seed + 31 * b, dtype, mach=float(mach[b]), b0=math.sqrt(1.2 / beta[b]), out=views[0][b])
        st.update(ens=ens, u0=flat[0], flat=flat, u=views[1], w=views[2])
        return st
    n = (case["nx"], case["ny"], case["nz"])
    if kind == "glm":
        st.update(s=_solver(case, seed, recon=case["recon"], riemann=case["riemann"]), u=_state(n, seed, dtype))
        st["s"].set_modes(2.0 * _modes(seed))
        st["w"] = torch.empty_like(st["u"])
    elif kind == "ct":
        st.update(s=_solver(case, seed, scheme="ct", recon=case["recon"], riemann=case["riemann"], emf=case["emf"]),
                  u=_ct_state(n, seed, dtype))
        st["s"].set_modes(2.0 * _modes(seed))
        st["w"] = torch.empty_like(st["u"])
    elif kind == "march":
        st.update(s=_solver(case, seed, scheme="march1d", recon=case["recon"], riemann="hll", nsp=case["nsp"]),
                  u=_state(n, seed, dtype, species=case["nsp"]))
        st["w"] = torch.empty_like(st["u"])
    elif kind == "adjoint":
        st.update(s=_solver(case, seed, recon=case["recon"], riemann=case["riemann"]), u=_state(n, seed, dtype))
        st["s"].set_modes(2.0 * _modes(seed))
        st["g"] = _fields(9, n, _gen(seed + 5)).to(dtype)
        st["w"] = torch.empty_like(st["u"])
    elif kind == "gradient":
        st.update(s=_solver(case, seed), u=_state(n, seed, dtype))
    elif kind == "loop":
        st.update(s=_solver(case, seed), u0=_state(n, seed, dtype))
        st["u"], st["w"] = torch.empty_like(st["u0"]), torch.empty_like(st["u0"])
        st["forcing"] = st["s"].forcing_state()
    else:
        st.update(s=_solver(case, seed), u=_state(n, seed, dtype))
    return st


# --------------------------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------------------------
def _f64(v):
    """Numbers of a result as 64-bit values."""
    if isinstance(v, dict):
        return {k: _f64(x) for k, x in v.items()}
    return np.float64(v) if isinstance(v, float) else v


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ensemble":
        state["flat"][1].copy_(state["u0"])
        t = state["ens"].run(state["u"], state["w"], case["steps"], forcing=True)
        return {"u": state["flat"][1 + case["steps"] % 2], "t": np.array(t)}
    s = state["s"]
    if kind in ("glm", "ct"):
        # a step of the host loop: the step with the next step's CFL fused, then its read-back
        dt = _dt(case)
        s.step(state["u"], state["w"], dt, t=TIME, ch=CH, glm_fac=s.glm_fac(CH, dt), do_turb=True, want_cfl=True)
        return {"u": state["w"], "cfl": np.array(s.cfl_result())}
    if kind == "march":
        # the bridge's step: dt and the cleaning parameters fixed by the caller
        dt = _dt(case)
        s.step(state["u"], state["w"], dt, ch=CH, glm_fac=s.glm_fac(CH, dt))
        return {"u": state["w"]}
    if kind == "adjoint":
        dt = _dt(case)
        s.adjoint_step(state["u"], state["g"], state["w"], dt, t=TIME, ch=CH, glm_fac=s.glm_fac(CH, dt), do_turb=True)
        return {"ubar": state["w"], "amp": np.float64(s.adjoint_amp_grad(reset=True))}
    if kind == "gradient":
        r = adjoint.ke_band_gradient(s, state["u"], case["steps"], kmin=4, kmax=8, checkpoint_every=case["every"])
        return {"loss": _f64(r["loss"]), "grad": r["grad_u0"], "amp": _f64(r["grad_amp"]), "u": r["u_final"]}
    if kind == "loop":
        state["u"].copy_(state["u0"])
        s.set_forcing_state(state["forcing"])
        t, u = s.run(state["u"], state["w"], case["steps"], forcing=True)
        return {"t": _f64(t), "u": u}
    d = s.diagnostics(state["u"])
    pdf, st = s.density_pdf(state["u"], nbins=case["nbins"], smin=-2.0, smax=2.0)
    return {"diag": _f64(d), "spectrum": s.ke_spectrum(state["u"], kmax=case["kmax"]), "pdf": pdf, "moments": _f64(st)}


# --------------------------------------------------------------------------------------------
# the work of a pass: every state read once and written once; flops of the scheme, counted from its
# formulas (a square root or a division as one)
# --------------------------------------------------------------------------------------------
FLOPS = {"glm": 1900.0, "ct": 2200.0, "march": 1900.0, "adjoint": 6500.0}


def work(case):
    size = 8 if case["dtype"] == "f64" else 4
    if case["kind"] == "ensemble":
        cells = sum(n ** 3 for n in _sizes(case)[0])
        # the pass restores its start (one copy), then steps
        return {"bytes": 18.0 * size * cells * (case["steps"] + 1), "flops": FLOPS["glm"] * cells * case["steps"]}
    cells = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "glm":
        return {"bytes": 18.0 * size * cells, "flops": FLOPS["glm"] * cells}
    if case["kind"] == "ct":
        return {"bytes": 16.0 * size * cells, "flops": FLOPS["ct"] * cells}
    if case["kind"] == "march":
        return {"bytes": (18.0 + 2 * case["nsp"]) * size * cells, "flops": (FLOPS["march"] + 150 * case["nsp"]) * cells}
    if case["kind"] == "adjoint":
        return {"bytes": 27.0 * size * cells, "flops": FLOPS["adjoint"] * cells}
    if case["kind"] == "gradient":
        # per step: the forward step, its recomputation and the reverse step; the loss reads the state
        # and writes its gradient
        return {"bytes": (63.0 * case["steps"] + 13) * size * cells,
                "flops": (2 * FLOPS["glm"] + FLOPS["adjoint"]) * cells * case["steps"]}
    if case["kind"] == "loop":
        return {"bytes": 18.0 * size * cells * (case["steps"] + 1), "flops": FLOPS["glm"] * cells * case["steps"]}
    # the state once (diagnostics); the spectrum and the PDF read planes of it again
    return {"bytes": (9.0 + 4 + 1) * size * cells, "flops": (40.0 + 12 * 2 * math.log2(cells)) * cells}


def tolerance(case):
    """About four times what the passes show against exact() over listed and drawn cases."""
    f64 = case["dtype"] == "f64"
    kind = case["kind"]
    if kind == "stats":                       # sums in 64 bits whatever the state's type
        return {"rel": 1e-12, "max": 1e-11}
    if kind in ("adjoint", "gradient"):
        # derivatives of limiter and fan branches: a cell at a switch may take either side (seen: 9e-4,
        # one value by its own size, in 32 bits; 4.8e-6 and 3.8e-3 in 64)
        return {"rel": 2e-5, "max": 1.5e-2} if f64 else {"rel": 4e-3, "max": 0.99}
    if kind in ("loop", "ensemble"):          # seen: 3.3e-7, one value 5e-4; in 64 bits 1.6e-14, 5e-13
        return {"rel": 6e-14, "max": 2e-12} if f64 else {"rel": 1.5e-6, "max": 2e-3}
    if f64:                                   # seen: 1.2e-16, one value 7e-14
        return {"rel": 1e-15, "max": 3e-13}
    return {"rel": 4e-7, "max": 2e-3}         # seen: 1.1e-7, one value 5e-4


# --------------------------------------------------------------------------------------------
# the same passes in plain torch, 64 bits
# --------------------------------------------------------------------------------------------
AXIS = (3, 2, 1)            # tensor axis of x, y, z in a (variable, z, y, x) tensor
TO = ((0, 1, 2, 3, 4, 5, 6, 7, 8), (0, 2, 3, 1, 4, 6, 7, 5, 8), (0, 3, 1, 2, 4, 7, 5, 6, 8))
FROM = (TO[0], TO[2], TO[1])


def _back(f, d):
    return torch.roll(f, 1, AXIS[d])


def _ahead(f, d):
    return torch.roll(f, -1, AXIS[d])


def _prim(c, pf):
    rho = c[0].clamp(min=SMALLR)
    v = c[1:4] / rho
    p = (GAMMA - 1) * (c[4] - 0.5 * (c[1:4] ** 2).sum(0) / rho - 0.5 * (c[5:8] ** 2).sum(0))
    return torch.cat([rho[None], v, p.clamp(min=pf)[None], c[5:9]])


def _cons(q):
    e = q[4] / (GAMMA - 1) + 0.5 * q[0] * (q[1:4] ** 2).sum(0) + 0.5 * (q[5:8] ** 2).sum(0)
    return torch.cat([q[:1], q[0] * q[1:4], e[None], q[5:9]])


def _flux(q):
    rho, vx, vy, vz, p, bx, by, bz = q[:8].unbind(0)
    b2 = bx * bx + by * by + bz * bz
    pt = p + 0.5 * b2
    e = p / (GAMMA - 1) + 0.5 * rho * (vx * vx + vy * vy + vz * vz) + 0.5 * b2
    vb = vx * bx + vy * by + vz * bz
    zero = torch.zeros_like(rho)
    return torch.stack([rho * vx, rho * vx * vx + pt - bx * bx, rho * vx * vy - bx * by, rho * vx * vz - bx * bz,
                        (e + pt) * vx - bx * vb, zero, vx * by - vy * bx, vx * bz - vz * bx, zero])


def _dir_flux(q, d):
    return _flux(q[list(TO[d])])[list(FROM[d])]


def _slope(q, d, recon):
    """Half slope along d (MonCen, or minmod)."""
    dl, dr = q - _back(q, d), _ahead(q, d) - q
    if recon == "minmod":
        s = 0.5 * torch.where(dl.abs() < dr.abs(), dl, dr)
    else:
        dc = 0.5 * (dl + dr)
        s = 0.5 * torch.sign(dc) * torch.minimum(2 * torch.minimum(dl.abs(), dr.abs()), dc.abs())
    return torch.where(dl * dr <= 0, torch.zeros_like(s), s)


def _ppm(q, d):
    qm, qp = _back(q, d), _ahead(q, d)
    sl, curve = 0.25 * (qp - qm), (qm - 2 * q + qp) / 12
    ql, qr = q - sl + curve, q + sl + curve
    dq = qr - ql
    diff, lim = (q - 0.5 * (ql + qr)) * dq, dq * dq / 6
    lo = torch.where(diff > lim, 3 * q - 2 * qr, ql)
    hi = torch.where(diff < -lim, 3 * q - 2 * ql, qr)
    flat = (qr - q) * (q - ql) <= 0
    return torch.where(flat, q, lo), torch.where(flat, q, hi)


def _root(x):
    return torch.sqrt(x.clamp(min=1e-300))


def _fast(q, bn):
    c2 = GAMMA * q[4] / q[0]
    d2 = 0.5 * ((q[5] ** 2 + q[6] ** 2 + q[7] ** 2) / q[0] + c2)
    return torch.sqrt(d2 + _root(d2 * d2 - c2 * bn * bn / q[0]))


def _llf(L, R, ch):
    s = torch.maximum(L[1].abs() + _fast(L, L[5]), R[1].abs() + _fast(R, R[5])).clamp(min=ch)
    return 0.5 * (_flux(L) + _flux(R)) - 0.5 * s * (_cons(R) - _cons(L))


def _hll(L, R, bn):
    a, b = _fast(L, bn), _fast(R, bn)
    sl = torch.minimum(L[1] - a, R[1] - b).clamp(max=0)
    sr = torch.maximum(L[1] + a, R[1] + b).clamp(min=0)
    return (sr * _flux(L) - sl * _flux(R) + sl * sr * (_cons(R) - _cons(L))) / (sr - sl)


def _hlld(L, R, bn):
    """Miyoshi & Kusano (2005)."""
    def side(q):
        d, u, v, w, p = q[:5].unbind(0)
        by, bz = q[6], q[7]
        b2 = bn * bn + by * by + bz * bz
        return d, u, v, w, p + 0.5 * b2, by, bz, p / (GAMMA - 1) + 0.5 * d * (u * u + v * v + w * w) + 0.5 * b2

    dl, ul, vl, wl, ptl, byl, bzl, el = side(L)
    dr, ur, vr, wr, ptr, byr, bzr, er = side(R)
    c = torch.maximum(_fast(L, bn), _fast(R, bn))
    sl = (torch.minimum(ul, ur) - c).clamp(max=0)
    sr = (torch.maximum(ul, ur) + c).clamp(min=0)
    al, ar = (sl - ul) * dl, (sr - ur) * dr
    den = ar - al
    sm = (ar * ur - al * ul - ptr + ptl) / den
    pts = (ar * ptl - al * ptr + ar * al * (ur - ul)) / den
    dls, drs = (al / (sl - sm)).clamp(min=1e-12), (ar / (sr - sm)).clamp(min=1e-12)
    ql, qr = torch.sqrt(dls), torch.sqrt(drs)
    sls, srs = sm - bn.abs() / ql, sm + bn.abs() / qr

    def star(d, u, v, w, pt, by, bz, e, s):
        k = d * (s - u) * (s - sm) - bn * bn
        tiny = k.abs() < 1e-12
        k = torch.where(tiny, torch.ones_like(k), k)
        fac, t = bn * (sm - u) / k, (d * (s - u) ** 2 - bn * bn) / k
        vs, ws = torch.where(tiny, v, v - by * fac), torch.where(tiny, w, w - bz * fac)
        bs, cs = torch.where(tiny, by, by * t), torch.where(tiny, bz, bz * t)
        vb, vbs = u * bn + v * by + w * bz, sm * bn + vs * bs + ws * cs
        return vs, ws, bs, cs, vbs, ((s - u) * e - pt * u + pts * sm + bn * (vb - vbs)) / (s - sm)

    vls, wls, bls, cls, vbl, els = star(dl, ul, vl, wl, ptl, byl, bzl, el, sl)
    vrs, wrs, brs, crs, vbr, ers = star(dr, ur, vr, wr, ptr, byr, bzr, er, sr)
    sg = torch.where(bn >= 0, torch.ones_like(bn), -torch.ones_like(bn))
    inv = 1 / (ql + qr)
    vss = (ql * vls + qr * vrs + (brs - bls) * sg) * inv
    wss = (ql * wls + qr * wrs + (crs - cls) * sg) * inv
    bss = (ql * brs + qr * bls + ql * qr * (vrs - vls) * sg) * inv
    css = (ql * crs + qr * cls + ql * qr * (wrs - wls) * sg) * inv
    vbs = sm * bn + vss * bss + wss * css
    zero = torch.zeros_like(bn)

    def pack(d, u, v, w, e, by, bz):
        return torch.stack([d, d * u, d * v, d * w, e, bn, by, bz, zero])

    def fan(q, U, Us, Uss, s, ss):
        f = _flux(torch.cat([q[:5], bn[None], q[6:8], zero[None]]))
        return f + s * (Us - U), f + ss * Uss - (ss - s) * Us - s * U

    fl, fll = fan(L, pack(dl, ul, vl, wl, el, byl, bzl), pack(dls, sm, vls, wls, els, bls, cls),
                  pack(dls, sm, vss, wss, els - ql * (vbl - vbs) * sg, bss, css), sl, sls)
    fr, frr = fan(R, pack(dr, ur, vr, wr, er, byr, bzr), pack(drs, sm, vrs, wrs, ers, brs, crs),
                  pack(drs, sm, vss, wss, ers + qr * (vbr - vbs) * sg, bss, css), sr, srs)
    return torch.where(sls >= 0, fl, torch.where(srs < 0, fr, torch.where(sm >= 0, fll, frr)))


def _riemann(L, R, d, riemann, ch):
    """Flux at a face of direction d, with Dedner's pair (ch None: a given normal field, no cleaning)."""
    L, R = L[list(TO[d])], R[list(TO[d])]
    if ch is None:
        bn, f5, f8 = L[5], torch.zeros_like(L[5]), torch.zeros_like(L[5])
    else:
        bn = 0.5 * (L[5] + R[5]) - 0.5 * (R[8] - L[8]) / ch
        f5, f8 = 0.5 * (L[8] + R[8]) - 0.5 * ch * (R[5] - L[5]), ch * ch * bn
        L, R = (torch.cat([q[:5], bn[None], q[6:]]) for q in (L, R))
    f = _hll(L, R, bn) if riemann == "hll" else _llf(L, R, ch) if riemann == "llf" else _hlld(L, R, bn)
    f = torch.cat([f[:5], f5[None], f[6:8], f8[None]])
    return f[list(FROM[d])]


def _floor(q, pf):
    return torch.cat([q[:1].clamp(min=SMALLR), q[1:4], q[4:5].clamp(min=pf), q[5:]])


def _finish(r, fac, acc, dt):
    """Void floor, psi damping, forcing kick with its energy floors."""
    void = r[0] < SMALLR
    e0 = PFL / (GAMMA - 1) + 0.5 * (r[5:8] ** 2).sum(0)
    rho = torch.where(void, torch.full_like(r[0], SMALLR), r[0])
    m = [torch.where(void, torch.zeros_like(r[0]), x) for x in r[1:4]]
    e = torch.where(void, e0, r[4])
    if acc is not None:
        on, fl, ek = rho >= MIN_RHO, rho * SMALLC ** 2, e
        for x in m:
            ek = torch.maximum(ek - 0.5 * x * x / rho, fl)
        k = [x + rho * a * dt for x, a in zip(m, acc)]
        for x in k:
            ek = torch.maximum(ek + 0.5 * x * x / rho, fl)
        m = [torch.where(on, y, x) for x, y in zip(m, k)]
        e = torch.where(on, ek, e)
    return torch.stack([rho, *m, e, r[5], r[6], r[7], r[8] * fac])


def _unsplit(u, dx, dt, ch, fac, recon, riemann, acc):
    h = dt / dx
    m0 = _prim(u, PFL)
    s = [_slope(m0, d, recon) for d in range(3)]
    div = sum(_dir_flux(m0 + s[d], d) - _dir_flux(m0 - s[d], d) for d in range(3))
    mh = _prim(_cons(m0) - 0.5 * h * div, PFL)
    mh = torch.where((mh[0] <= SMALLR) | (mh[4] <= PFL), m0, mh)
    r = u
    if recon == "ppm":
        up = torch.ones_like(m0[0], dtype=torch.bool)
        for d in range(3):
            p = m0[4:5]
            a, b = _back(p, d), _ahead(p, d)
            hi = torch.maximum(p, torch.maximum(a, b))
            lo = torch.minimum(p, torch.minimum(a, b)).clamp(min=1e-20)
            up = up & ~(hi / lo > 2)[0]
    for d in range(3):
        hi, lo = mh + s[d], mh - s[d]
        if recon == "ppm":
            el, eh = _ppm(m0, d)
            hi, lo = torch.where(up, mh + eh - m0, hi), torch.where(up, mh + el - m0, lo)
        hi, lo = (torch.where((f[0] < SMALLR) | (f[4] < PFL), m0, f) for f in (hi, lo))
        f = _riemann(_floor(hi, PFL), _floor(_ahead(lo, d), PFL), d, riemann, ch)
        r = r + h * (_back(f, d) - f)
    return _finish(r, fac, acc, dt)


def _full(q, d):
    a, c = _back(q, d), _ahead(q, d)
    dl, dr, dc = q - a, c - q, 0.5 * (c - a)
    s = torch.sign(dl) * torch.minimum(dc.abs(), 2 * torch.minimum(dl.abs(), dr.abs()))
    return torch.where(dl * dr <= 0, torch.zeros_like(s), s)


def _hancock1d(q, s, d, h):
    return _prim(_cons(q) - 0.5 * h * (_dir_flux(q + 0.5 * s, d) - _dir_flux(q - 0.5 * s, d)), SMALLP)


def _march_faces(m0, d, h, recon):
    s = _full(m0, d)
    mh = _hancock1d(m0, s, d, h)
    if recon == "ppm":
        lo, hi = _ppm(m0, d)
        return hi + mh - m0, lo + mh - m0
    return mh + 0.5 * s, mh - 0.5 * s


def _march_step(u, dx, dt, ch, fac, recon, nsp):
    h = dt / dx
    m0 = _prim(u[:9], SMALLP)
    r, x = u[:9], u[9:] / u[0].clamp(min=SMALLR)
    rx = u[9:]
    for d in range(3):
        hi, lo = (_floor(f, SMALLP) for f in _march_faces(m0, d, h, recon))
        f = _riemann(hi, _ahead(lo, d), d, "hll", ch)
        r = r + h * (_back(f, d) - f)
        if nsp:
            s = _full(x, d)
            un = u[1 + d] / u[0].clamp(min=SMALLR)
            xh = x - 0.5 * h * un * s
            if recon == "ppm":
                el, eh = _ppm(x, d)
                xhi, xlo = eh + xh - x, el + xh - x
            else:
                xhi, xlo = xh + 0.5 * s, xh - 0.5 * s
            g = torch.where(f[0] >= 0, f[0] * xhi, f[0] * _ahead(xlo, d))
            rx = rx + h * (_back(g, d) - g)
    return torch.cat([r[:8], r[8:9] * fac, rx])


def _upwind(f, minus, plus):
    return torch.where(f > 0, minus, torch.where(f < 0, plus, 0.5 * (minus + plus)))


def _ct_cells(q):
    b = torch.stack([0.5 * (q[5 + d] + _ahead(q[5 + d:6 + d], d)[0]) for d in range(3)])
    return torch.cat([q[:5], b, torch.zeros_like(q[:1])])


def _ct_step(q, dx, dt, recon, riemann, emf, acc):
    h = dt / dx
    c = _ct_cells(q)
    m0 = _prim(c, SMALLP)
    r, flux = c, []
    for d in range(3):
        hi, lo = (_floor(f, SMALLP) for f in _march_faces(m0, d, h, recon))
        bn = q[5 + d:6 + d]                              # field of the lower face
        put = lambda f, b: torch.cat([f[:5 + d], b, f[6 + d:8], torch.zeros_like(b)])  # noqa: E731
        f = _riemann(put(_back(hi, d), bn), put(lo, bn), d, riemann, None)
        flux.append(f)                                   # at the lower face of each cell
        r = r + h * (f - _ahead(f, d))
    r = _finish(torch.cat([r[:5], c[5:]]), 1.0, acc, dt)
    v, b = m0[1:4], m0[5:8]
    out = [r[:5]]
    edge = []
    for e in range(3):
        i, j = (e + 1) % 3, (e + 2) % 3                  # the two axes across the edge
        ec = -(v[i] * b[j] - v[j] * b[i])[None]
        ea, eb = -flux[i][5 + j:6 + j], flux[j][5 + i:6 + i]
        ma, mb = flux[i][:1], flux[j][:1]
        ean, eas, ebe, ebw = ea, _back(ea, j), eb, _back(eb, i)
        emean = 0.25 * (ebe + ebw + ean + eas)
        if emf == "contact":
            e00, e10, e01 = ec, _back(ec, i), _back(ec, j)
            e11 = _back(e10, j)
            dn = _upwind(ma, e10 - ebw, e00 - ebe)
            ds = _upwind(_back(ma, j), ebw - e11, ebe - e01)
            de = _upwind(mb, e01 - eas, e00 - ean)
            dw = _upwind(_back(mb, i), eas - e11, ean - e10)
            emean = emean + 0.25 * (ds - dn) + 0.25 * (dw - de)
        edge.append(emean)
    for d in range(3):
        i, j = (d + 1) % 3, (d + 2) % 3
        out.append(q[5 + d:6 + d] - h * ((_ahead(edge[j], i) - edge[j]) - (_ahead(edge[i], j) - edge[i])))
    return torch.cat(out)


def _accel(modes, n, z, ramp):
    """The forcing acceleration on the planes z: ramp * sum over the +- pairs of 2 Re(a e^{2 pi i k.x})."""
    k = torch.tensor(MODES, dtype=torch.float64, device="cuda")
    ph = [torch.exp(2j * math.pi * k[:, a:a + 1] * (torch.arange(n[a], device="cuda", dtype=torch.float64) + 0.5) / n[a])
          for a in range(3)]
    plane = (ph[1][:, :, None] * ph[0][:, None, :]).reshape(61, -1)
    a = torch.complex(*torch.as_tensor(modes, dtype=torch.float64, device="cuda").unbind(-1))
    out = [((a[:, i:i + 1] * ph[2][:, z]).T @ plane).real.reshape(len(z), n[1], n[0]) for i in range(3)]
    return 2.0 * ramp * torch.stack(out)


def _speeds(c):
    q = _prim(c, PFL)
    s = [q[1 + d].abs() + _fast(q, q[5 + d]) for d in range(3)]
    return float((s[0] + s[1] + s[2]).max()), float(torch.stack(s).max())


def _slabs(n, ghost, thick=None):
    """(planes of a slab with its ghosts, planes of the slab)."""
    nx, ny, nz = n
    thick = thick or max(1, min(nz, (1 << 22) // (nx * ny)))
    for z0 in range(0, nz, thick):
        z1 = min(nz, z0 + thick)
        yield torch.arange(z0 - ghost, z1 + ghost, device="cuda") % nz, torch.arange(z0, z1, device="cuda")


def _sweep(u, n, ghost, f, modes=None, ramp=0.0):
    """f(slab of u with ghosts in 64 bits, acceleration on it) over all slabs."""
    out = torch.empty(u.shape, dtype=torch.float64, device="cuda")
    for ext, own in _slabs(n, ghost):
        acc = None if modes is None else _accel(modes, n, ext, ramp)
        out[:, own] = f(u[:, ext].double(), acc)[:, ghost:ghost + len(own)]
    return out


def _max_speeds(u, n, cells=None):
    m = []
    for ext, own in _slabs(n, 1):
        c = u[:, ext].double()
        m.append(_speeds((cells(c) if cells else c)[:, 1:1 + len(own)]))
    return tuple(max(x) for x in zip(*m))


def _fac(ch, dt):
    return math.exp(-ch / CP * dt)


def _philox(counter, key):
    """Philox4x32-10 (Salmon et al., SC'11) of arrays of counters, [4][n]."""
    c = [np.asarray(x, dtype=np.uint64) for x in counter]
    k0, k1 = int(key[0]), int(key[1])
    mask = np.uint64(0xFFFFFFFF)
    for _ in range(10):
        a, b = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & mask, (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), a & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _ou(modes, seed, counter, amp):
    """One Ornstein-Uhlenbeck update of the solenoidal modes."""
    dtf = TURB_T / NDT
    alpha, beta = 1.0 - dtf / TURB_T, math.sqrt(2.0 * dtf / TURB_T)
    k = np.array(MODES, dtype=float)
    kk = np.sqrt((k * k).sum(1))
    sig = amp * math.sqrt((1 - alpha * alpha) / (8 * beta * beta * (1 / kk ** 2).sum()))
    q = np.arange(61)
    r = []
    for part in (0, 1):
        r += _philox([np.full(61, counter), q, np.full(61, part), np.zeros(61, dtype=int)], (seed, 0x9E3779B9))
    z = np.empty((61, 3, 2))
    for i in range(3):
        u1, u2 = ((r[2 * i + j].astype(float) + 0.5) * 2.0 ** -32 for j in (0, 1))
        z[:, i, 0] = np.sqrt(-2 * np.log(u1)) * np.cos(2 * math.pi * u2)
        z[:, i, 1] = np.sqrt(-2 * np.log(u1)) * np.sin(2 * math.pi * u2)
    khat = k / kk[:, None]
    z -= khat[:, :, None] * np.einsum("mi,mic->mc", khat, z)[:, None, :]
    return alpha * modes + beta * (sig / kk)[:, None, None] * z


def _clock(u, n, seed, amp, steps, step):
    """The driver's loop: forcing updates on their cadence, dt from the CFL maxima, ch the largest signal
    speed; step(u, i, dt, ch, fac, modes, ramp) advances."""
    t, due, counter, modes = 0.0, 0.0, 0, np.zeros((61, 3, 2))
    for i in range(steps):
        if t >= due:
            modes, counter, due = _ou(modes, seed, counter, amp), counter + 1, due + TURB_T / NDT
        ctot, ch = _max_speeds(u, n)
        dt = min(COURANT / n[0] / ctot, due - t)
        u = step(u, i, dt, ch, _fac(ch, dt), modes, min(t / TURB_T, 1.0))
        t += dt
    return u, t


def _loop_exact(u, n, seed, amp, steps):
    def step(u, i, dt, ch, fac, modes, ramp):
        return _sweep(u, n, 2, lambda s, a: _unsplit(s, 1.0 / n[0], dt, ch, fac, "mc", "hlld", a), modes, ramp)

    return _clock(u.double(), n, seed, amp, steps, step)


def _vjp(u, ubar, n, dt, ch, fac, recon, riemann, modes, ramp):
    """(ubar pulled back through one step, dL/d log(amplitude))."""
    out = torch.zeros(u.shape, dtype=torch.float64, device="cuda")
    damp = 0.0
    for ext, own in _slabs(n, 2, max(1, min(n[2], (1 << 19) // (n[0] * n[1])))):
        x = u[:, ext].double().requires_grad_(True)
        scale = torch.ones((), dtype=torch.float64, device="cuda", requires_grad=True)
        y = _unsplit(x, 1.0 / n[0], dt, ch, fac, recon, riemann, _accel(modes, n, ext, ramp) * scale)
        gx, ga = torch.autograd.grad(y[:, 2:2 + len(own)], (x, scale), ubar[:, own].double())
        out.index_add_(1, ext, gx)
        damp += float(ga)
        del x, y, gx
    return out, damp


def _spectrum_density(u, n):
    w = u[1:4].double() / torch.sqrt(u[0].double())
    f = torch.fft.fftn(w, dim=(1, 2, 3)) / (n[0] * n[1] * n[2])
    k = [torch.fft.fftfreq(m, device="cuda", dtype=torch.float64) * m for m in (n[2], n[1], n[0])]
    kk = torch.sqrt(k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2)
    return 0.5 * (f.real ** 2 + f.imag ** 2).sum(0), torch.floor(kk + 0.5).long()


def exact(case, seed):
    return _f64(_exact(case, seed))


def _exact(case, seed):
    st = prepare(case, seed)
    kind = case["kind"]
    if kind == "ensemble":
        sizes, mach, _ = _sizes(case)
        got, times, at = [], [], 0
        for b, m in enumerate(sizes):
            u0 = st["u0"][at:at + 9 * m ** 3].view(9, m, m, m)
            u, t = _loop_exact(u0, (m, m, m), int(seed) % 1000003 + b, 2.0 * float(mach[b]), case["steps"])
            got.append(u.reshape(-1))
            times.append(t)
            at += 9 * m ** 3
        return {"u": torch.cat(got), "t": np.array(times)}
    n, dt, sd = (case["nx"], case["ny"], case["nz"]), COURANT / case["nx"] / SIGNAL, 1 + int(seed) % 1000003
    dx, modes, ramp, fac = 1.0 / case["nx"], 2.0 * _modes(seed), TIME / TURB_T, _fac(CH, dt)
    if kind == "glm":
        u = _sweep(st["u"], n, 2, lambda s, a: _unsplit(s, dx, dt, CH, fac, case["recon"], case["riemann"], a), modes, ramp)
        return {"u": u, "cfl": np.array(_max_speeds(u, n))}
    if kind == "ct":
        u = _sweep(st["u"], n, 4, lambda s, a: _ct_step(s, dx, dt, case["recon"], case["riemann"], case["emf"], a), modes, ramp)
        return {"u": u, "cfl": np.array(_max_speeds(u, n, _ct_cells))}
    if kind == "march":
        return {"u": _sweep(st["u"], n, 2, lambda s, a: _march_step(s, dx, dt, CH, fac, case["recon"], case["nsp"]))}
    if kind == "adjoint":
        g, damp = _vjp(st["u"], st["g"], n, dt, CH, fac, case["recon"], case["riemann"], modes, ramp)
        return {"ubar": g, "amp": damp / 2.0}
    if kind == "gradient":
        tape = []

        def step(u, i, dt, ch, fac, modes, ramp):
            tape.append((u, dt, ch, fac, modes, ramp))
            return _sweep(u, n, 2, lambda s, a: _unsplit(s, dx, dt, ch, fac, "mc", "hlld", a), modes, ramp)

        u, _ = _clock(st["u"].double(), n, sd, 2.0, case["steps"], step)
        x = u.clone().requires_grad_(True)
        p, shell = _spectrum_density(x, n)
        loss = p[(shell >= 4) & (shell <= 8)].sum()
        g = torch.autograd.grad(loss, x)[0]
        amp = 0.0
        for v, dt, ch, fac, modes, ramp in reversed(tape):
            g, a = _vjp(v, g, n, dt, ch, fac, "mc", "hlld", modes, ramp)
            amp += a / 2.0
        return {"loss": float(loss.detach()), "grad": g, "amp": amp, "u": u}
    if kind == "loop":
        u, t = _loop_exact(st["u0"], n, sd, 2.0, case["steps"])
        return {"t": t, "u": u}
    u = st["u"]
    p, shell = _spectrum_density(u, n)
    spectrum = torch.stack([p[shell == k].sum() for k in range(case["kmax"] + 1)]).cpu().numpy()
    x = u.double()
    rho = x[0]
    ke2 = ((x[1:4] ** 2).sum(0) / rho.clamp(min=SMALLR)).sum()
    div = sum(_ahead(x[5 + d:6 + d], d) - _back(x[5 + d:6 + d], d) for d in range(3))[0].abs() / (2 * dx)
    s = torch.log(rho / rho.mean())
    inside = (s >= -2.0) & (s < 2.0)
    hist = torch.bincount(((s[inside] + 2.0) * (case["nbins"] / 4.0)).long(), minlength=case["nbins"])
    return {"diag": {"mass": float(rho.sum()), "ke2": float(ke2), "vrms": math.sqrt(float(ke2) / float(rho.sum())),
                     "divbmax": float(div.max()), "rhomin": float(rho.min()), "etot": float(x[4].sum()),
                     "divb_l2": math.sqrt(float((div ** 2).mean())), "psi_l2": math.sqrt(float((x[8] ** 2).mean())),
                     "finite": 1, "nonfinite_cells": 0},
            "spectrum": spectrum, "pdf": hist.cpu().numpy() / (rho.numel() * 4.0 / case["nbins"]),
            "moments": {"rho_mean": float(rho.mean()), "s_mean": float(s.mean()), "sigma_s": float(s.std(unbiased=False))}}
