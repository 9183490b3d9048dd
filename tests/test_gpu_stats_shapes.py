"""The spectrum, band loss and PDF kernels at the edges of their tiles: grids that are no multiple of the
32 rows or columns of a staged chunk, from one to several groups of wavenumbers per block and per grid,
and planes that allow no 16-byte loads."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def _state(n, dtype, seed=0, shift=0):
    """A positive-density GLM state; shift > 0: the planes start `shift` elements off a 16-byte boundary."""
    nx, ny, nz = n
    g = torch.Generator().manual_seed(seed)
    u = torch.randn((9, nz, ny, nx), generator=g, dtype=torch.float64)
    u[0] = torch.exp(0.5 * u[0])
    buf = torch.empty(u.numel() + 8, dtype=dtype, device="cuda")
    v = buf[shift:shift + u.numel()].view(9, nz, ny, nx)
    v.copy_(u.to("cuda"))
    return v


def _density(u):
    """|w^|^2 / 2 per mode and its shell, by FFT in FP64."""
    w = u[1:4].double() / torch.sqrt(u[0].double())
    nz, ny, nx = w.shape[1:]
    f = torch.fft.fftn(w, dim=(1, 2, 3)) / (nx * ny * nz)
    k = [torch.fft.fftfreq(m, device="cuda", dtype=torch.float64) * m for m in (nz, ny, nx)]
    kk = torch.sqrt(k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2)
    return 0.5 * (f.real ** 2 + f.imag ** 2).sum(0), torch.floor(kk + 0.5).long()


def test_spectrum_forms_w_to_two_roundings():
    """w = m rsqrt(rho) is no worse than m / sqrt(rho) by a root and a division of half an ulp each.  One cell of a
    4^3 box carries momentum, so every sum of the transform is exact and E(0) = (w / 64)^2 / 2: the bound is twice
    w's 2 u and the square's u, u = 2^-53 (measured 3.92 u; by root and division 3.91 u)."""
    from fractions import Fraction
    from glmmhdturb_b200 import Solver
    s = Solver(4, dtype="f64", gamma=5 / 3)
    u = torch.zeros((9, 4, 4, 4), dtype=torch.float64, device="cuda")
    u[0] = 1.0
    rng = np.random.default_rng(3)
    worst = 0.0
    for rho, m in zip(np.exp(rng.uniform(-2, 2, 1500)), rng.uniform(0.5, 4.0, 1500)):
        u[0, 0, 0, 0], u[1, 0, 0, 0] = float(rho), float(m)
        ref = Fraction(float(m)) ** 2 / Fraction(float(rho)) / (2 * 64 ** 2)
        worst = max(worst, abs(float(Fraction(float(s.ke_spectrum(u, kmax=1)[0])) / ref - 1)))
    assert worst <= 5.0 * 2.0 ** -53


# wavenumbers per axis: one group of the x stage, several warps of groups, more than one block of them
@pytest.mark.parametrize("n,kmax", [((3, 3, 3), 1), ((33, 31, 32), 4), ((32, 65, 12), 5), ((70, 45, 47), 19),
                                    ((61, 66, 64), 24)])
@pytest.mark.parametrize("dtype", ["f32", "f64"])
def test_spectrum_matches_fft(n, kmax, dtype):
    from glmmhdturb_b200 import Solver
    u = _state(n, torch.float64 if dtype == "f64" else torch.float32, seed=kmax)
    s = Solver(n, dtype=dtype, gamma=5 / 3)
    got = s.ke_spectrum(u, kmax=kmax)
    p, shell = _density(u)
    ref = torch.stack([p[shell == k].sum() for k in range(kmax + 1)]).cpu().numpy()
    # a mode is a sum of N^3 terms of size w/N^3 along three axes: its rounding is below
    # (nx + ny + nz) eps times the rms field, and a shell adds up squares of such modes
    tol = 4.0 * sum(n) * EPS * max(1.0, float(p.sum()))
    assert np.abs(got - ref).max() <= tol, (got, ref)


@pytest.mark.parametrize("n,kmin,kmax", [((33, 31, 34), 1, 4), ((40, 44, 39), 4, 19)])
def test_band_loss_matches_autograd(n, kmin, kmax):
    from glmmhdturb_b200 import Solver
    u = _state(n, torch.float64, seed=7)
    s = Solver(n, dtype="f64", gamma=5 / 3)
    loss, g = s.ke_band_loss(u, kmin, kmax)
    x = u.clone().requires_grad_(True)
    p, shell = _density(x)
    ref = p[(shell >= kmin) & (shell <= kmax)].sum()
    gref = torch.autograd.grad(ref, x)[0]
    tol = 4.0 * sum(n) * EPS
    assert abs(loss - float(ref.detach())) <= tol * max(1.0, float(p.detach().sum()))
    assert float((g - gref).norm() / gref.norm()) <= 16 * tol   # a band is a part of the whole field


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", [(1, 1, 1), (5, 3, 7), (64, 48, 33), (130, 65, 31)])
def test_density_pdf_counts(n, shift):
    from glmmhdturb_b200 import Solver
    u = _state(n, torch.float32, seed=3, shift=shift)
    s = Solver(n, dtype="f32", gamma=5 / 3)
    pdf, st = s.density_pdf(u, nbins=50, smin=-1.0, smax=1.0)
    rho = u[0].double()
    ln = torch.log(rho / rho.mean())
    cells = rho.numel()
    inside = ln[(ln >= -1.0) & (ln < 1.0)]
    ref = torch.bincount(((inside + 1.0) * 25.0).long(), minlength=50).cpu().numpy() / (cells * 0.04)
    # a cell within rounding of a bin edge may count on either side of it
    assert np.abs(pdf - ref).sum() * cells * 0.04 <= 2
    assert abs(st["rho_mean"] - float(rho.mean())) <= cells * EPS
    assert abs(st["s_mean"] - float(ln.mean())) <= cells * EPS
    assert abs(st["sigma_s"] - float(ln.std(unbiased=False))) <= max(1e-12, np.sqrt(cells * EPS))
