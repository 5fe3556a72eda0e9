"""The Poisson solve over column lengths: blocks that end in a shorter one, groups of
interface values that end in a shorter one, and the sweeps of short and very long columns,
against a dense cosine / Fourier solve in numpy (the operator of compute_potential.c:48-138).

Tolerance: that of the solve at block multiples (1e-11 in the FP64 form, 1e-10 in the mixed
one), or the rounding of an elimination over a matrix of condition number (n / pi)^2, that is
eps n^2 to be safe, where that is more (n > 300)."""
import math

import numpy as np
import pytest

from ellipsesinflows_gb300 import PREC_FP64, PREC_MIXED, Simulation, make_config

pytestmark = pytest.mark.gpu

GAMMA = (45.0 - 25.0) / 60.0   # RK stage 2 (src/param/init.c:177-189)
LY = 2.0


def dense_solve(q, dx, dy):
    jt, it = q.shape
    k = np.arange(it)
    C = np.cos(math.pi * ((k[:, None] * (2 * k[None, :] + 1)) % (4 * it)) / (2 * it))
    lam = (-4.0 / dx**2 * np.sin(math.pi * k / (2 * it)) ** 2)[None, :] \
        - (4.0 / dy**2 * np.sin(math.pi * np.arange(jt // 2 + 1) / jt) ** 2)[:, None]
    lam[0, 0] = 1.0
    c = np.fft.rfft(q @ C.T, axis=0) / lam
    c[0, 0] = 0.0
    c = np.fft.irfft(c, n=jt, axis=0)
    c[:, 0] *= 0.5
    return (2.0 / it) * (c @ C)


@pytest.mark.parametrize("prec,tol", [(PREC_FP64, 1e-11), (PREC_MIXED, 1e-10)], ids=["fp64", "mixed"])
@pytest.mark.parametrize("itot", [16, 36])
# shorter last blocks of 1, 2, M - 1 rows for the three block sizes; last groups of 1, 2 and
# full size; equal blocks whose number no group size divides (432, 528, 1000, 1028, 2052);
# sweeps over few (9, 48) and groups of 32 (8209) interface values; the sequential solve (7)
@pytest.mark.parametrize("jtot", [7, 9, 10, 11, 17, 23, 33, 47, 48, 129, 145, 161, 430, 432, 528, 529, 1000, 1028, 2052, 8209])
def test_column_lengths(prec, tol, itot, jtot, gpu_lib):
    s = Simulation(make_config(itot, jtot, ly=LY, Re=100.0, precision=prec))
    rng = np.random.default_rng(jtot)
    ux, uy, p = np.zeros((jtot + 2, itot + 1)), np.zeros((jtot + 2, itot + 2)), np.zeros((jtot + 2, itot + 2))
    ux[1:-1, 1:-1] = rng.standard_normal((jtot, itot - 1))
    uy[1:-1, 1:-1] = rng.standard_normal((jtot, itot))
    for a in (ux, uy):
        a[0], a[-1] = a[-2], a[1]
    s.push_fluid(ux, uy, p)
    s.dt = 1.0e-3
    s.compute_potential(2)
    psi = s.pull_fluid()[3][1:-1, 1:-1]
    dx, dy = 1.0 / itot, LY / jtot
    div = (ux[1:-1, 1:] - ux[1:-1, :-1]) / dx + (uy[2:, 1:-1] - uy[1:-1, 1:-1]) / dy
    want = dense_solve(div / (GAMMA * 1.0e-3), dx, dy)
    a, b = psi - psi.mean(), want - want.mean()
    assert np.abs(a - b).max() / np.abs(b).max() < max(tol, 2.2e-16 * jtot**2)
