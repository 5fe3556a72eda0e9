"""Weights of the double-precision indicator against extended precision.

With the fluid at rest and a particle of unit x-velocity the field response of the momentum
exchange is the weight w = 1 - tanh(2 d / h)^2 of every cell of the particle's box
(src/suspensions/auxiliary.c:19-59, exchange.c:61-72), d the distance to the ellipse. Shapes: a
circle, aspect ratios to 20 (cells next to the evolute, where the general iteration runs), an
ellipse small enough that all its cells are near, one with a major axis of 400 cells; the boxes
reach from d = 0 to where tanh is 1, over both ends of the tables and the change to float pairs.

Bound of an error, in units of u = 2^-53: tanh is rounded once, half the spacing u of the
doubles below 1, and a tenth of it for what the float pairs and the table leave: 0.6 u, which is
1.2 u in w = 1 - tanh^2; w's own rounding, w u; and the distance's: the offset, its rotation
and scaling and the foot are about ten roundings of quantities no larger than A + 30 (A the
major semi-axis, in units of h / 2), so 10 u (A + 30) in z = 2 d / h, times |dw/dz| = 2 w tanh."""
import numpy as np
import pytest

from ellipsesinflows_gb300 import NFIELDS, PREC_FP64, F, Simulation, make_config

pytestmark = pytest.mark.gpu

L = np.longdouble
U = 2.0 ** -53
LY = 2.0
# cells across, semi-axes in cells, angles
SHAPES = {
    "circle": (96, 10.0, 10.0, (0.0, 0.7)),
    "ratio_2": (96, 12.0, 6.0, (0.0, 0.4, 2.2)),
    "ratio_3_small": (96, 3.0, 2.0, (0.3, 1.1, 2.9)),
    "ratio_6": (256, 24.0, 4.0, (0.0, 0.8, 1.9)),
    "ratio_20": (512, 40.0, 2.0, (0.2, 1.3)),
    "large": (512, 200.0, 60.0, (0.5,)),
}


def exact(it, jt, rec, i, j):
    """w, z and tanh of the cells (i, j), 1-based"""
    dx, dy = 1.0 / it, LY / jt
    h = L(min(dx, dy))
    xf = np.arange(it + 1) * dx
    xf[it] = 1.0
    xc, yc = 0.5 * (xf[:-1] + xf[1:]), 0.5 * (2 * np.arange(1, jt + 1) - 1) * dy
    X, Y = (xc[i - 1].astype(L) - L(rec[F["x"]])) / h, (yc[j - 1].astype(L) - L(rec[F["y"]])) / h
    a, b, az = L(rec[F["a"]]) / h, L(rec[F["b"]]) / h, L(rec[F["az"]])
    c, s = np.cos(az), np.sin(az)
    px, py = np.abs(c * X + s * Y), np.abs(c * Y - s * X)
    # the foot's parameter: bisection in double, Newton steps in extended precision (the distance
    # is stationary in it)
    x, y, A, B = (np.asarray(v, dtype=np.float64) for v in (px, py, a, b))
    lo, hi = np.zeros_like(x), np.full_like(x, np.pi / 2)
    for _ in range(52):
        t = 0.5 * (lo + hi)
        ct, st = np.cos(t), np.sin(t)
        up = (y - B * st) * B * ct - (x - A * ct) * A * st > 0
        lo, hi = np.where(up, t, lo), np.where(up, hi, t)
    t = (0.5 * (lo + hi)).astype(L)
    for _ in range(3):
        ct, st = np.cos(t), np.sin(t)
        vx, vy = px - a * ct, py - b * st
        g = vy * b * ct - vx * a * st
        K = (a * st) ** 2 + (b * ct) ** 2 + vx * a * ct + vy * b * st
        step = np.where(np.abs(g) < 1e-3 * np.abs(K), g / np.where(K == 0, L(1), K), L(0))
        t = np.clip(t + step, L(0), L(np.pi) / 2)
    z = 2 * np.hypot(px - a * np.cos(t), py - b * np.sin(t))
    e = np.exp(-2 * z)
    return 4 * e / (1 + e) ** 2, z, (1 - e) / (1 + e)


@pytest.mark.parametrize("shape", list(SHAPES))
def test_weights_against_extended_precision(shape, gpu_lib):
    it, a, b, angles = SHAPES[shape]
    jt = 2 * it
    sim = Simulation(make_config(it, jt, ly=LY, Re=100.0, precision=PREC_FP64))
    sim.push_fluid(np.zeros((jt + 2, it + 1)), np.zeros((jt + 2, it + 2)), np.zeros((jt + 2, it + 2)))
    for k, az in enumerate(angles):
        rec = np.zeros((1, NFIELDS))
        for name, v in (("den", 1.0), ("a", a / it), ("b", b / it), ("az", az), ("ux", 1.0),
                        ("x", 0.5 + (0.31 - 0.17 * k) / it), ("y", 1.0 + (0.11 + 0.23 * k) / it)):
            rec[0, F[name]] = v
        sim.push_particles(rec)
        sim.dt = 1.0e-3
        sim.exchange_momentum()
        w = np.array(sim.pull_ibm_fields()[0])
        r = rec[0]
        R = (a + 3.0) / it
        i = np.arange(max(1, int((r[F["x"]] - R) * it) + 2), min(it, int((r[F["x"]] + R) * it)) + 1)
        j = np.arange(max(1, int((r[F["y"]] - R) * it) + 2), min(jt, int((r[F["y"]] + R) * it)) + 1)
        jj, ii = [v.ravel() for v in np.meshgrid(j, i, indexing="ij")]
        # cells at most 14 from the ellipse by its gauge; inside and outside of those w is zero
        c, s = np.cos(az), np.sin(az)
        X, Y = (ii - 0.5) - r[F["x"]] * it, (jj - 0.5) - r[F["y"]] * it
        rho = np.hypot((c * X + s * Y) / a, (c * Y - s * X) / b)
        near = b * np.abs(rho - 1.0) < 14.0
        assert np.all(w[jj[~near], ii[~near]] == 0.0)
        jj, ii = jj[near], ii[near]
        want, z, th = exact(it, jt, r, ii, jj)
        err = np.abs(w[jj, ii].astype(L) - want)
        tol = U * (1.2 + want + 10.0 * (2.0 * a + 30.0) * 2.0 * want * th)
        worst = np.argmax(err / tol)
        print("%s az %.1f: %d cells, worst %.2f of its bound (z %.2f, error %.2e)"
              % (shape, az, len(z), float(err[worst] / tol[worst]), float(z[worst]), float(err[worst])))
        assert np.all(err <= tol)
