"""Contact forces of one ellipse with many partners at once (collision.c:75-367).

A warp fits up to sixteen pairs at a time, two lanes each, with the walls after the last
pair: partner counts around that number, with and without a wall, against the C
restatement. The tolerance is the one of the stage tests (sums over contacts, 1e-10 of the
largest force); the fits stop on the same rule, so both sides run the same iterations.
"""
import math

import numpy as np
import pytest

from ellipsesinflows_gb300 import Simulation, cases
from ellipsesinflows_gb300.capi import F
from ellipsesinflows_gb300.cases import particle_records
from oracle import port

FIELDS = ["cfx0", "cfy0", "ctz0"]


def ring(n, wall, seed=3):
    """a large tilted ellipse with n small ones, each turned away from the normal, 3e-4 into its
    rim at irregular places, the listed order mixed; wall: the large one 1e-3 into the wall
    x = 0, the small ones off that side"""
    rng = np.random.default_rng(seed)
    a, b, r, q, tilt = 0.11, 0.09, 0.006, 0.8, 0.3
    cx = math.hypot(a * math.cos(tilt), b * math.sin(tilt)) - 1e-3 if wall else 0.5
    lo, hi = (-0.6 * math.pi, 0.5 * math.pi) if wall else (0.0, 2.0 * math.pi)
    t = lo + (np.arange(n) + rng.uniform(0.4, 0.6, n)) / max(n, 1) * (hi - lo)
    nx, ny = b * np.cos(t), a * np.sin(t)
    nn = np.hypot(nx, ny)
    nx, ny = nx / nn, ny / nn
    turn = rng.uniform(0.3, 1.2, n)
    reach = np.hypot(r * np.cos(turn), q * r * np.sin(turn)) - 3e-4
    # contact points at the small ellipses' support points, not on the line through their centres
    along = (r * r - (q * r) ** 2) * np.sin(turn) * np.cos(turn) / (reach + 3e-4)
    X = a * np.cos(t) + reach * nx + along * ny
    Y = b * np.sin(t) + reach * ny - along * nx
    c, s = math.cos(tilt), math.sin(tilt)
    x, y = np.append(cx + c * X - s * Y, cx), np.append(1.0 + s * X + c * Y, 1.0)
    aa, bb = np.append(np.full(n, r), a), np.append(np.full(n, q * r), b)
    az = np.append((np.arctan2(ny, nx) + tilt + turn) % (2 * math.pi), tilt)
    order = rng.permutation(n + 1)
    return particle_records(*(v[order] for v in (np.append(np.full(n, 1.1), 1.0), aa, bb, x, y, az)))


def forces(sim, case, rec):
    sim.push_fluid(*case.fluid())
    sim.push_particles(rec)
    sim.compute_collision_force(0)
    return sim.pull_particles()[:, [F[f] for f in FIELDS]]


@pytest.mark.parametrize("wall", [False, True], ids=["free", "wall"])
@pytest.mark.parametrize("n", [0, 1, 15, 16, 17, 40])
def test_ring_has_contacts(n, wall):
    """every ellipse is in contact, with a torque that is not rounding"""
    case = cases.contact_cluster()
    rec = ring(n, wall)
    got = np.abs(forces(port.PortSolver(case.config()), case, rec))
    force = np.max(got[:, :2], axis=1)
    assert np.count_nonzero(force) == (n + 1 if n or wall else 0)
    if n or wall:
        assert np.max(got[:, 2] * rec[:, F["a"]]) > 0.01 * np.max(force)


@pytest.mark.gpu
@pytest.mark.parametrize("wall", [False, True], ids=["free", "wall"])
@pytest.mark.parametrize("n", [0, 1, 15, 16, 17, 40])
def test_many_contacts_match_oracle(n, wall, gpu_lib):
    case = cases.contact_cluster()
    rec = ring(n, wall)
    want = forces(port.PortSolver(case.config()), case, rec)
    got = forces(Simulation(case.config()), case, rec)
    for k in range(3):
        assert np.max(np.abs(got[:, k] - want[:, k])) <= 1e-10 * np.max(np.abs(want[:, k:k + 1] if k == 2 else want[:, :2]))
