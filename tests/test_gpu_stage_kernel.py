"""The persistent sub-iteration kernel of a suspension advanced alone (subiter.cu) against the
host-driven loop of single kernels: bitwise the same state and the same sub-iteration counts.

Particle counts: none, one whose tasks are cut into slices, a few, contacts (units of unequal
length), the largest count that runs the stage kernel on 152 SMs and the next one (a loop of
kernels), in both forms; by eif_integrate, by eif_advance, and for the adjoint's recording."""
import numpy as np
import pytest

from ellipsesinflows_gb300 import PREC_FP64, PREC_MIXED, Simulation, cases

pytestmark = pytest.mark.gpu

MOST = 270   # particles whose units (one each and one per eight) are at most 2 x 152


def build(name):
    if name == "contacts":
        return cases.contact_cluster()
    n = {"none": 0, "one": 1, "few": 6, "most": MOST, "more": MOST + 1}[name]
    if n > 6:
        return cases.poiseuille(itot=128, jtot=256, n=n, a=0.02, b=0.014, seed=3)
    if n == 0:
        case = cases.poiseuille(itot=64, jtot=128, n=1, a=0.05, b=0.03, seed=3)
        case.particles = case.particles[:0]
        return case
    if n == 1:
        return cases.couette_circle(itot=128, jtot=256)
    return cases.poiseuille(itot=64, jtot=128, n=n, a=0.08, b=0.05, seed=5)


def run(case, prec, how):
    s = Simulation(case.config(precision=prec))
    s.push_fluid(*case.fluid())
    s.push_particles(case.particles)
    subs = None
    if how == "integrate":
        subs = [list(s.step()) for _ in range(3)]
    else:
        s.advance(3)
    return [np.array(f) for f in s.pull_fluid()[:3]] + [np.array(s.pull_particles())], subs


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("name", ["none", "one", "few", "contacts", "most", "more"])
def test_stage_kernel_equals_host_driven_loop(name, prec, gpu_lib, monkeypatch):
    case = build(name)
    got, subs = run(case, prec, "integrate")
    adv, _ = run(case, prec, "advance")
    monkeypatch.setenv("EIF_NO_GRAPHS", "1")
    want, wsubs = run(case, prec, "integrate")
    assert subs == wsubs
    for a, b, c in zip(got, want, adv):
        assert np.array_equal(a, b) and np.array_equal(c, b)


def gradient(s, case, steps):
    rng = np.random.default_rng(8)
    s.push_fluid(*case.fluid())
    s.push_particles(case.particles)
    s.dt = 1.0e-3
    s.adjoint_begin(steps)
    for _ in range(steps):
        s.adjoint_forward(record=True)
    sx, sy = s.shapes()
    s.adjoint_seed(rng.standard_normal(sx), rng.standard_normal(sy))
    for _ in range(steps):
        s.adjoint_backward()
    return [np.array(a) for a in s.adjoint_pull()] + [np.array(s.adjoint_pull_particles()), np.array(s.adjoint_wall_gradient())]


def test_gradient_again_in_kept_buffers(gpu_lib, monkeypatch):
    """a second recording of the same shape, one after another shape, and one after a larger
    particle set was pushed in between give the first one's bits; so does the host-driven loop"""
    case, big = cases.adjoint_couette(itot=64, jtot=128, n=3), cases.adjoint_couette(itot=64, jtot=128, n=6)
    s = Simulation(case.config())
    first = gradient(s, case, 2)
    for other, steps in ((case, 2), (case, 3), (big, 2)):
        gradient(s, other, steps)
        again = gradient(s, case, 2)
        assert all(np.array_equal(a, b) for a, b in zip(first, again))
    monkeypatch.setenv("EIF_NO_GRAPHS", "1")
    host = gradient(Simulation(case.config()), case, 2)
    assert all(np.array_equal(a, b) for a, b in zip(first, host))
