"""The single stage calls (eif_exchange_momentum, eif_compute_inertia, a recorded adjoint step)
after whole steps, which run as captured graphs: they see the particles where the steps left
them. Two steps first, so that the graphs of both buffer parities exist, then a stage call,
which leaves boxes, weights and band lists that the next step makes out of date."""
import numpy as np
import pytest

from ellipsesinflows_gb300 import PREC_FP64, PREC_MIXED, Batch, F, Simulation, cases

pytestmark = pytest.mark.gpu

DT = 2.0e-3


def moving():
    """ellipses that cross a good part of a cell in a step"""
    case = cases.poiseuille(itot=96, jtot=192, n=6, a=0.06, b=0.035, seed=4)
    case.particles[:, F["uy"]] += 2.0
    return case


def fields(s):
    """the field response, the records and the velocities after an exchange at the present state"""
    s.exchange_momentum()
    return [np.array(a) for a in s.pull_ibm_fields()] + [np.array(s.pull_particles())]


def inertia(s):
    s.reset_particle_increments()
    s.compute_inertia(0)
    return [np.array(s.pull_particles())]


def fresh(s, case, prec):
    """a new context at the state of s"""
    f = Simulation(case.config(precision=prec))
    f.push_fluid(*[np.array(a) for a in s.pull_fluid()[:3]])
    f.push_particles(np.array(s.pull_particles()))
    f.dt = s.dt
    return f


@pytest.mark.parametrize("what", [fields, inertia], ids=["exchange", "inertia"])
@pytest.mark.parametrize("how", ["integrate", "advance", "batch"])
@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_stage_call_after_a_captured_step(prec, how, what, gpu_lib):
    case = moving()
    s = Simulation.from_case(case, precision=prec)
    s.dt = DT
    batch = Batch([s]) if how == "batch" else None

    def step():
        if how == "integrate":
            s.integrate()
        elif how == "advance":
            s.advance(1)
        else:
            batch.advance(1)

    step()
    step()
    before = what(s)
    step()
    f = fresh(s, case, prec)
    got, want = what(s), what(f)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    assert not np.array_equal(got[0], before[0])
    if batch:
        batch.close()


def test_recorded_step_after_an_unrecorded_one(gpu_lib):
    case = cases.adjoint_couette(itot=64, jtot=128, n=3)
    s = Simulation(case.config())
    s.push_fluid(*case.fluid())
    s.push_particles(case.particles)
    s.dt = DT
    s.adjoint_begin(1)
    s.adjoint_forward(record=False)
    s.adjoint_forward(record=False)
    s.exchange_momentum()
    s.adjoint_forward(record=False)
    f = fresh(s, case, PREC_FP64)
    f.adjoint_begin(1)
    out = []
    for q in (s, f):
        q.adjoint_forward(record=True)
        out.append([np.array(a) for a in q.pull_fluid()[:3]] + [np.array(q.pull_particles())])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
