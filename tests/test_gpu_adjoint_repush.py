"""A recording whose particles were replaced by a larger set and put back between
eif_adjoint_begin and the steps (the records' buffer stays larger) gives the gradient of one
without that, and leaves the records as they were."""
import numpy as np
import pytest

from ellipsesinflows_gb300 import Simulation, cases

pytestmark = pytest.mark.gpu


def gradient(case, other):
    rng = np.random.default_rng(8)
    s = Simulation(case.config())
    s.push_fluid(*case.fluid())
    s.push_particles(case.particles)
    s.dt = 1.0e-3
    s.adjoint_begin(2)
    if other is not None:
        s.push_particles(other.particles)
        s.push_particles(case.particles)
    for _ in range(2):
        s.adjoint_forward(record=True)
    records = np.array(s.pull_particles())
    sx, sy = s.shapes()
    s.adjoint_seed(rng.standard_normal(sx), rng.standard_normal(sy))
    for _ in range(2):
        s.adjoint_backward()
    assert np.array_equal(records, s.pull_particles())
    return [np.array(a) for a in s.adjoint_pull()] + [np.array(s.adjoint_pull_particles()), np.array(s.adjoint_wall_gradient())]


def test_gradient_after_a_larger_set_was_pushed(gpu_lib):
    case, big = cases.adjoint_couette(itot=64, jtot=128, n=3), cases.adjoint_couette(itot=64, jtot=128, n=6)
    for a, b in zip(gradient(case, None), gradient(case, big)):
        assert np.array_equal(a, b)
