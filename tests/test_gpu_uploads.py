"""What the host uploads is on the device before the kernels that read it, which run on streams
that do not wait for the null stream."""
import numpy as np
import pytest

from ellipsesinflows_gb300 import Simulation, cases

pytestmark = pytest.mark.gpu


def test_descriptors_of_new_stage_kernels(gpu_lib, monkeypatch):
    """Recorded adjoint steps right after pushes that change the particle count: every push
    makes a new plan of the stage kernel, which is launched as soon as its descriptors are
    uploaded. The state is that of the host-driven loop, every time."""
    some = [cases.adjoint_couette(itot=64, jtot=128, n=n) for n in (3, 6)]

    def step(s, case):
        s.push_fluid(*case.fluid())
        s.push_particles(case.particles)
        s.dt = 1.0e-3
        s.adjoint_begin(1)
        s.adjoint_forward(record=True)
        return [np.array(a) for a in s.pull_fluid()[:3]] + [np.array(s.pull_particles())]

    monkeypatch.setenv("EIF_NO_GRAPHS", "1")
    want = [step(Simulation(c.config()), c) for c in some]
    monkeypatch.delenv("EIF_NO_GRAPHS")
    s = Simulation(some[0].config())
    for k in range(16):
        for a, b in zip(step(s, some[k % 2]), want[k % 2]):
            assert np.array_equal(a, b)
