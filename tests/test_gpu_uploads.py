"""What the host uploads is on the device before the kernels that read it, which run on streams
that do not wait for the null stream."""
import numpy as np
import pytest

from ellipsesinflows_gb300 import PREC_FP64, PREC_MIXED, F, Simulation, cases

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


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_radii_of_pageable_records(prec, gpu_lib):
    """The radii pushed from pageable memory decide where a particle's sums are kept in the
    stage kernel. The same particles in two orders have the same total, so the buffers and
    graphs are kept between these pushes; every step is that of a fresh context."""
    case = cases.poiseuille(itot=96, jtot=192, n=8, a=0.05, b=0.03, seed=6)
    rec = case.particles
    size = np.linspace(0.5, 1.0, len(rec))
    orders = []
    for scale in (size, size[::-1]):
        r = rec.copy()
        r[:, F["a"]] *= scale
        r[:, F["b"]] *= scale
        orders.append(r)

    def step(s, r):
        s.push_fluid(*case.fluid())
        s.push_particles(r)
        s.advance(1)
        return [np.array(a) for a in s.pull_fluid()[:3]] + [np.array(s.pull_particles())]

    want = [step(Simulation(case.config(precision=prec)), r) for r in orders]
    s = Simulation(case.config(precision=prec))
    for k in range(16):
        for a, b in zip(step(s, orders[k % 2]), want[k % 2]):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
def test_tables_of_new_buffers(prec, gpu_lib):
    """A new context, and a push of another particle count, upload tables that the first stage
    call reads at once: always the same field response."""
    case = cases.poiseuille(itot=96, jtot=192, n=8, a=0.05, b=0.03, seed=6)
    case.particles[:, F["vz"]] = 1.0
    first = None
    for _ in range(8):
        with Simulation(case.config(precision=prec)) as s:
            for n in (8, 3, 8):
                s.push_fluid(*case.fluid())
                s.push_particles(case.particles[:n])
                s.dt = 1.0e-3
                s.exchange_momentum()
            got = [np.array(a) for a in s.pull_ibm_fields()]
        first = first or got
        for a, b in zip(got, first):
            assert np.array_equal(a, b) and np.abs(a).max() > 0.0
