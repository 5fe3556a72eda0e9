"""A suspension advanced alone where its stage kernel cannot be had, or beside others.

EIF_TEST_NO_STAGE_KERNEL=1 makes the set-up of the stage kernel fail as it does without
cooperative launches or without room for its grid: the steps and the adjoint's recording run
the loops of kernels then, with the same bits. And contexts that step at the same time, each
from a thread of its own, every one with a stage kernel that fills the GPU, get the bits of
separate runs."""
import threading

import numpy as np
import pytest

from ellipsesinflows_gb300 import PREC_FP64, PREC_MIXED, Simulation, cases
from test_gpu_stage_kernel import build, gradient, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("name", ["one", "few", "contacts"])
def test_loops_of_kernels_instead(name, prec, gpu_lib, monkeypatch):
    case = build(name)
    want, wsubs = run(case, prec, "integrate")
    monkeypatch.setenv("EIF_TEST_NO_STAGE_KERNEL", "1")
    got, subs = run(case, prec, "integrate")
    adv, _ = run(case, prec, "advance")
    assert subs == wsubs
    for a, b, c in zip(got, want, adv):
        assert np.array_equal(a, b) and np.array_equal(c, b)


def test_recording_without_the_stage_kernel(gpu_lib, monkeypatch):
    case = cases.adjoint_couette(itot=64, jtot=128, n=3)
    want = gradient(Simulation(case.config()), case, 2)
    monkeypatch.setenv("EIF_TEST_NO_STAGE_KERNEL", "1")
    got = gradient(Simulation(case.config()), case, 2)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_contexts_stepping_in_threads(gpu_lib):
    specs = [(cases.couette_circle(itot=128, jtot=256), PREC_FP64),
             (cases.poiseuille(itot=128, jtot=256, n=120, a=0.025, b=0.015, seed=3), PREC_MIXED),
             (cases.poiseuille(itot=96, jtot=192, n=24, a=0.05, b=0.03, seed=5), PREC_FP64),
             (cases.contact_cluster(), PREC_MIXED)]
    rounds, steps = 6, 5

    def work(s, out, k):
        try:
            for _ in range(rounds):
                s.advance(steps)
                s.step()
            out[k] = [np.array(f) for f in s.pull_fluid()[:3]] + [np.array(s.pull_particles())]
        except Exception as e:  # reported by the test's own thread
            out[k] = e

    want, got = [None] * len(specs), [None] * len(specs)
    for k, (case, prec) in enumerate(specs):
        work(Simulation.from_case(case, precision=prec), want, k)
    sims = [Simulation.from_case(case, precision=prec) for case, prec in specs]
    threads = [threading.Thread(target=work, args=(s, got, k)) for k, s in enumerate(sims)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(got, want):
        assert isinstance(b, list), b
        assert isinstance(a, list), a
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
