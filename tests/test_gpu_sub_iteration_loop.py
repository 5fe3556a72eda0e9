"""The loop of kernels that runs the sub-iterations of larger suspensions (k_ibm_loop_f, k_sub_end,
the stage front on two streams) against single kernels one after another with a wait behind each
(k_ibm_sum_f or k_ibm_work_f, k_chunk_reduce, k_increment): bitwise the same state and counts.

Particle counts: multiples of the eight that a block of k_sub_end takes and the counts beside them.
Sizes: boxes of one row segment and of two, and of fewer rows than a warp takes at a time."""
import numpy as np
import pytest

from ellipsesinflows_gb300 import PREC_FP64, PREC_MIXED, Simulation, cases

pytestmark = pytest.mark.gpu


def run(case, prec):
    s = Simulation(case.config(precision=prec))
    s.push_fluid(*case.fluid())
    s.push_particles(case.particles)
    subs = [list(s.step()) for _ in range(2)]
    return [np.array(f) for f in s.pull_fluid()[:3]] + [np.array(s.pull_particles())], subs


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n,itot,a,b", [(271, 128, 0.02, 0.014), (272, 96, 0.02, 0.014), (273, 128, 0.006, 0.004),
                                        (279, 512, 0.02, 0.012), (3, 768, 0.09, 0.06)])
def test_loop_equals_single_kernels(n, itot, a, b, prec, gpu_lib, monkeypatch):
    case = cases.poiseuille(itot=itot, jtot=2 * itot, n=n, a=a, b=b, seed=7)
    got, subs = run(case, prec)
    monkeypatch.setenv("EIF_SYNC_DEBUG", "1")
    want, wsubs = run(case, prec)
    assert subs == wsubs
    for x, y in zip(got, want):
        assert np.array_equal(x, y)
