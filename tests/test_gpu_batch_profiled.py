"""Batches whose members have kernel timing enabled while the step is captured: the launches
are then in one stream, in both forms of the sub-iteration loop (a loop node per suspension,
EIF_BATCH_SUBITER=branches, or the stage kernel), and the loops end as they do without it."""
import pytest

from ellipsesinflows_gb300 import Batch, Simulation
from test_gpu_batch import assert_same, members, subiter_mode  # noqa: F401

pytestmark = pytest.mark.gpu


def test_batch_with_profiled_members(gpu_lib, subiter_mode):  # noqa: F811
    specs = members()
    solo = [Simulation.from_case(f(), precision=p) for f, p in specs]
    together = [Simulation.from_case(f(), precision=p) for f, p in specs]
    for s in solo:
        s.advance(3)
    for s in together:
        s._call("profile_enable", s.ctx, 1)
    with Batch(together) as batch:
        batch.advance(3)
    for a, b in zip(solo, together):
        assert_same(a, b)
