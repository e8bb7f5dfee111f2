"""A call whose launch CUDA refuses returns an error and leaves nothing behind: the next call on the context, of any
simulation, works."""
import numpy as np
import pytest

import elastic_cases as E
import vd_cases as V
from vd_cases import sw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family", ["el", "vd"])
def test_call_after_a_refused_launch(family):
    """The elastic gradient takes at most 65535 rows (one block row each in the correlation)."""
    ctx = sw._lib.Context(0)
    tall = E.small_case("mt", nt=12, nx=16, nz=66000, halo=2)
    shot = tall.shots[0]
    refused = E.GpuElastic(ctx, tall, gradient=True, check_freq=5)
    case = (E if family == "el" else V).small_case(nt=40, nx=60, nz=50, halo=6)
    sim = E.GpuElastic(ctx, case) if family == "el" else V.GpuVD(ctx, case)
    want = sim.forward(case.shots)
    with pytest.raises(sw._lib.SwError):
        refused.gradient([shot], [np.ones((12, 2, len(shot.rec)))])
    got = sim.forward(case.shots)
    refused.close()
    sim.close()
    ctx.close()
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
