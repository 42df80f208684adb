"""Agent counts whose 32-agent words do not fill a warp's vectors: the tile
the streaming kernel chooses leaves lanes over, and gives the state of the
one-agent-per-lane tile bit for bit."""
import numpy as np
import pytest

import sbx

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sbx.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("prec", [sbx.BF16, sbx.F32, sbx.F64])
@pytest.mark.parametrize("fused", [1, 0])
@pytest.mark.parametrize("agents", [65, 160, 224, 290, 608])
@pytest.mark.parametrize("make", [lambda: sbx.gen_rmat(11, 8, seed=3), lambda: sbx.gen_er(333, 0.1, pm1=True, seed=3)])
def test_left_over_lanes_change_nothing(ctx, prec, fused, agents, make):
    g = make()
    prob = ctx.problem(g)
    base = dict(dt=0.5, steps=2000, run_steps=200, agents=agents, seed=5, precision=prec, fused=fused,
                kernel=sbx.KERNEL_STREAM, update_window=0)
    r1, c1 = ctx.solve(prob, sbx.params(**base))
    s1 = ctx.state(g.n, agents)
    r2, c2 = ctx.solve(prob, sbx.params(lane_agents=1, row_lanes=32, **base))
    s2 = ctx.state(g.n, agents)
    assert r2["lane_agents"] == 1
    for a, b in zip(s1, s2):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(c1, c2)
    assert r1["bifurcated"] == r2["bifurcated"]
