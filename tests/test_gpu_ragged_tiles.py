"""Tiles with left-over lanes at odd counts of 32-agent words, where the exact
tile walks one agent a lane and is about twice as slow: the tile that AUTO takes
is one, and it gives the state of the exact tile bit for bit."""
import numpy as np
import pytest

import sbx

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sbx.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("prec", [sbx.BF16, sbx.F16, sbx.F32])
@pytest.mark.parametrize("agents", [96, 160, 352, 608])
@pytest.mark.parametrize("fused", [1, 0])
@pytest.mark.parametrize("make", [lambda: sbx.gen_er(9000, 20.0 / 8999, pm1=True, seed=3),
                                  lambda: sbx.gen_rmat(16, 8, seed=3)])
def test_auto_leaves_lanes_over(ctx, prec, agents, fused, make):
    g = make()
    prob = ctx.problem(g)
    base = dict(dt=0.5, steps=2000, run_steps=200, agents=agents, seed=5, precision=prec, fused=fused,
                kernel=sbx.KERNEL_STREAM)
    r, cut = ctx.solve(prob, sbx.params(**base))
    assert agents % (r["lane_agents"] * r["row_lanes"]) != 0
    state = ctx.state(g.n, agents)
    r1, cut1 = ctx.solve(prob, sbx.params(lane_agents=1, row_lanes=32, **base))
    assert r1["lane_agents"] == 1
    for a, b in zip(state, ctx.state(g.n, agents)):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(cut, cut1)
