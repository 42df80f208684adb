"""Agents per CTA of the resident FP32 TSP kernel: even waves when there are
more agents than CTAs hold, the same result for every number asked for."""
import numpy as np
import pytest
import torch

import sbx

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sbx.Context(0)
    yield c
    c.close()


def solve(ctx, cities, agents, **kw):
    xc, yc = sbx.gen_cities(cities, 1000.0, seed=cities)
    p = ctx.tsp_problem_cities(xc, yc, sbx.DIST_EUC_2D_FLOAT, A=1.0, penalty_scale=1.0)
    r, lengths = ctx.solve(p, sbx.params(dt=0.1, steps=400, agents=agents, seed=5, precision=sbx.F32, **kw))
    return r, (lengths,) + ctx.tours(cities, agents) + ctx.state(cities * cities, agents)


@pytest.mark.parametrize("cities", [9, 16, 17, 22, 29, 32])
@pytest.mark.parametrize("agents", [1, 152, 153, 1300, 2500, 5000])
def test_even_waves(ctx, cities, agents):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    r, _ = solve(ctx, cities, agents)
    ka = r["agents_per_block"]
    waves = -(-(-(-agents // ka)) // sms)
    assert ka == -(-agents // (waves * sms))


@pytest.mark.parametrize("cities,per_block", [(17, [1, 15, 16, 30]), (29, [8, 9, 17]), (32, [8, 9, 16]), (16, [1, 32])])
def test_agents_per_block_change_nothing(ctx, cities, per_block):
    _, want = solve(ctx, cities, 70)
    for ka in per_block:
        r, got = solve(ctx, cities, 70, agents_per_block=ka)
        assert r["agents_per_block"] == ka
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)
