"""Light rows (few neighbours, walked by records) beside a heavy one: the state
of the one-agent-per-lane tile at counts of segments around the warps' stride,
and no more time than the same rows without a heavy one."""
import numpy as np
import pytest

import sbx

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sbx.Context(0)
    yield c
    c.close()


def star(n, seed):
    rng = np.random.default_rng(seed)
    leaf, hub = np.arange(1, n), np.zeros(n - 1, np.int64)
    w = rng.choice([-1.0, 1.0], n - 1)
    rowptr = np.concatenate([[0], np.arange(n) + n - 1])
    return sbx.Graph(n, rowptr, np.concatenate([leaf, hub]), np.concatenate([w, w]), float(w.sum()))


@pytest.mark.parametrize("prec,lanes", [(sbx.F64, 2), (sbx.F32, 4), (sbx.BF16, 8)])
@pytest.mark.parametrize("n,segments", [(150, 1), (150, 3), (300, 16), (3000, 2), (9000, 5)])
def test_segments_of_light_rows(ctx, prec, lanes, n, segments):
    g = star(n, n)
    prob = ctx.problem(g)
    agents = 32 * lanes * segments
    base = dict(dt=0.5, steps=2000, run_steps=200, agents=agents, seed=5, precision=prec, kernel=sbx.KERNEL_STREAM,
                row_lanes=32)
    out = []
    for v in (lanes, 1):
        _, cut = ctx.solve(prob, sbx.params(lane_agents=v, **base))
        out.append((cut,) + ctx.state(g.n, agents))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("prec", [sbx.F64, sbx.F32, sbx.F16])
@pytest.mark.parametrize("degree", [1.0, 3.0, 6.5, 9.0])
@pytest.mark.parametrize("fused", [1, 0])
@pytest.mark.parametrize("agents", [32, 256, 300, 1536])
def test_records_by_the_share_of_light_rows(ctx, prec, degree, fused, agents):
    # no heavy row: records where at least half of the rows are light (here up
    # to a mean degree of about 6.5) in a state past 12 MB, the row pointers
    # otherwise
    g = sbx.gen_er(2500, degree / 2499, pm1=True, seed=int(10 * degree))
    prob = ctx.problem(g)
    base = dict(dt=0.5, steps=2000, run_steps=200, agents=agents, seed=5, precision=prec, fused=fused,
                kernel=sbx.KERNEL_STREAM)
    out = []
    for tile in ({}, dict(lane_agents=1, row_lanes=32)):
        _, cut = ctx.solve(prob, sbx.params(**tile, **base))
        out.append((cut,) + ctx.state(g.n, agents))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_many_segments_fill_the_gpu(ctx):
    # 300 rows of 16 segments: 1.2 times the time of rows that have no records;
    # whole rows a warp took 2.9 times
    base = dict(dt=0.5, steps=2000, run_steps=300, agents=1024, seed=5, precision=sbx.F64, kernel=sbx.KERNEL_STREAM)
    us = []
    for g in (star(300, 1), sbx.gen_er(300, 14.0 / 299, pm1=True, seed=1)):
        prob = ctx.problem(g)
        us.append(min(ctx.solve(prob, sbx.params(**base))[0]["time_us"] for _ in range(5)))
    assert us[0] < 2.0 * us[1], us
