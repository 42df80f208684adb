"""The on-chip batch kernel (count mode 4, staging 3) against the step per
launch: the same states and cuts, at row counts around the edges of its slices
and rounds, in clusters of one, two and four CTAs, with padded agents, for
every state type it takes."""
import numpy as np
import pytest

import sbx

pytestmark = pytest.mark.gpu

EDGES = [5, 31, 32, 33, 64, 100, 511, 513, 1023, 1025, 1500, 2100, 3000, 4200]


@pytest.fixture(scope="module")
def ctx():
    c = sbx.Context(0)
    yield c
    c.close()


def edges(pm1):
    sizes = EDGES + [700 + 13 * i for i in range(40)]
    return [sbx.gen_er(n, min(1.0, (6 + i % 30) / (n - 1)), pm1=pm1, seed=i) for i, n in enumerate(sizes)]


def past_16383():
    # a bin whose sign words have no complement beside them
    return [sbx.gen_rgg(16500, 12.0, seed=1)] + [sbx.gen_rgg(1000, 10.0, seed=2 + i) for i in range(60)]


def check(ctx, graphs, agents, prec, states):
    probs = [ctx.problem(g) for g in graphs]
    base = dict(dt=0.5, steps=2000, run_steps=200, seed=11, precision=prec)
    res, vals, _ = ctx.solve_batch(probs, agents, sbx.params(**base))
    assert res[0]["count_mode"] == 4 and res[0]["staging"] == 3
    got = [ctx.batch_state(i, graphs[i].n, agents[i]) for i in states]
    res2, vals2, _ = ctx.solve_batch(probs, agents, sbx.params(kernel=sbx.KERNEL_STREAM, **base))
    assert res2[0]["staging"] != 3
    np.testing.assert_array_equal(vals, vals2)
    for k, i in enumerate(states):
        for a, b in zip(got[k], ctx.batch_state(i, graphs[i].n, agents[i])):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("prec", [sbx.BF16, sbx.F16, sbx.F32])
@pytest.mark.parametrize("agents", [32, 64, 100])
@pytest.mark.parametrize("pm1", [True, False])
def test_edges_of_slices_rounds_and_clusters(ctx, prec, agents, pm1):
    gs = edges(pm1)
    ag = [agents - (i % 3 if agents > 32 else 0) for i in range(len(gs))]
    check(ctx, gs, ag, prec, range(len(EDGES)))


@pytest.mark.parametrize("prec", [sbx.BF16, sbx.F32])
def test_rows_past_the_complemented_planes(ctx, prec):
    gs = past_16383()
    check(ctx, gs, [64] * len(gs), prec, [0, 7])


@pytest.mark.parametrize("threads", [0, 512, 640, 1024])
def test_low_degree_with_a_cta_size(ctx, threads):
    # a CTA size of the plane kernel is taken, also by a low-degree class
    gs = [sbx.gen_torus(20 + i, 30, seed=i + 1) for i in range(6)]
    probs = [ctx.problem(g) for g in gs]
    base = dict(dt=0.5, steps=1000, run_steps=100, seed=3, precision=sbx.BF16)
    _, want, _ = ctx.solve_batch(probs, [64] * 6, sbx.params(kernel=sbx.KERNEL_STREAM, **base))
    _, got, _ = ctx.solve_batch(probs, [64] * 6, sbx.params(block_threads=threads, **base))
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("prec", [sbx.F32, sbx.BF16])
def test_streaming_tile_without_a_kernel(ctx, prec):
    # agents that fill few SMs: a tile asked for is run, one that no kernel has is refused
    g = sbx.gen_torus(80, 90, seed=2)
    p = ctx.problem(g)
    base = dict(dt=0.5, steps=1000, run_steps=100, agents=256, seed=3, precision=prec)
    res, got = ctx.solve(p, sbx.params(lane_agents=2, **base))
    assert res["lane_agents"] == 2
    _, want = ctx.solve(p, sbx.params(**base))
    np.testing.assert_array_equal(got, want)
    with pytest.raises(sbx.SbxError):
        ctx.solve(p, sbx.params(lane_agents=3, **base))
