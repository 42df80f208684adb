"""The resident FP64 kernel (small graphs, chosen by itself) against the
oracle: bit-exact states, cuts and windows, fused and unfused, with and without
the early exit, at row counts around a warp and agents around a word."""
import numpy as np
import pytest

import sbx
from conftest import oracle_graph

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sbx.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("fused", [1, 0])
@pytest.mark.parametrize("uw", [0, 1])
@pytest.mark.parametrize("n,agents", [(9, 1), (31, 31), (33, 33), (300, 64)])
def test_small_fp64_solves_equal_the_oracles(ctx, oracle, fused, uw, n, agents):
    g = sbx.gen_er(n, min(1.0, 8.0 / (n - 1)), pm1=True, seed=n)
    kw = dict(dt=0.25, steps=900, agents=agents, seed=n + 1, fused=fused, threshold=3)
    r, cut = ctx.solve(ctx.problem(g), sbx.params(precision=sbx.F64, update_window=uw, **kw))
    assert r["kernel_used"] == sbx.KERNEL_RESIDENT
    x, y, s = ctx.state(g.n, agents)
    o = oracle.maxcut_solve(oracle_graph(oracle, g), oracle.params(uw=uw, **kw), want_state=True)
    assert r["steps_run"] == o["result"]["steps_run"] and r["bifurcated"] == o["result"]["bifurcated"]
    np.testing.assert_array_equal(cut, o["cut"])
    np.testing.assert_array_equal(s, o["spins"])
    np.testing.assert_array_equal(x, o["x"])
    np.testing.assert_array_equal(y, o["y"])
