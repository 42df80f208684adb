"""The resident FP64 kernel on dense and star-shaped +-1 graphs: bit-exact with
the oracle, and taken by AUTO only where its step is the shorter one."""
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


def star(n, seed):
    rng = np.random.default_rng(seed)
    w = rng.choice([-1.0, 1.0], n - 1)
    rowptr = np.concatenate([[0], np.arange(n) + n - 1])
    cols = np.concatenate([np.arange(1, n), np.zeros(n - 1, np.int64)])
    return sbx.Graph(n, rowptr, cols, np.concatenate([w, w]), float(w.sum()))


def dense(n, degree):
    return sbx.gen_er(n, min(1.0, degree / (n - 1)), pm1=True, seed=n)


@pytest.mark.parametrize("make,agents", [(lambda: star(200, 1), 40), (lambda: star(300, 2), 33),
                                         (lambda: dense(150, 149), 64), (lambda: dense(300, 200), 33)])
def test_equals_the_oracle(ctx, oracle, make, agents):
    g = make()
    kw = dict(dt=0.25, steps=600, agents=agents, seed=3, fused=1, threshold=3)
    r, cut = ctx.solve(ctx.problem(g), sbx.params(precision=sbx.F64, **kw))
    assert r["kernel_used"] == sbx.KERNEL_RESIDENT
    x, y, s = ctx.state(g.n, agents)
    o = oracle.maxcut_solve(oracle_graph(oracle, g), oracle.params(**kw), want_state=True)
    np.testing.assert_array_equal(cut, o["cut"])
    np.testing.assert_array_equal(s, o["spins"])
    np.testing.assert_array_equal(x, o["x"])
    np.testing.assert_array_equal(y, o["y"])


# sizes where one of the two steps is a fifth shorter or more
@pytest.mark.parametrize("make,agents,resident", [
    (lambda: dense(1000, 900), 128, False), (lambda: dense(600, 500), 304, False), (lambda: star(1000, 1), 128, False),
    (lambda: star(600, 1), 304, False), (lambda: dense(300, 12), 128, True), (lambda: dense(300, 200), 304, True),
    (lambda: dense(100, 64), 512, True), (lambda: dense(3000, 24), 128, False), (lambda: star(300, 1), 304, True)])
def test_taken_where_its_step_is_shorter(ctx, make, agents, resident):
    r, _ = ctx.solve(ctx.problem(make()), sbx.params(dt=0.5, steps=500, run_steps=100, agents=agents, precision=sbx.F64))
    assert r["kernel_used"] == (sbx.KERNEL_RESIDENT if resident else sbx.KERNEL_STREAM)
