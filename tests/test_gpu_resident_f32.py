"""The tensor-memory resident kernel with FP32 state (four agents a CTA; AUTO
takes it, it cannot be asked for): state, window spins, cuts and steps equal
the streaming kernel's bit for bit for all +1, +-1 and real weights, with and
without the early exit, at rows on both sides of tensor memory's 8,192 and at
the last that fits; and which sizes AUTO gives it."""
import numpy as np
import pytest

import sbx

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sbx.Context(0)
    yield c
    c.close()


def graph(n, degree, weights, seed):
    g = sbx.gen_er(n, degree / (n - 1), pm1=weights != "unit", seed=seed)
    if weights != "real":
        return g
    rng = np.random.default_rng(seed)
    r = np.repeat(np.arange(g.n, dtype=np.int64), np.diff(g.rowptr))
    edges, at = np.unique(np.minimum(r, g.col) * g.n + np.maximum(r, g.col), return_inverse=True)
    w = rng.uniform(-1.0, 1.0, edges.size)
    return sbx.Graph(g.n, g.rowptr, g.col, w[at], float(w.sum()))


@pytest.mark.parametrize("uw", [0, 1])
@pytest.mark.parametrize("weights", ["unit", "pm1", "real"])
@pytest.mark.parametrize("n,degree,agents", [(3300, 9.0, 453), (8192, 3.0, 450), (8193, 6.0, 450), (9217, 30.0, 604),
                                             (14101, 5.0, 450)])
def test_equals_streaming(ctx, uw, weights, n, degree, agents):
    g = graph(n, degree, weights, n)
    prob = ctx.problem(g)
    base = dict(dt=0.5, steps=1200, agents=agents, seed=9, precision=sbx.F32, update_window=uw,
                threshold=3 if uw else 0)
    r1, cut1 = ctx.solve(prob, sbx.params(**base))
    assert r1["kernel_used"] == sbx.KERNEL_RESIDENT_SPLIT and r1["agents_per_block"] == 4
    s1 = ctx.state(g.n, agents)
    r2, cut2 = ctx.solve(prob, sbx.params(kernel=sbx.KERNEL_STREAM, **base))
    s2 = ctx.state(g.n, agents)
    for a, b in zip(s1, s2):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(cut1, cut2)
    for k in ("steps_run", "windows_run", "bifurcated", "max", "ps"):
        assert r1[k] == r2[k], k


# sizes where one of the two steps is well over a fifth shorter
@pytest.mark.parametrize("n,degree,weights,agents,split", [
    (3136, 12.0, "pm1", 32, False), (3136, 12.0, "pm1", 608, True), (5929, 4.0, "pm1", 32, False),
    (5929, 4.0, "pm1", 1024, True), (14000, 5.0, "pm1", 64, False), (14000, 5.0, "pm1", 608, True),
    (12500, 16.0, "real", 480, True), (9000, 40.0, "real", 608, True), (9000, 85.0, "real", 100, False),
    (6000, 8.0, "real", 32, False), (14102, 4.0, "pm1", 608, False)])
def test_taken_where_its_step_is_shorter(ctx, n, degree, weights, agents, split):
    r, _ = ctx.solve(ctx.problem(graph(n, degree, weights, 1)),
                     sbx.params(dt=0.5, steps=1000, run_steps=100, agents=agents, precision=sbx.F32))
    assert r["kernel_used"] == (sbx.KERNEL_RESIDENT_SPLIT if split else sbx.KERNEL_STREAM)
