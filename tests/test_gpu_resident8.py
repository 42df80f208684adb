"""The resident kernel of eight agents a CTA on rows of more neighbours than
one pass of its byte counters holds (120), against the streaming kernel: the
same states, for complete graphs around the passes' edges and a star."""
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
    w = np.random.default_rng(seed).choice([-1.0, 1.0], n - 1)
    rowptr = np.concatenate([[0], np.arange(n) + n - 1])
    cols = np.concatenate([np.arange(1, n), np.zeros(n - 1, np.int64)])
    return sbx.Graph(n, rowptr, cols, np.concatenate([w, w]), float(w.sum()))


def check(ctx, g, agents, prec, fused):
    prob = ctx.problem(g)
    base = dict(dt=0.5, steps=1000, run_steps=200, agents=agents, seed=3, precision=prec, fused=fused)
    out = []
    for kernel in (sbx.KERNEL_AUTO, sbx.KERNEL_STREAM):
        r, cut = ctx.solve(prob, sbx.params(kernel=kernel, **base))
        assert r["kernel_used"] == (sbx.KERNEL_RESIDENT if kernel == sbx.KERNEL_AUTO else sbx.KERNEL_STREAM)
        out.append((cut,) + ctx.state(g.n, agents))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("prec,fused", [(sbx.F32, 1), (sbx.F32, 0), (sbx.BF16, 1), (sbx.F16, 1)])
@pytest.mark.parametrize("pm1", [True, False])
@pytest.mark.parametrize("n", [120, 121, 122, 125, 129, 241, 242, 600])
def test_complete_graphs(ctx, prec, fused, pm1, n):
    check(ctx, sbx.gen_er(n, 1.0, pm1=pm1, seed=n), 21, prec, fused)


@pytest.mark.parametrize("prec", [sbx.F32, sbx.BF16])
@pytest.mark.parametrize("n", [122, 700, 2900])
def test_stars(ctx, prec, n):
    check(ctx, star(n, n), 21, prec, 1)
