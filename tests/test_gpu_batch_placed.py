"""The on-chip batch kernel's plan in the rows' order (few steps so far) and
with its entries placed by bank: the same states."""
import numpy as np
import pytest

import sbx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [sbx.BF16, sbx.F32])
@pytest.mark.parametrize("pm1", [True, False])
def test_order_of_the_entries_changes_nothing(prec, pm1):
    gs = [sbx.gen_er(n, min(1.0, (3 + 5 * i) / (n - 1)), pm1=pm1, seed=i) for i, n in
          enumerate([5, 33, 100, 700, 1025, 1500, 2100, 3000, 4200, 900, 800, 600])]
    agents = [64] * len(gs)
    ctx = sbx.Context(0)
    probs = [ctx.problem(g) for g in gs]
    base = dict(dt=0.5, steps=5000, run_steps=400, seed=2, precision=prec)
    out = []
    for kw in (dict(kernel=sbx.KERNEL_STREAM), {}, {}, {}, {}):   # 400, 800, 1,200 and 1,600 steps of the plan
        res, vals, _ = ctx.solve_batch(probs, agents, sbx.params(**base, **kw))
        assert (res[0]["staging"] == 3) == (not kw)
        out.append([vals] + [a for i in range(len(gs)) for a in ctx.batch_state(i, gs[i].n, 64)])
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)
    ctx.close()


@pytest.mark.parametrize("prec", [sbx.BF16, sbx.F32])
def test_a_layout_that_does_not_fit_takes_another_kernel(prec):
    # clusters of one, two and four CTAs; the flag makes them report a misfit
    gs = [sbx.gen_er(n, 20.0 / (n - 1), pm1=True, seed=n) for n in [300, 700, 1500, 3000, 5000, 5100, 5200, 900, 1000]]
    agents = [64] * len(gs)
    ctx = sbx.Context(0)
    probs = [ctx.problem(g) for g in gs]
    base = dict(dt=0.5, steps=2000, run_steps=200, seed=2, precision=prec)
    res, want, _ = ctx.solve_batch(probs, agents, sbx.params(**base))
    assert res[0]["staging"] == 3
    res, got, _ = ctx.solve_batch(probs, agents, sbx.params(flags=sbx.FLAG_TEST_GIVEUP, **base))
    assert res[0]["staging"] != 3
    np.testing.assert_array_equal(got, want)
    res, got, _ = ctx.solve_batch(probs, agents, sbx.params(**base))   # the same batch does not try again
    assert res[0]["staging"] != 3
    np.testing.assert_array_equal(got, want)
    ctx.close()
