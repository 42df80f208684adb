"""Which kernel AUTO gives a batch class (+-1, fused): the on-chip kernel, the
resident batch, the plane kernel or the streaming step, at classes where one is
clearly the shortest, and the same cuts as the streaming step each time."""
import numpy as np
import pytest

import sbx

pytestmark = pytest.mark.gpu

CHIP, RESIDENT, PLANE, STREAM = "chip", "resident", "plane", "stream"


@pytest.fixture(scope="module")
def ctx():
    c = sbx.Context(0)
    yield c
    c.close()


def tori(count, side):
    return [sbx.gen_torus(side, side + i % 3, seed=i + 1) for i in range(count)]


def er(count, n, degree):
    return [sbx.gen_er(n - i, degree / (n - i - 1), pm1=True, seed=i + 1) for i in range(count)]


def ran(r):
    if r["staging"] == 3:
        return CHIP
    if r["kernel_used"] == sbx.KERNEL_RESIDENT:
        return RESIDENT
    return PLANE if r["count_mode"] == 4 else STREAM


@pytest.mark.parametrize("make,agents,prec,kernel", [
    (lambda: tori(1, 100), 64, sbx.BF16, STREAM),        # us a step: 3.4, on chip 5.9, resident batch 9.0
    (lambda: tori(1, 31), 64, sbx.BF16, RESIDENT),       # 1.4, on chip 1.8, streaming 2.5
    (lambda: tori(1, 31), 96, sbx.F16, RESIDENT),
    (lambda: tori(16, 31), 64, sbx.BF16, CHIP),          # 2.5, streaming 4.1, resident batch 12
    (lambda: tori(1, 100), 96, sbx.BF16, STREAM),        # 4.2, on chip 5.9
    (lambda: er(1, 10000, 60.0), 96, sbx.BF16, STREAM),  # 7.7, on chip 11.2
    (lambda: er(1, 15000, 24.0), 64, sbx.BF16, PLANE),   # 6.6, on chip 10.4
    (lambda: er(24, 4000, 24.0), 64, sbx.BF16, CHIP),
    (lambda: tori(1, 100), 32, sbx.F32, STREAM),         # 3.2, on chip 4.5
    (lambda: er(1, 15000, 60.0), 64, sbx.F32, STREAM),   # 8.8, on chip 13.3
    (lambda: er(24, 1000, 24.0), 64, sbx.F32, CHIP)])
def test_the_shortest_step_is_taken(ctx, make, agents, prec, kernel):
    gs = make()
    probs = [ctx.problem(g) for g in gs]
    base = dict(dt=0.5, steps=1000, run_steps=200, seed=4, precision=prec)
    res, got, _ = ctx.solve_batch(probs, [agents] * len(gs), sbx.params(**base))
    assert ran(res[0]) == kernel
    _, want, _ = ctx.solve_batch(probs, [agents] * len(gs), sbx.params(kernel=sbx.KERNEL_STREAM, **base))
    np.testing.assert_array_equal(got, want)
