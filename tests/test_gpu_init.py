"""The init kernel at the edges of its chunks and rounds: with dt = 0 the
steps leave the state as it began, so the state read back is glibc's rand()
stream, converted, rounded to the storage type and laid out."""
import numpy as np
import pytest

import sbx

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sbx.Context(0)
    yield c
    c.close()


def stored(v, prec):
    f = v.astype(np.float32)
    if prec == sbx.F64:
        return v
    if prec == sbx.F16:
        return f.astype(np.float16).astype(np.float64)
    if prec == sbx.BF16:
        u = f.view(np.uint32)
        u = (u + 0x7fff + ((u >> 16) & 1)) & np.uint32(0xffff0000)
        return u.view(np.float32).astype(np.float64)
    return f.astype(np.float64)


# one agent a row; a round's 31 agents and one more or less; padded agents; a
# whole number of rounds; chunks of more than one round (20 million outputs)
@pytest.mark.parametrize("prec", [sbx.F32, sbx.BF16, sbx.F16, sbx.F64])
@pytest.mark.parametrize("side,agents", [(3, 1), (4, 30), (4, 31), (5, 33), (31, 64), (100, 1024)])
def test_initial_state_is_the_rand_stream(ctx, oracle, prec, side, agents):
    g = sbx.gen_torus(side, side, seed=side)
    ctx.solve(ctx.problem(g), sbx.params(dt=0.0, steps=100, agents=agents, seed=agents + 5, precision=prec,
                                         kernel=sbx.KERNEL_STREAM, flags=sbx.FLAG_NO_TUNE))
    x, y, _ = ctx.state(g.n, agents)
    ox, oy = oracle.init_maxcut(g.n, agents, agents + 5)
    assert np.array_equal(x, stored(ox, prec))
    assert np.array_equal(y, stored(oy, prec))
