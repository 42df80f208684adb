"""The FP32 TSP kernel with a row's cities split over one, two or four threads
(the agents per block decide): identical states, tours and lengths, at city
counts around the parts' edges."""
import numpy as np
import pytest

import sbx

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sbx.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("N", [2, 3, 8, 9, 16, 17, 24, 29, 32])
def test_parts_agree(ctx, N):
    xc, yc = sbx.gen_cities(N, 1000.0, seed=N)
    prob = ctx.tsp_problem_cities(xc, yc, sbx.DIST_EUC_2D_FLOAT)
    got = []
    # as many agents a block as one, two and four threads a row allow
    for block in (512 // N, max(1, 480 // N // 2), 1):
        r, lengths = ctx.solve(prob, sbx.params(dt=0.1, steps=500, agents=50, seed=3, kernel=sbx.KERNEL_RESIDENT,
                                                agents_per_block=block))
        assert r["agents_per_block"] == block
        got.append((lengths,) + ctx.state(N * N, 50) + ctx.tours(N, 50))
    for g in got[1:]:
        for a, b in zip(got[0], g):
            np.testing.assert_array_equal(a, b)
