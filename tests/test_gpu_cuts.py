"""The cut kernels at the edges of their shares: words per entry group, runs
shorter than a group's batch and longer, rows of no and of thousands of
entries, blocks of rows of the non-integer sum."""
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


def star(n):
    """Row 0 joined to every row but the last, which has no entry; +-1."""
    w = np.where(np.arange(n - 2) % 3 == 0, -1.0, 1.0)
    rowptr = np.concatenate([[0, n - 2], n - 2 + np.arange(1, n - 1), [2 * (n - 2)]]).astype(np.int32)
    col = np.concatenate([np.arange(1, n - 1), np.zeros(n - 2)]).astype(np.int32)
    return sbx.Graph(n, rowptr, col, np.concatenate([w, w]), w.sum())


def real(g, seed):
    rng = np.random.default_rng(seed)
    r = np.repeat(np.arange(g.n, dtype=np.int64), np.diff(g.rowptr))
    _, at = np.unique(np.minimum(r, g.col) * g.n + np.maximum(r, g.col), return_inverse=True)
    w = rng.uniform(-1, 1, at.max() + 1)
    return sbx.Graph(g.n, g.rowptr, g.col, w[at], float(w.sum()))


GRAPHS = [("torus", lambda: sbx.gen_torus(20, 20, seed=2)), ("rmat", lambda: sbx.gen_rmat(12, 8, seed=2)),
          ("star", lambda: star(3001)), ("er", lambda: sbx.gen_er(60, 0.5, pm1=True, seed=2))]


def check(ctx, oracle, g, agents):
    _, cut = ctx.solve(ctx.problem(g), sbx.params(dt=0.5, steps=100, agents=agents, seed=4, kernel=sbx.KERNEL_STREAM,
                                                  flags=sbx.FLAG_NO_TUNE))
    _, _, s = ctx.state(g.n, agents)
    assert np.array_equal(cut, oracle.cut(oracle_graph(oracle, g), s, agents))


@pytest.mark.parametrize("agents", [1, 64, 97, 200, 400, 1056])
@pytest.mark.parametrize("name,make", GRAPHS)
def test_unit_cuts_equal_the_oracles(ctx, oracle, name, make, agents):
    check(ctx, oracle, make(), agents)


@pytest.mark.parametrize("n,agents", [(50, 1), (700, 33), (4097, 1024)])
def test_real_cuts_equal_the_oracles(ctx, oracle, n, agents):
    check(ctx, oracle, real(sbx.gen_rgg(n, 8.0, seed=n), n), agents)
