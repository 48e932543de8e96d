"""FP64 gradients around the number of branches up to which leaves and internal branches share a launch, bit for bit the
same with subtree checkpoints, whose blocks are small enough to share one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taxa", [4, 149, 150])                  # a caterpillar has 2 taxa - 3 such items: 295 and 297
@pytest.mark.parametrize("P", [1, 100])
def test_checkpointed_gradients_have_the_same_bits(taxa, P):
    from hyphy3 import _capi
    rng = np.random.default_rng(taxa + P)
    parent = [-1]
    at = 0
    for _ in range(taxa - 1):
        parent += [at, at]
        at = len(parent) - 1
    parent = np.array(parent, dtype=np.int32)
    n = parent.size
    leaf = np.array([u not in parent for u in range(n)], dtype=np.uint8)
    taxon = np.full(n, -1, dtype=np.int32)
    taxon[leaf == 1] = np.arange(taxa)
    states = rng.integers(0, 61, (P, taxa)).astype(np.int8)
    masks = np.uint64(1) << states.astype(np.uint64)
    lost = rng.random((P, taxa)) < 0.1
    states[lost], masks[lost] = -1, 0
    pi = rng.dirichlet(np.full(61, 8.0))
    q = rng.uniform(0.1, 1.0, (61, 61))
    q = (q + q.T) * pi[None, :]
    np.fill_diagonal(q, 0.0)
    np.fill_diagonal(q, -q.sum(1))
    bl = rng.uniform(0.01, 0.2, n)
    ctx = _capi.Context(0)
    pr = _capi.Problem(ctx, parent, leaf, taxon, states, masks, np.ones(P))
    out = []
    for target in (0, 9):
        pr.set_memory_budget(0, target)
        pr.set_model(pi=pi, Q=q)
        r = pr.eval(bl, _capi.WANT_LNL | _capi.WANT_GRAD_T)
        out.append((r["lnl"], r["grad_t"].copy()))
    pr.close()
    ctx.close()
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])
    assert np.all(np.isfinite(out[0][1])) and np.count_nonzero(out[0][1]) == n - 1
