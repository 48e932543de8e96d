"""Workspace of the mixed path: a gradient operand is stored, and has room, only where one is read."""
import numpy as np
import pytest

from gpu_helpers import problem_from_oracle
from test_gpu_fp64_shapes import SHAPES, _alignment

pytestmark = pytest.mark.gpu
PAR = {"alpha": 1.0, "beta": 0.4, "theta": [0.7, 1.3, 0.9, 1.6, 0.8]}
TREES = dict(SHAPES, binary="(((a:0.1,b:0.2):0.1,(c:0.3,d:0.05):0.2):0.1,((e:0.4,f:0.1):0.2,g:0.3):0.2);")


def _bytes(oracle, _capi, ctx, tree, sites):
    aln = _alignment(oracle, tree, sites, np.random.default_rng(sites))
    e = oracle.mg94(aln, PAR)
    pr = problem_from_oracle(ctx, oracle, tree, aln)
    pr.set_tuning(a_chunk=1024)
    pr.set_model(pi=aln.pi, Q=e["Q"], lam=e["lam"], U=e["U"], V=e["V"], precision=_capi.PREC_MIXED)
    b = pr.checkpoint_info()["workspace_bytes"]
    pr.close()
    return b


@pytest.mark.parametrize("shape", sorted(TREES))
def test_room_for_stored_operands_only(oracle, shape):
    from hyphy3 import _capi
    tree = oracle.Tree.parse(TREES[shape])
    n = tree.num_nodes()
    kids = [[c for c in range(n) if tree.parent[c] == u] for u in range(n)]
    internal = sum(1 for k in kids if k)
    stored = sum(1 for c in range(n) if tree.parent[c] >= 0 and not (not kids[c] and len(kids[tree.parent[c]]) == 2))
    ctx = _capi.Context(0)
    step = _bytes(oracle, _capi, ctx, tree, 200) - _bytes(oracle, _capi, ctx, tree, 100)      # 256 and 128 patterns
    # for 128 patterns more: FP32 D, messages, U and the stored operands; five exponents a node; four FP64 values and, per
    # node, two flags
    assert step == 128 * ((3 * internal + stored) * 64 * 4 + internal * 5 * 4 + 4 * 8) + internal * 2 * 4
    ctx.close()


@pytest.mark.parametrize("shape", sorted(TREES))
def test_shared_slots_of_a_batch(oracle, shape):
    # problems of other shapes evaluate in the same slot before and after: the same bits as alone
    from hyphy3 import _capi
    ctx = _capi.Context(0)
    probs, alone, bls = [], [], []
    for name in (shape, "binary", shape, "star", shape):
        tree = oracle.Tree.parse(TREES[name])
        aln = _alignment(oracle, tree, 150, np.random.default_rng(len(name)))
        e = oracle.mg94(aln, PAR)
        kw = dict(pi=aln.pi, Q=e["Q"], lam=e["lam"], U=e["U"], V=e["V"], precision=_capi.PREC_MIXED)
        pr = problem_from_oracle(ctx, oracle, tree, aln)
        pr.set_model(**kw)
        bls.append(np.array(tree.branch_lengths))
        r = pr.eval(bls[-1])
        alone.append((r["lnl"], r["grad_t"].copy()))
        probs.append((pr, kw))
    batch = _capi.Batch(ctx, [p for p, _ in probs], n_slots=1)
    for pr, kw in probs:
        pr.set_model(**kw)
    for (lnl, grad), r in zip(alone, batch.eval(bls)):
        assert r["lnl"] == lnl and np.array_equal(r["grad_t"], grad)
    batch.close()
    for pr, _ in probs:
        pr.close()
    ctx.close()
