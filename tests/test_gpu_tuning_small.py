"""Tunings of problems whose own chunk is smaller than 256 patterns: what is reported is what runs, and can be set again."""
import numpy as np
import pytest

from gpu_helpers import problem_from_oracle
from test_gpu_fp64_shapes import SHAPES, _alignment

pytestmark = pytest.mark.gpu
PAR = {"alpha": 1.0, "beta": 0.4, "theta": [0.7, 1.3, 0.9, 1.6, 0.8]}


def _same(a, b):
    return a["lnl"] == b["lnl"] and np.array_equal(a["grad_t"], b["grad_t"])


@pytest.mark.parametrize("precision_name", ["fp64", "mixed"])
@pytest.mark.parametrize("sites", [90, 300, 700])
def test_reported_shapes_are_the_ones_that_run(oracle, precision_name, sites):
    from hyphy3 import _capi
    tree = oracle.Tree.parse(SHAPES["caterpillar"])
    aln = _alignment(oracle, tree, sites, np.random.default_rng(sites))
    e = oracle.mg94(aln, PAR)
    prec = _capi.PREC_FP64 if precision_name == "fp64" else _capi.PREC_MIXED
    kw = dict(pi=aln.pi, Q=e["Q"], lam=e["lam"], U=e["U"], V=e["V"], precision=prec)
    bl = np.array(tree.branch_lengths)
    ctx = _capi.Context(0)
    pr = problem_from_oracle(ctx, oracle, tree, aln)
    pr.set_model(**kw)
    base, shapes = pr.eval(bl), pr.get_tuning()
    base = {"lnl": base["lnl"], "grad_t": base["grad_t"].copy()}
    # spelled out, the shapes are the same shapes
    pr.set_tuning(**shapes)
    assert pr.get_tuning() == shapes
    assert _same(pr.eval(bl), base)
    # the tuner reports what it installs and records, the second time (from its own record) as the first
    for _ in range(2):
        best, ms = pr.autotune(bl, reps=3)
        assert ms > 0 and pr.get_tuning() == best
        tuned = pr.eval(bl)
        tuned = {"lnl": tuned["lnl"], "grad_t": tuned["grad_t"].copy()}
        pr.set_tuning(**best)
        assert _same(pr.eval(bl), tuned)
        other = problem_from_oracle(ctx, oracle, tree, aln)
        other.set_model(**kw)
        assert other.get_tuning() == best
        assert _same(other.eval(bl), tuned)
        other.close()
    pr.close()
    ctx.close()


def test_chunks_that_a_tuning_can_ask_for(oracle):
    from hyphy3 import _capi
    tree = oracle.Tree.parse(SHAPES["polytomies"])
    aln = _alignment(oracle, tree, 400, np.random.default_rng(4))
    e = oracle.mg94(aln, PAR)
    bl = list(tree.branch_lengths)
    ref = np.array(oracle.branch_length_gradients(tree, aln, PAR, bl)[1])
    ctx = _capi.Context(0)
    pr = problem_from_oracle(ctx, oracle, tree, aln)
    for prec, tol in ((_capi.PREC_FP64, 1e-10), (_capi.PREC_MIXED, 1e-5)):      # each path's parity bound
        pr.set_model(pi=aln.pi, Q=e["Q"], lam=e["lam"], U=e["U"], V=e["V"], precision=prec)
        for chunk in (64, 128, 192, 320, 512, 1024):
            pr.set_tuning(a_chunk=chunk)
            assert pr.get_tuning()["a_chunk"] == min(chunk, 512)                # 400 patterns, padded to 512
            assert np.linalg.norm(pr.eval(np.array(bl))["grad_t"] - ref) <= tol * np.linalg.norm(ref)
    for chunk in (-64, 1, 63, 100, 200):
        with pytest.raises(_capi.H3GError):
            pr.set_tuning(a_chunk=chunk)
    pr.close()
    ctx.close()


@pytest.mark.parametrize("sites,least", [(90, 128), (300, 256), (700, 256), (1500, 256)])
def test_mixed_chunks_keep_both_halves_of_a_cta_busy(oracle, sites, least):
    # four 64-pattern tiles in a chunk, or all there are
    from hyphy3 import _capi
    tree = oracle.Tree.parse(SHAPES["cherries"])
    aln = _alignment(oracle, tree, sites, np.random.default_rng(sites))
    e = oracle.mg94(aln, PAR)
    ctx = _capi.Context(0)
    pr = problem_from_oracle(ctx, oracle, tree, aln)
    pr.set_model(pi=aln.pi, Q=e["Q"], lam=e["lam"], U=e["U"], V=e["V"], precision=_capi.PREC_MIXED)
    assert pr.get_tuning()["a_chunk"] >= least
    pr.close()
    ctx.close()
