"""Installing a model: the arrays that reach the device, and problems told apart by their content."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,nm", [(1, 1), (4, 3), (61, 1), (61, 5), (64, 2)])
def test_installed_arrays(S, nm):
    # the eigensystem comes back as it was given, bit for bit, whatever was installed before
    from hyphy3 import _capi
    ctx = _capi.Context(0)
    pr = _capi.Problem(ctx, np.array([-1, 0, 0, 0], dtype=np.int32), np.array([0, 1, 1, 1], dtype=np.uint8),
                       np.array([-1, 0, 1, 2], dtype=np.int32), np.zeros((1, 3), dtype=np.int8),
                       np.zeros((1, 3), dtype=np.uint64), np.ones(1))
    rng = np.random.default_rng(S + nm)
    for n_dirs in (0, 2):
        U, V = rng.standard_normal((2, nm, S, S))
        lam = -rng.random((nm, S))
        pr.set_model(pi=np.full(S, 1 / S), Q=rng.standard_normal((nm, S, S)), lam=lam, U=U, V=V, class_w=np.full(nm, 1 / nm),
                     dQ=rng.standard_normal((n_dirs, nm, S, S)) if n_dirs else None, dQ_model=rng.standard_normal((nm, S, S)))
        for k in range(nm):
            e = pr.get_eigensystem(k)
            assert np.array_equal(e["lam"], lam[k]) and np.array_equal(e["U"], U[k]) and np.array_equal(e["V"], V[k])
    pr.close()
    ctx.close()


@pytest.mark.parametrize("taxa", [3, 8, 64, 67, 130])
def test_alignments_that_differ_in_one_state(taxa):
    # one taxon's codon, or the ambiguity code of its unresolved codon, changes: another problem, and the first
    # alignment's value comes back
    import _hyphy3 as h3
    names = [f"t{i}" for i in range(taxa)]
    tree = h3.Tree.from_newick("(" + ",".join(f"{n}:0.1" for n in names) + ");")
    rows = ["ATGAAACCC" if i % 2 else "ATGAAGCCT" for i in range(taxa)]
    at = taxa - 1

    def lnl(last):
        aln = h3.Alignment.from_sequences(names, rows[:at] + [last])
        return h3.compute_branch_length_gradients(tree, aln, h3.MG94Parameters())[0]

    variants = ["ATGAAACCC", "ATGAATCCC", "ATGAARCCC", "ATGAAYCCC", "ATGAANCCC", "ATG---CCC"]
    first = [lnl(v) for v in variants]
    assert [lnl(v) for v in variants] == first
    assert len(set(first[:5])) == 5
