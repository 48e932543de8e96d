"""The work that programs have this library do, for timing it.

Each case is one call pattern of the package over sizes that the benchmark workloads, the tests and
the analyses use: from an 8-taxon gene to the 1024-taxon, 5000-codon alignment.  Alignments are
simulated under MG94xREV down random trees (branch lengths ~ Exp), like the benchmark's.  An
optimiser never evaluates one point twice, so a pass of the likelihood cases evaluates two different
parameter points, with the model installed anew where the parameters belong to it.

exact() restates the quantities in FP64 with plain torch: transition matrices by matrix_exp,
pruning with per-node scaling, gradients by automatic differentiation.
"""
import math
import pathlib
import sys

import numpy as np
import torch

_PYTHON = str(pathlib.Path(__file__).resolve().parent.parent / "hyphy-3_b200" / "python")
if _PYTHON not in sys.path:
    sys.path.insert(0, _PYTHON)

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"

# ------------------------------------------------------------------------------- genetic code
# amino acids of the 64 codons, nucleotides in A, C, G, T order, first position slowest
_AMINO = "KNKNTTTTRSRSIIMIQHQHPPPPRRRRLLLLEDEDAAAAGGGGVVVV*Y*YSSSS*CWCLFLF"
_NUC = "ACGT"
_SENSE = [c for c in range(64) if _AMINO[c] != "*"]
S = len(_SENSE)                                       # 61
_POS = np.array([[c >> 4, (c >> 2) & 3, c & 3] for c in _SENSE])
_PAIRS = [(0, 1), (0, 3), (1, 2), (1, 3), (2, 3)]     # AC AT CG CT GT (AG = 1)


def _steps():
    """Per codon pair: one-nucleotide change, synonymous, its position, from and to."""
    one = np.zeros((S, S), bool)
    syn = np.zeros((S, S), bool)
    at = np.zeros((3, S, S), int)
    for i in range(S):
        for j in range(S):
            d = np.flatnonzero(_POS[i] != _POS[j])
            if len(d) == 1:
                one[i, j] = True
                syn[i, j] = _AMINO[_SENSE[i]] == _AMINO[_SENSE[j]]
                at[:, i, j] = d[0], _POS[i, d[0]], _POS[j, d[0]]
    return one, syn, at


_ONE, _SYN, _AT = _steps()

# Text of a cell: the sense codons, a gap, and codons known up to purine / pyrimidine at the third position.
GAP = S
_TOKENS = [_NUC[a] + _NUC[b] + _NUC[c] for a, b, c in _POS] + ["---"] + \
          [_NUC[p >> 2] + _NUC[p & 3] + y for p in range(16) for y in "RY"]
_TEXT = np.array(_TOKENS, dtype="S3")


def _token_sets():
    """[tokens, 61]: the sense codons each token may stand for."""
    v = np.zeros((len(_TOKENS), S))
    v[:S] = np.eye(S)
    v[GAP] = 1.0
    for k in range(32):
        for s, c in enumerate(_SENSE):
            if c >> 2 == k >> 1 and (c & 1) == (k & 1):       # R = A, G (even), Y = C, T (odd)
                v[S + 1 + k, s] = 1.0
    return v


def _generator(theta, beta, pos, alpha=1.0):
    """MG94xREV generators [len(beta), 61, 61], differentiable in theta and beta."""
    dev = beta.device
    r = torch.ones(4, 4, dtype=torch.float64, device=dev)
    idx = torch.zeros(4, 4, dtype=torch.long, device=dev)
    full = torch.cat([torch.ones(1, dtype=torch.float64, device=dev), theta])
    for x, (a, b) in enumerate(_PAIRS):
        idx[a, b] = idx[b, a] = x + 1
    r = full[idx]
    p, f, t = (torch.as_tensor(a, device=dev) for a in _AT)
    base = r[f, t] * pos[p, t] * torch.as_tensor(_ONE, device=dev)
    syn = torch.as_tensor(_SYN, device=dev)
    q = base[None] * torch.where(syn[None], torch.full_like(base, alpha)[None], beta[:, None, None])
    return q - torch.diag_embed(q.sum(2))


# ------------------------------------------------------------------------------- trees and alignments
def _tree(kind, taxa, mean, rng):
    """An unrooted binary tree in Newick creation order: (parent, length, leaf number or -1)."""
    kids = {0: []}
    if kind == "yule":                                # split a random leaf until there are enough
        kids[0] = [1, 2, 3]
        leaves, nxt = [1, 2, 3], 4
        while len(leaves) < taxa:
            u = leaves.pop(int(rng.integers(len(leaves))))
            kids[u] = [nxt, nxt + 1]
            leaves += [nxt, nxt + 1]
            nxt += 2
    else:                                             # insert each taxon on a random branch
        kids[0] = [1, 2, 3]
        up, nxt = {1: 0, 2: 0, 3: 0}, 4
        edges = [1, 2, 3]
        for _ in range(taxa - 3):
            e = edges[int(rng.integers(len(edges)))]
            mid, leaf = nxt, nxt + 1
            nxt += 2
            u = up[e]
            kids[u][kids[u].index(e)] = mid
            kids[mid] = [e, leaf]
            up[mid], up[e], up[leaf] = u, mid, mid
            edges += [mid, leaf]
    parent, leaf_no, stack, n_leaf = [], [], [(0, -1)], 0
    while stack:                                      # preorder, children in order
        u, p = stack.pop()
        i = len(parent)
        parent.append(p)
        ch = kids.get(u, [])
        if ch:
            leaf_no.append(-1)
            stack += [(c, i) for c in reversed(ch)]
        else:
            leaf_no.append(n_leaf)
            n_leaf += 1
    length = rng.exponential(mean, size=len(parent))
    length[0] = 0.0
    return np.array(parent), length, np.array(leaf_no)


def _children(parent):
    kids = [[] for _ in parent]
    for i, p in enumerate(parent):
        if p >= 0:
            kids[p].append(i)
    return kids


def _newick(parent, length, leaf_no):
    kids = _children(parent)
    text = [""] * len(parent)
    for u in range(len(parent) - 1, -1, -1):          # children have larger ids
        s = "(" + ",".join(text[c] for c in kids[u]) + ")" if kids[u] else f"t{leaf_no[u]}"
        text[u] = s + (f":{length[u]:.10g}" if u else ";")
        for c in kids[u]:
            text[c] = ""
    return text[0]


def _simulate(parent, length, leaf_no, sites, theta, pos, omegas, omega_w, rates, rate_w, gaps, rng):
    """Tokens [taxa, sites] of sequences evolved down the tree."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(rng.integers(1 << 40)))
    th, ps, om = (torch.as_tensor(np.asarray(x, float), device=DEVICE) for x in (theta, pos, omegas))
    q = _generator(th, om, ps)
    codon = torch.as_tensor(_POS, device=DEVICE)
    pi = ps[0][codon[:, 0]] * ps[1][codon[:, 1]] * ps[2][codon[:, 2]]
    pi = pi / pi.sum()
    sq = pi.sqrt()
    lam, e = torch.linalg.eigh((sq[:, None] * q / sq[None, :] + (sq[:, None] * q / sq[None, :]).transpose(1, 2)) / 2)
    u, v = e / sq[:, None], e.transpose(1, 2) * sq[None, None, :]
    cls = torch.as_tensor(rng.choice(len(omegas), size=sites, p=np.asarray(omega_w) / np.sum(omega_w)), device=DEVICE)
    rt = torch.as_tensor(rng.choice(len(rates), size=sites, p=np.asarray(rate_w) / np.sum(rate_w)), device=DEVICE)
    combo = cls * len(rates) + rt
    rate = torch.as_tensor(np.asarray(rates, float), device=DEVICE)
    depth = np.zeros(len(parent), int)
    for i in range(1, len(parent)):
        depth[i] = depth[parent[i]] + 1
    state = torch.zeros(len(parent), sites, dtype=torch.long, device=DEVICE)
    state[0] = torch.multinomial(pi, sites, replacement=True, generator=g)
    for d in range(1, depth.max() + 1):
        every = np.flatnonzero(depth == d)
        for k in range(0, len(every), 32):
            nodes = torch.as_tensor(every[k:k + 32], device=DEVICE)
            t = torch.as_tensor(length[every[k:k + 32]], device=DEVICE)
            ex = torch.exp(lam[None, :, None, :] * rate[None, None, :, None] * t[:, None, None, None])   # node, omega, rate, 61
            p = ((u[None, :, None] * ex[..., None, :]) @ v[None, :, None]).clamp_min(0)
            cum = (p / p.sum(-1, keepdim=True)).cumsum(-1).float().flatten(1, 2)                          # node, combo, 61, 61
            par = state[torch.as_tensor(parent[every[k:k + 32]], device=DEVICE)]
            rows = cum[torch.arange(len(nodes), device=DEVICE)[:, None], combo[None, :], par]
            x = torch.rand(len(nodes), sites, 1, device=DEVICE, generator=g)
            state[nodes] = (rows < x).sum(-1).clamp_max(S - 1)
    at_leaf = np.flatnonzero(leaf_no >= 0)
    tok = state[torch.as_tensor(at_leaf, device=DEVICE)]
    if gaps > 0:
        x = torch.rand(tok.shape, device=DEVICE, generator=g)
        amb = S + 1 + 2 * (4 * codon[tok, 0] + codon[tok, 1]) + (codon[tok, 2] & 1)
        tok = torch.where(x < gaps, torch.full_like(tok, GAP), torch.where(x < 1.33 * gaps, amb, tok))
    return tok.to(torch.uint8).cpu().numpy()


_OMEGAS = {1: ([0.5], [1.0]), 2: ([0.2, 2.0], [0.8, 0.2]), 3: ([0.1, 1.0, 5.0], [0.6, 0.3, 0.1])}
_RATES = {1: ([1.0], [1.0]), 2: ([0.4, 1.6], [0.5, 0.5]), 3: ([0.25, 0.75, 2.0], [1 / 3] * 3),
          4: ([0.03, 0.28, 0.92, 2.77], [0.25] * 4)}


def _data(case, seed):
    """Everything a case's inputs are made of, from the seed alone."""
    rng = np.random.default_rng([int(seed) & 0x7FFFFFFF, 20261205])
    kind = case.get("tree", "random")
    parent, length, leaf_no = _tree(kind, case["taxa"], 0.05 if kind == "yule" else 0.1, rng)
    theta, pos = rng.uniform(0.5, 2.0, 5), rng.dirichlet(np.ones(4) * 4, size=3)
    K, M = case.get("classes", 1), case.get("rates", 1)
    om, ow = _OMEGAS[K]
    rt, rw = _RATES[M]
    sites = (case["sites"] + 1) // 2 if case["kind"] == "compress" else case["sites"]
    tok = _simulate(parent, length, leaf_no, sites, theta, pos, om, ow, rt, rw, case.get("gaps", 0.0), rng)
    points = []
    for _ in range(2):                                # two steps of an optimiser around the truth
        points.append({"bl": length * rng.uniform(0.8, 1.25, len(length)) + 1e-4 * (np.arange(len(length)) > 0),
                       "theta": theta * rng.uniform(0.9, 1.1, 5), "omegas": np.asarray(om) * rng.uniform(0.8, 1.25, K),
                       "omega_bg": 0.4 * rng.uniform(0.8, 1.25), "weights": rng.dirichlet(np.asarray(ow) * 50),
                       "rates": np.asarray(rt), "rate_w": np.asarray(rw)})
    test = rng.uniform(size=len(parent)) < 0.5
    return {"parent": parent, "length": length, "leaf_no": leaf_no, "tok": tok, "points": points, "test": test,
            "theta": theta}


def _alignment(d):
    import hyphy3
    names = [f"t{i}" for i in range(len(d["tok"]))]
    return hyphy3.Alignment.from_sequences(names, [_TEXT[r].tobytes().decode() for r in d["tok"]], "Universal", device=True)


def _params(theta, beta):
    import hyphy3
    p = hyphy3.MG94Parameters()
    p.theta_AC, p.theta_AT, p.theta_CG, p.theta_CT, p.theta_GT = (float(x) for x in theta)
    p.beta = float(beta)
    return p


def _gene_sizes(case):
    """Taxa and codons of the genes: uneven, the same for every seed."""
    rng = np.random.default_rng([case["genes"], case["taxa"], case["sites"]])
    return [{"kind": "branch", "taxa": int(rng.integers(8, case["taxa"] + 1)), "sites": int(rng.integers(100, case["sites"] + 1))}
            for _ in range(case["genes"])]


def _problem(ctx, d, aln):
    from hyphy3 import _capi
    states, masks, weights = aln.pattern_arrays()
    leaf = d["leaf_no"] >= 0
    return _capi.Problem(ctx, d["parent"].astype(np.int32), leaf.astype(np.uint8), d["leaf_no"].astype(np.int32), states, masks,
                         weights)


# ------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call: branch gradients of one gene (the 8-taxon configuration), where launches and host work count
        {"name": "branch_8x300", "kind": "branch", "taxa": 8, "sites": 300},
        # a step of a global MG94 fit with a test / background split, at the size of the test suite's genes: every
        # evaluation has another omega, so the model is installed and diagonalised each time
        {"name": "joint_23x254", "kind": "joint", "taxa": 23, "sites": 254, "background": True},
        # a step of a BUSTED fit (the 64-taxon configuration: 3 omega classes, gaps and ambiguous codons), FP64
        {"name": "mixture_64x1000", "kind": "mixture", "taxa": 64, "sites": 1000, "classes": 3, "gaps": 0.03},
        # the same through torch.autograd in single precision and the split-precision path
        {"name": "mixed_64x1000", "kind": "mixed", "taxa": 64, "sites": 1000, "classes": 3, "gaps": 0.03},
        # the largest configuration: 1024 taxa, 5000 codons, 2 omega classes x 4 rates, through torch.autograd
        {"name": "mixed_1024x5000", "kind": "mixed", "taxa": 1024, "sites": 5000, "classes": 2, "rates": 4, "tree": "yule"},
        # the same tree and model in FP64 on a shorter alignment
        {"name": "mixture_1024x1200", "kind": "mixture", "taxa": 1024, "sites": 1200, "classes": 2, "rates": 4, "tree": "yule"},
        # values only (line searches, per-site evidence ratios): 3 omega classes x 3 synonymous rates
        {"name": "value_256x2000", "kind": "value", "taxa": 256, "sites": 2000, "classes": 3, "rates": 3},
        # many genes of uneven size in one batch (a step of their joint branch-length fit), FP64
        {"name": "genes_24", "kind": "genes", "genes": 24, "taxa": 512, "sites": 3000},
        # per-site fits: FEL on the 256-taxon tree, 400 codons of it
        {"name": "fel_256x400", "kind": "fel", "taxa": 256, "sites": 400, "classes": 3},
        # MEME on a gene of the size that the reference analyses are shown on
        {"name": "meme_18x120", "kind": "meme", "taxa": 18, "sites": 120, "classes": 3},
        # a step of the nucleotide GTR fit that every analysis starts with
        {"name": "gtr_256x1000", "kind": "gtr", "taxa": 256, "sites": 1000},
        # loading: translation, counts and pattern compression of an alignment in host memory
        {"name": "compress_512x12000", "kind": "compress", "taxa": 512, "sites": 12000, "gaps": 0.02},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["branch", "joint", "mixture", "mixture", "mixed", "mixed", "mixed", "value", "genes", "fel", "meme", "gtr",
                       "compress"])
    gaps = rng.choice([0.0, 0.02])
    if kind == "genes":
        return {"kind": kind, "genes": _log(rng, 2, 20), "taxa": _log(rng, 16, 512), "sites": _log(rng, 150, 3000)}
    if kind == "fel":
        return {"kind": kind, "taxa": _log(rng, 10, 256), "sites": _log(rng, 60, 400), "classes": 3, "gaps": gaps}
    if kind == "meme":
        return {"kind": kind, "taxa": _log(rng, 8, 18), "sites": _log(rng, 40, 120), "classes": 3, "gaps": gaps}
    if kind == "compress":
        return {"kind": kind, "taxa": _log(rng, 64, 512), "sites": _log(rng, 300, 12000), "gaps": gaps}
    if kind in ("branch", "joint", "gtr"):
        case = {"kind": kind, "taxa": _log(rng, 6, 256), "sites": _log(rng, 80, 2000), "gaps": gaps}
        return dict(case, background=rng.random() < 0.5) if kind == "joint" else case
    case = {"kind": kind, "taxa": _log(rng, 8, 1024), "sites": _log(rng, 100, 5000 if kind == "mixed" else 2000),
            "classes": rng.choice([1, 2, 3]), "rates": rng.choice([1, 2, 3, 4]), "gaps": gaps, "tree": rng.choice(["random", "yule"])}
    cells = case["taxa"] * case["sites"] * case["rates"]
    most = 1024 * 5000 * 4 if kind == "mixed" else 1024 * 1200 * 4
    if cells > most:                                  # stay below the largest listed one
        case["sites"] = case["sites"] * most // cells
    return case


def prepare(case, seed):
    import hyphy3
    from hyphy3 import _capi
    kind = case["kind"]
    if kind == "genes":
        ctx = _capi.Context(0)
        rng = np.random.default_rng([int(seed) & 0x7FFFFFFF, 7])
        probs, bls = [], []
        for one in _gene_sizes(case):
            d = _data(one, int(rng.integers(1 << 30)))
            aln = _alignment(d)
            probs.append(_problem(ctx, d, aln))
            bls.append([p["bl"] for p in d["points"]])
            q = _generator(torch.as_tensor(d["theta"]), torch.tensor([0.5], dtype=torch.float64),
                           torch.as_tensor(np.array(aln.pos_nuc_frequencies))).numpy()
            probs[-1].model_of_case = {"pi": np.array(aln.codon_frequencies), "Q": q}
        batch = _capi.Batch(ctx, probs, 8)
        for p in probs:
            p.set_model(**p.model_of_case)
        return {"kind": kind, "batch": batch, "points": [[b[i] for b in bls] for i in range(2)], "ctx": ctx}
    d = _data(case, seed)
    if kind == "compress":
        # columns of a deep alignment are all distinct: half of the sites are new ones, the others repeat them
        rng = np.random.default_rng([int(seed) & 0x7FFFFFFF, 11])
        new = d["tok"].shape[1]
        cols = rng.permutation(np.concatenate([np.arange(new), rng.integers(0, new, case["sites"] - new)]))
        text = np.ascontiguousarray(_TEXT[d["tok"][:, cols]])
        rows = text.view(np.uint8).reshape(len(text), -1)
        sense = np.full(64, -1, np.int8)
        sense[_SENSE] = np.arange(S)
        return {"kind": kind, "ctx": _capi.Context(0), "rows": np.ascontiguousarray(rows), "sense": sense}
    aln = _alignment(d)
    if kind in ("fel", "meme"):
        ctx = _capi.Context(0)
        pos, pi = torch.as_tensor(np.array(aln.pos_nuc_frequencies)), np.array(aln.codon_frequencies)
        th = torch.as_tensor(d["theta"])
        q = [_generator(th, torch.tensor([b], dtype=torch.float64), pos, a)[0].numpy() for a, b in ((1.0, 0.0), (0.0, 1.0), (1.0, 0.5))]
        mu = -float(pi @ np.diag(q[2]))
        for m in q[:2]:
            np.fill_diagonal(m, 0.0)
        return {"kind": kind, "ctx": ctx, "problem": _problem(ctx, d, aln),
                "site": np.array(aln.site_to_pattern), "model": {"pi": pi, "Qs": q[0], "Qn": q[1], "branch_lengths": d["points"][0]["bl"] * 3.0 / mu}}
    tree = hyphy3.Tree.from_newick(_newick(d["parent"], d["length"], d["leaf_no"]))
    st = {"kind": kind, "tree": tree, "points": d["points"]}
    if kind == "gtr":
        aln = aln.to_nucleotide_alignment()
    st["aln"], st["site"] = aln, np.array(aln.site_to_pattern)
    if kind == "gtr":
        return st
    st["test"] = [bool(x) for x in d["test"]] if case.get("background") else None
    if kind == "branch":
        st["params"] = _params(d["theta"], 0.5)
    if kind == "mixed":                               # single-precision parameters of a torch program
        for p in d["points"]:
            p["tensors"] = [torch.tensor(p[k], dtype=torch.float32, requires_grad=True) for k in ("bl", "omegas", "weights", "theta")]
    return st


def run(state):
    import hyphy3
    kind = state["kind"]
    if kind == "compress":
        return state["ctx"].alignment_compress(state["rows"], state["sense"])
    if kind == "genes":
        out = []
        for bls in state["points"]:
            r = state["batch"].eval(bls)
            out.append({"lnl": np.array([g["lnl"] for g in r]), "grad": np.concatenate([g["grad_t"] for g in r])})
        return out
    if kind in ("fel", "meme"):                       # a row per site, as the analyses report
        r = state["problem"].fel_run(**state["model"]) if kind == "fel" else state["problem"].meme_run(**state["model"])
        return {k: v[state["site"]] for k, v in r.items()}
    tree, aln = state["tree"], state["aln"]
    out = []
    hyphy3.set_precision("mixed" if kind == "mixed" else "fp64")
    for p in state["points"]:
        if kind == "branch":
            lnl, grad = hyphy3.compute_branch_length_gradients(tree, aln, state["params"], p["bl"])
            out.append((lnl, np.array(grad)))
        elif kind == "joint":
            r = hyphy3.compute_joint_frechet_gradients(tree, aln, _params(p["theta"], p["omegas"][0]), p["bl"], state["test"],
                                                       p["omega_bg"] if state["test"] else -1.0)
            out.append((r["log_likelihood"], np.array(r["grad_branches"]),
                        np.array([r["grad_omega"], r["grad_omega_bg"]] + r["grad_theta"])))
        elif kind == "mixture":
            r = hyphy3.compute_mixture_gradients(tree, aln, _params(p["theta"], 1.0), p["bl"], p["omegas"], p["weights"], p["rates"],
                                                 p["rate_w"])
            syn = r["grad_syn_weights"] if len(p["rates"]) > 1 else []
            out.append((r["log_likelihood"], np.array(r["grad_branches"]),
                        np.concatenate([r["grad_omegas"], r["grad_weights"], r["grad_theta"], syn]),
                        np.array(r["site_log_likelihoods"])[state["site"]]))
        elif kind == "value":
            r = hyphy3.compute_mixture_gradients(tree, aln, _params(p["theta"], 1.0), p["bl"], p["omegas"], p["weights"], p["rates"],
                                                 p["rate_w"], want_gradients=False)
            out.append((r["log_likelihood"], np.array(r["site_log_likelihoods"])[state["site"]]))
        elif kind == "mixed":
            lnl = hyphy3.autograd.mixture_log_likelihood(*p["tensors"], tree, aln, syn_rates=list(p["rates"]),
                                                         syn_weights=list(p["rate_w"]))
            out.append((lnl.detach(), *torch.autograd.grad(lnl, p["tensors"])))
        elif kind == "gtr":
            g, m = hyphy3.GTRParameters(), hyphy3.GTRMatrix()
            g.theta_AC, g.theta_AT, g.theta_CG, g.theta_CT, g.theta_GT = (float(x) for x in p["theta"])
            m.update(g, aln.nuc_frequencies)
            lnl, site = hyphy3.compute_gtr_log_likelihood(tree, aln, m)
            at, grad, theta = hyphy3.compute_gtr_gradients(tree, aln, g, p["bl"])
            out.append((lnl, np.array(site)[state["site"]], at, np.array(grad), np.array(theta)))
    hyphy3.set_precision("fp64")
    return out


# ------------------------------------------------------------------------------- what a pass needs
def work(case):
    kind, T, sites = case["kind"], case.get("taxa"), case["sites"]
    if kind == "compress":
        return {"bytes": T * sites * 3 + sites * 8 + T * sites // 2 * 9, "flops": 0}
    if kind == "genes":
        T, sites = 260 if T >= 512 else (T + 8) // 2, (sites + 100) // 2
    n_int, br = T - 2, 2 * T - 3
    K, M = case.get("classes", 1), case.get("rates", 1)
    if kind in ("fel", "meme"):
        # about 60 evaluations of a site's likelihood (FEL), 300 of two components (MEME): two mat-vecs per internal branch
        # and component, one per leaf, and one symmetric eigenproblem (9 S^3) per component
        evals, comp = (60, 1) if kind == "fel" else (300, 2)
        return {"bytes": T * sites * 9 + 200.0 * sites, "flops": sites * evals * comp * (2.0 * S * S * (2 * n_int + T) + 9.0 * S ** 3)}
    s = 4 if kind == "gtr" else S
    cols = sites * (3 if kind == "gtr" else 1) * M
    passes = 1 if kind == "value" else 3              # inside, outside, gradient contraction
    one = 2.0 * s * s * n_int * cols * passes + 2.0 * s ** 3 * br * K * M * (1 if kind == "value" else 4)
    if kind == "gtr":
        one += 2.0 * s * s * n_int * cols
    n = 2 * case.get("genes", 1)
    return {"bytes": n * (T * sites + 8.0 * (br + sites)), "flops": n * one}


# ------------------------------------------------------------------------------- FP64 restatement
def _cf3x4(tok):
    """Codon and corrected positional frequencies of the tokens (CF3x4), and the nucleotides' overall ones."""
    counts = np.zeros((3, 4))
    n = np.bincount(tok.ravel(), minlength=len(_TOKENS))
    for k, text in enumerate(_TOKENS):
        for p in range(3):
            if text[p] in _NUC:
                counts[p, _NUC.index(text[p])] += n[k]

    def floor(f):
        f = np.maximum(f, 1e-8)
        return f / f.sum()
    overall = floor(counts.sum(0) / counts.sum())
    target = np.stack([floor(c / c.sum()) for c in counts])
    x = target.copy()

    def product():
        f = x[0][_POS[:, 0]] * x[1][_POS[:, 1]] * x[2][_POS[:, 2]]
        return f / f.sum()
    for _ in range(200):
        f, old = product(), x.copy()
        for p in range(3):
            x[p] *= target[p] / np.maximum(np.bincount(_POS[:, p], weights=f, minlength=4), 1e-12)
        x /= x.sum(1, keepdims=True)
        if np.abs(x - old).max() < 1e-14:
            break
    return product(), x, overall


def _patterns(tok):
    """Distinct columns [patterns, taxa], their weights and the pattern of each site."""
    cols, site, count = np.unique(tok.T, axis=0, return_inverse=True, return_counts=True)
    return cols, count.astype(float), site.reshape(-1)


def _prune(parent, leaf_no, table, cols, weight, P, pi, rate_w, want):
    """lnL, per-pattern lnL and, when wanted, the gradients of lnL in P [rates, nodes, s, s] and rate_w."""
    kids = _children(parent)
    M, n, s, _ = P.shape
    P = P.detach().requires_grad_(want)
    rw = rate_w.detach().requires_grad_(want)
    table = torch.as_tensor(table, dtype=torch.float64, device=P.device)
    sites = []
    chunk = max(64, int(2e9 / (8.0 * len(parent) * M * s)))
    for c0 in range(0, len(cols), chunk):
        obs = torch.as_tensor(cols[c0:c0 + chunk].astype(np.int64), device=P.device)
        w = torch.as_tensor(weight[c0:c0 + chunk], device=P.device)
        part, logs = [None] * n, torch.zeros(M, len(obs), dtype=torch.float64, device=P.device)
        for u in range(n - 1, -1, -1):
            if leaf_no[u] >= 0:
                part[u] = P[:, u] @ table[obs[:, leaf_no[u]]].T
                continue
            x = part[kids[u][0]]
            for c in kids[u][1:]:
                x = x * part[c]
            for c in kids[u]:
                part[c] = None
            top = x.detach().amax(1, keepdim=True)
            logs = logs + torch.log(top[:, 0])
            x = x / top
            part[u] = (pi[None, :, None] * x).sum(1) if u == 0 else P[:, u] @ x
        ll = torch.logsumexp(torch.log(rw)[:, None] + torch.log(part[0]) + logs, 0)
        if want:
            (ll * w).sum().backward()
        sites.append(ll.detach())
    site = torch.cat(sites)
    lnl = (site * torch.as_tensor(weight, device=site.device)).sum()
    return lnl, site, P.grad, rw.grad


def _through(make, dP, params):
    """Gradients in params of sum dP . P, P = make(rows) built in slices of the nodes [rates, rows, s, s]."""
    total = [torch.zeros_like(p) for p in params]
    for a in range(0, dP.shape[1], 128):
        got = torch.autograd.grad((make(slice(a, a + 128)) * dP[:, a:a + 128]).sum(), params, allow_unused=True)
        total = [t if g is None else t + g for t, g in zip(total, got)]
    return total


def _codon_exact(d, point, kind, test):
    dev = DEVICE
    f64 = dict(dtype=torch.float64, device=dev)
    pi, pos, _ = _cf3x4(d["tok"])
    pi_t, pos_t = torch.as_tensor(pi, **f64), torch.as_tensor(pos, **f64)
    single = kind == "mixed"

    def leaf(x):
        return torch.as_tensor(np.asarray(x, np.float32 if single else np.float64).astype(np.float64), **f64).requires_grad_(True)
    bl, theta, weights = leaf(point["bl"]), leaf(point["theta"]), leaf(point["weights"])
    omegas, om_bg = leaf(point["omegas"]), leaf([point["omega_bg"]])
    if kind in ("branch", "genes"):
        theta, omegas, weights = leaf(d["theta"]), leaf([0.5]), leaf([1.0])
    elif kind == "joint":
        weights = leaf([1.0])
    rates, rate_w = torch.as_tensor(point["rates"], **f64), torch.as_tensor(point["rate_w"], **f64)
    is_test = torch.as_tensor(test if test is not None else np.ones(len(d["parent"]), bool), device=dev)

    def make(rows):
        q = _generator(theta, torch.cat([omegas, om_bg]) if kind == "joint" else omegas, pos_t)
        t = bl[rows, None] * torch.ones(1, len(q), **f64)
        if kind == "joint":                           # unit-rate time of each model
            t = t * 3.0 / -(torch.diagonal(q, dim1=1, dim2=2) * pi_t).sum(1)
        p = torch.matrix_exp(q[None, None] * (rates[:, None, None] * t[None])[..., None, None])
        if kind == "joint":
            return torch.where(is_test[None, rows, None, None], p[:, :, 0], p[:, :, 1])
        return (weights[None, None, :, None, None] * p).sum(2)
    n = len(d["parent"])
    with torch.no_grad():
        P = torch.cat([make(slice(a, a + 128)) for a in range(0, n, 128)], 1)
    cols, weight, of = _patterns(d["tok"])
    lnl, site, dP, drw = _prune(d["parent"], d["leaf_no"], _token_sets(), cols, weight, P, pi_t, rate_w, kind != "value")
    if kind == "value":
        return lnl.item(), site.cpu().numpy()[of]
    dP[:, 0] = 0
    gb, gt, gw, go, gbg = _through(make, dP, [bl, theta, weights, omegas, om_bg])
    gb = gb.cpu().numpy()
    gb[0] = 0.0
    if kind in ("branch", "genes"):
        return lnl.item(), gb
    if kind == "joint":
        return lnl.item(), gb, torch.cat([go, gbg if test is not None else torch.zeros_like(gbg), gt]).cpu().numpy()
    if kind == "mixed":
        return tuple(torch.as_tensor(x).cpu() for x in (lnl, gb, go, gw, gt))
    return lnl.item(), gb, torch.cat([go, gw, gt] + [drw] * (len(rates) > 1)).cpu().numpy(), site.cpu().numpy()[of]


def _gtr_exact(d, point):
    f64 = dict(dtype=torch.float64, device=DEVICE)
    _, _, freq = _cf3x4(d["tok"])
    pi = torch.as_tensor(freq, **f64)
    iupac = {c: [c == x for x in _NUC] for c in _NUC} | {"-": [1] * 4, "R": [1, 0, 1, 0], "Y": [0, 1, 0, 1]}
    text = _TEXT[d["tok"]].view("S1").reshape(len(d["tok"]), -1)
    chars = sorted(iupac)
    cols, weight, of = _patterns(np.searchsorted(np.array(chars, dtype="S1"), text))
    table = np.array([iupac[c] for c in chars], float)
    bl = torch.as_tensor(point["bl"], **f64).requires_grad_(True)
    theta = torch.as_tensor(point["theta"], **f64).requires_grad_(True)

    def make(rows, t):
        idx = torch.zeros(4, 4, dtype=torch.long, device=DEVICE)
        for x, (a, b) in enumerate(_PAIRS):
            idx[a, b] = idx[b, a] = x + 1
        q = torch.cat([torch.ones(1, **f64), theta])[idx] * pi[None] * (1 - torch.eye(4, **f64))
        q = q - torch.diag(q.sum(1))
        q = q / -(torch.diagonal(q) * pi).sum()
        return torch.matrix_exp(q[None, None] * t[None, rows, None, None])
    every = slice(0, len(d["parent"]))
    rw = torch.ones(1, **f64)
    with torch.no_grad():
        at_tree, at_point = make(every, torch.as_tensor(_as_printed(d["length"]), **f64)), make(every, bl)
    lnl, site, _, _ = _prune(d["parent"], d["leaf_no"], table, cols, weight, at_tree, pi, rw, False)
    lnl2, _, dP, _ = _prune(d["parent"], d["leaf_no"], table, cols, weight, at_point, pi, rw, True)
    dP[:, 0] = 0
    gb, gt = _through(lambda rows: make(rows, bl), dP, [bl, theta])
    gb = gb.cpu().numpy()
    gb[0] = 0.0
    return lnl.item(), site.cpu().numpy()[of], lnl2.item(), gb, gt.cpu().numpy()


def _as_printed(length):
    return np.array([float(f"{x:.10g}") for x in length])


def exact(case, seed):
    kind = case["kind"]
    if kind in ("fel", "meme", "compress"):           # searches (their path is the result's definition) and whole numbers
        return None
    if kind == "genes":
        rng = np.random.default_rng([int(seed) & 0x7FFFFFFF, 7])
        parts = []
        for one in _gene_sizes(case):
            d = _data(one, int(rng.integers(1 << 30)))
            parts.append([_codon_exact(d, p, "genes", None) for p in d["points"]])
        return [{"lnl": np.array([g[i][0] for g in parts]), "grad": np.concatenate([g[i][1] for g in parts])} for i in range(2)]
    d = _data(case, seed)
    if kind == "gtr":
        return [_gtr_exact(d, p) for p in d["points"]]
    return [_codon_exact(d, p, kind, d["test"] if case.get("background") else None) for p in d["points"]]
