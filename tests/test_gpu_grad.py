"""GPU adjoint gradient (pcsf_grad) against the oracle's outside pass and finite differences.

Tolerances: FP64 engine, per-branch d lpr / d t within 1e-7 relative (abs
floor 1e-8) of the oracle (the oracle differentiates P(t) = exp(tQ)
analytically, the kernel applies dP/dt = Q P to P after the clamp /
renormalise row rule); FP32 (compensated or blocked) per entry within 1e-4
relative plus 2e-6 per column of the region.  d lpr / d rho against a central difference of the
FP64 engine's lpr with h = 1e-5: within 1e-6 relative.
"""
import numpy as np
import pytest

import phylocsf_gb300 as P
from phylocsf_gb300 import synth
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu

_E = {}
_G = {}     # oracle gradients, shared by the precisions


def engine(name, prec):
    if (name, prec) not in _E:
        ps = synth.load_params(name)
        _E[(name, prec)] = P.Engine(ps.tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision=prec)
    return _E[(name, prec)]


def _data(name, lengths, seed):
    ps = synth.load_params(name)
    rng = np.random.default_rng(seed)
    gf = synth.gap_fractions(rng, len(lengths), ps.tree.nl, 0.05, 0.4, 0.2)
    return synth.simulate(ps, np.asarray(lengths), (np.arange(len(lengths)) % 2).astype(np.int32), gf, seed)


@pytest.fixture(scope="module", autouse=True)
def _fast():
    O.set_sparse_leaves(True)


@pytest.mark.parametrize("prec", ["fp64", "fp32c", "fp32b"])
@pytest.mark.parametrize("name", ["12flies", "29mammals", "58mammals", "100vertebrates"])
def test_branch_gradient_matches_oracle(prec, name):
    e = engine(name, prec)
    mc, mn, ot, tree = H.oracle_models(name)
    lengths = [90, 1, 200, 0] if name in ("12flies", "29mammals") else [90, 1, 333, 0, 700, 64]
    offs, leaves = _data(name, lengths, seed=21)
    b = e.batch(offs, leaves)
    for model, om in ((0, mc), (1, mn)):
        for rho in (0.3, 1.0, 2.5):
            lpr, db, drho, st = e.grad(b, model, rho)
            assert (st == 0).all()
            for r in range(len(offs) - 1):
                lv = H.u8_to_oracle(leaves[offs[r]:offs[r + 1]])
                key = (name, model, rho, r)
                if key not in _G:
                    _G[key] = O.grad_branches(om, ot, rho, lv)
                lo, go = _G[key]
                if lv.shape[0] == 0:
                    assert np.all(db[r] == 0.0) and lpr[r] == 0.0
                    continue
                if prec == "fp64":
                    assert lpr[r] == pytest.approx(lo, rel=1e-9)
                    err = np.abs(db[r] - go) - (1e-7 * np.abs(go) + 1e-8)
                    k = int(np.argmax(err))
                    assert err[k] <= 0, (model, rho, r, k, db[r][k], go[k], tree.branch[k])
                else:
                    # per entry: 1e-4 relative plus 2e-6 per column (the FP32 rounding of each
                    # column's term), so near-zero entries are held to an absolute bound
                    err = np.abs(db[r] - go) - (1e-4 * np.abs(go) + 2e-6 * lv.shape[0])
                    k = int(np.argmax(err))
                    assert err[k] <= 0, (model, rho, r, k, db[r][k], go[k])
                assert drho[r] == pytest.approx(float(tree.branch[: tree.n - 1] @ db[r]), rel=1e-12, abs=1e-12)


def test_rho_gradient_matches_central_difference():
    e = engine("58mammals", "fp64")
    offs, leaves = _data("58mammals", [150, 700], seed=3)
    b = e.batch(offs, leaves)
    h = 1e-5
    for model in (0, 1):
        for rho in (0.5, 1.0, 3.0):
            _, _, drho, st = e.grad(b, model, rho)
            fp = e.lpr(b, model, rho + h)[0]
            fm = e.lpr(b, model, rho - h)[0]
            fd = (fp - fm) / (2 * h)
            assert np.allclose(drho, fd, rtol=1e-6, atol=1e-6), (drho, fd)


def test_gradient_zero_at_mle():
    """At the fitted rho the derivative in rho is close to zero (relative to its scale)."""
    e = engine("29mammals", "fp64")
    offs, leaves = _data("29mammals", [400], seed=8)
    res = e.score_batch(offs, leaves, P.MLE)
    b = e.batch(offs, leaves)
    _, _, d1, _ = e.grad(b, 0, res[0]["rho_c"])
    _, _, d2, _ = e.grad(b, 0, res[0]["rho_c"] * 1.2)
    assert abs(d1[0]) < 0.05 * abs(d2[0])


@pytest.mark.parametrize("prec", ["fp64", "fp32b"])
@pytest.mark.parametrize("name", ["12flies", "100vertebrates"])
def test_recomputed_leaf_partials_identical(name, prec):
    """The adjoint with leaf children's partials recomputed in the outside pass (a third less
    scratch per CTA) gives bit-identical lpr, branch gradients and d / d rho, and reports the
    smaller scratch."""
    ps = synth.load_params(name)
    e = P.Engine(ps.tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision=prec)
    offs, leaves = _data(name, [90, 1, 333, 0, 700], seed=31)
    b = e.batch(offs, leaves)
    stored = e.grad_scratch_bytes()
    ref = [e.grad(b, m, rho) for m in (0, 1) for rho in (0.3, 2.5)]
    e.set_grad_recompute(True)
    assert e.grad_scratch_bytes() < 0.7 * stored
    got = [e.grad(b, m, rho) for m in (0, 1) for rho in (0.3, 2.5)]
    for x, y in zip(ref, got):
        for u, v in zip(x, y):
            assert u.tobytes() == v.tobytes()


@pytest.mark.parametrize("name,prec", [("12flies", "fp32b"), ("12flies", "fp64"), ("58mammals", "fp32c")])
@pytest.mark.parametrize("lengths", [[1], [31, 32, 33], [0, 65, 7]])
def test_gradient_tiles(name, prec, lengths):
    """Regions at the edges of the adjoint's 32-column tiles: the gradient of a region is the sum of
    its columns' gradients taken one by one (FP64 sums of at most 65 terms that carry the same FP32
    values: 1e-12 of the largest entry)."""
    ps = synth.load_params(name)
    rng = np.random.default_rng(4)
    gf = synth.gap_fractions(rng, len(lengths), ps.tree.nl, 0.05, 0.4, 0.2)
    offs, leaves = synth.simulate(ps, np.array(lengths), np.zeros(len(lengths), np.int32), gf, 4)
    e = P.Engine(ps.tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision=prec)
    _, db, dr, st = e.grad(e.batch(offs, leaves), 0, 0.8)
    n = int(offs[-1])
    _, db1, dr1, st1 = e.grad(e.batch(np.arange(n + 1), leaves), 0, 0.8)
    assert (st == 0).all() and (st1 == 0).all()
    for r in range(len(lengths)):
        s = slice(int(offs[r]), int(offs[r + 1]))
        scale = np.abs(db1).max() * max(lengths)
        assert np.abs(db[r] - db1[s].sum(0)).max() <= 1e-12 * scale
        assert abs(dr[r] - dr1[s].sum()) <= 1e-12 * scale * ps.tree.branch[:ps.tree.n - 1].sum()


def _two_inner(n, rng):
    """A tree whose nodes have two internal children wherever they can."""
    labels = iter(range(n))

    def rec(k):
        if k == 1:
            return "s%d:%.6f" % (next(labels), rng.uniform(0.005, 0.4))
        b = 1 if k < 4 else max(2, k // 3)
        return "(%s,%s):%.6f" % (rec(k - b), rec(b), rng.uniform(0.001, 0.2))

    return rec(n).rsplit(":", 1)[0]


@pytest.mark.parametrize("prec", ["fp64", "fp32b"])
@pytest.mark.parametrize("nl", [4, 7, 40])
def test_gradient_two_internal_children(prec, nl):
    """Both sides of a node compute a beta, whose exponents start from that side's own: those of the other
    side or of another column would move entries by powers of two.  64 columns, one by one and together.
    Tolerances: FP64 as above; FP32 1e-4 relative plus 1e-5 per column (partials carry up to ~40 x 3
    roundings of 6e-8, against terms of at most the largest |Q_aa| of about 2)."""
    rng = np.random.default_rng(nl)
    tree = P.Tree.from_newick(_two_inner(nl, rng))
    lch, rch = (np.full(tree.n, -1, np.int32) for _ in range(2))
    for i in range(tree.n - 1):
        (lch if lch[tree.parent[i]] < 0 else rch)[tree.parent[i]] = i
    ps = synth.load_params("12flies")
    L = 64
    gf = synth.gap_fractions(rng, 1, nl, 0.05, 0.4, 0.2)
    _, leaves = synth.simulate(synth.ParamSet("t", tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n), np.array([L]),
                               np.ones(1, np.int32), gf, nl)
    mc = O.OModel.from_ecm(ps.S_c, ps.pi_c)
    ot = O.OTree(O.Tree(tree.labels, tree.parent, lch, rch, tree.branch))
    e = P.Engine(tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision=prec)
    for rho in (0.4, 2.0):
        _, db, _, st = e.grad(e.batch(np.arange(L + 1), leaves), 0, rho)
        whole = e.grad(e.batch([0, L], leaves), 0, rho)[1][0]
        assert (st == 0).all()
        ref = np.array([O.grad_branches(mc, ot, rho, H.u8_to_oracle(leaves[c:c + 1]))[1] for c in range(L)])
        for got, want, cols in ((db, ref, 1), (whole, ref.sum(0), L)):
            tol = 1e-7 * np.abs(want) + 1e-8 * cols if prec == "fp64" else 1e-4 * np.abs(want) + 1e-5 * cols
            assert (np.abs(got - want) <= tol).all(), (rho, cols, np.abs(got - want).max())


def test_gradient_memory():
    """The sums that the adjoint keeps for a call: one row of doubles per branch and tile of 32 columns
    (22 MB here; with the work list and the allocator's granularity 48 MiB at most), and the same gradient as the region's copies alone
    give (FP64 sums of n terms: 1e-12)."""
    import torch

    e = engine("12flies", "fp32b")
    offs, leaves = _data("12flies", [4000], seed=6)
    one, short = e.batch(offs, leaves), e.batch([0, 40], leaves[:40])
    n = 1000
    b = e.batch([0, 4000 * n], np.tile(leaves, (n, 1)))
    _, g1, _, _ = e.grad(one, 0, 0.9)
    e.grad(short, 0, 0.9)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    _, g, _, st = e.grad(b, 0, 0.9)
    assert (st == 0).all()
    assert free - torch.cuda.mem_get_info()[0] <= 48 << 20
    assert np.abs(g[0] - n * g1[0]).max() <= 1e-12 * n * np.abs(g1).max()
