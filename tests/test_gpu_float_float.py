"""The tensor-core float-float kernel on trees and lengths at the edges of its tiles, operands and
stack, against the FP64 engine at a given rho.

Tolerance: a column's partials carry ~2^-48 relative per operation; with at most ~120 nodes and
64 terms each that is below 1e-12 of |lpr| (+1e-12 for an lpr near zero), the bound the kernel is
documented with."""
import numpy as np
import pytest

import phylocsf_gb300 as P
from phylocsf_gb300 import synth

pytestmark = pytest.mark.gpu


def _balanced(n, rng):
    labels = iter(range(n))

    def rec(k):
        if k == 1:
            return "s%d:%.6f" % (next(labels), rng.uniform(0.005, 0.4))
        return "(%s,%s):%.6f" % (rec(k // 2), rec(k - k // 2), rng.uniform(0.0005, 0.2))

    return rec(n).rsplit(":", 1)[0]


def _caterpillar(n, rng):
    t = "(s0:%.6f,s1:%.6f)" % (rng.uniform(0.005, 0.3), rng.uniform(0.005, 0.3))
    for k in range(2, n):
        leaf, inner = "s%d:%.6f" % (k, rng.uniform(0.005, 0.3)), "%s:%.6f" % (t, rng.uniform(0.0, 0.05))
        t = "(%s,%s)" % ((inner, leaf) if k % 2 else (leaf, inner))
    return t


# 2 leaves: no contraction; 90: the largest balanced tree that the FP64 engine takes; caterpillars: nothing ever waits; balanced: the deepest stack
@pytest.mark.parametrize("shape,nl", [("balanced", 2), ("balanced", 3), ("balanced", 64), ("balanced", 90),
                                      ("caterpillar", 9), ("caterpillar", 130)])
def test_trees(shape, nl):
    rng = np.random.default_rng(nl)
    tree = P.Tree.from_newick((_balanced if shape == "balanced" else _caterpillar)(nl, rng))
    ps = synth.load_params("12flies")
    par = synth.ParamSet("t", tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n)
    lengths = np.array([1, 127, 128, 129, 0, 300])
    gf = synth.gap_fractions(rng, len(lengths), nl, 0.0, 0.4, 0.2)
    offs, leaves = synth.simulate(par, lengths, (np.arange(len(lengths)) % 2).astype(np.int32), gf, 7)
    leaves[offs[1]:offs[1] + 5] = 64                      # columns with nothing known
    e = P.Engine(tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision="fp32b")
    f = P.Engine(tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision="fp64")
    assert e.exact_available
    e.set_exact_threshold(0)
    b, b64 = e.batch(offs, leaves), f.batch(offs, leaves)
    for rho in (0.02, 1.0, 9.0):
        l, el, st = e.lpr(b, 0, rho)
        l64, el64, st64 = f.lpr(b64, 0, rho)
        assert (st == 0).all() and (st64 == 0).all()
        assert np.all(np.abs(l - l64) <= 1e-12 * np.abs(l64) + 1e-12), (rho, l - l64)
        assert np.all(np.abs(el - el64) <= 1e-12 * np.abs(el64) + 1e-12), (rho, el - el64)


# leaf states beside the operands in shared memory (362), and read where they lie (363, 450)
@pytest.mark.parametrize("nl", [362, 363, 450])
def test_large_trees(nl):
    rng = np.random.default_rng(nl)
    tree = P.Tree.from_newick(_caterpillar(nl, rng))
    ps = synth.load_params("12flies")
    par = synth.ParamSet("t", tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n)
    lengths = np.array([1, 127, 0, 300])
    gf = synth.gap_fractions(rng, len(lengths), nl, 0.0, 0.4, 0.2)
    offs, leaves = synth.simulate(par, lengths, np.zeros(len(lengths), np.int32), gf, 7)
    e = P.Engine(tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision="fp32b")
    f = P.Engine(tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision="fp64")
    assert e.exact_available
    e.set_exact_threshold(0)
    l, el, st = e.lpr(e.batch(offs, leaves), 0, 1.0)
    l64, el64, st64 = f.lpr(f.batch(offs, leaves), 0, 1.0)
    assert (st == 0).all() and (st64 == 0).all()
    assert np.all(np.abs(l - l64) <= 1e-12 * np.abs(l64) + 1e-12)
    assert np.all(np.abs(el - el64) <= 1e-12 * np.abs(el64) + 1e-12)


def _error_bound(tree, prior, Pt, leaves):
    """Per column, to first order, the most that the kernel's lpr may differ from exact arithmetic on the
    same P(t).  With r the largest off-diagonal entry of a row of P and m the largest of a column's
    partials: an entry of P is held to 2^-62 r (seven 9-bit digits below a power of two of at most 2 r), a
    partial to 2^-59 m, digit products beyond the eighth group are below 2^-60 r m, everything else is
    float-float (2^-45 of the terms of a sum, of a product).  A 64-bit evaluation adds 66 roundings of
    positive terms a node, twice."""
    nl, n = tree.nl, tree.n
    children = [[] for _ in range(n)]
    for i in range(n - 1):
        children[tree.parent[i]].append(i)
    alpha, err = {}, {}
    for node in range(nl, n):
        v, dv = 1.0, 0.0
        for c in children[node]:
            if c < nl:
                x = Pt[c][:, leaves[:, c]]
                dx = 2.0 ** -48 * x
            else:
                al = alpha[c]
                off = Pt[c] - np.diag(np.diag(Pt[c]))
                r, m = off.max(1)[:, None], al.max(0)[None]
                x = Pt[c] @ al
                dx = (Pt[c] @ err[c] + 2.0 ** -62 * r * al.sum(0) + 2.0 ** -59 * off.sum(1)[:, None] * m +
                      2.0 ** -60 * r * m + 2.0 ** -45 * (al + x))
            v, dv = v * x, dv * x + v * dx + 2.0 ** -45 * v * x
        m = v.max(0)
        alpha[node], err[node] = v / m, dv / m
    return prior @ err[n - 1] / (prior @ alpha[n - 1]) + 132 * (nl - 1) * 2.0 ** -53


# Columns whose two halves of the tree hold codons three substitutions apart, at scales where such a change
# is millions of times rarer than a single one: what the columns weigh is far below the largest entry of
# every row of P and every partial.
@pytest.mark.parametrize("name", ["12flies", "58mammals", "120mammals"])
def test_discordant_columns(name):
    ps = synth.load_params(name)
    tree, rng = ps.tree, np.random.default_rng(11)
    below = [{i} if i < tree.nl else set() for i in range(tree.n)]
    for i in range(tree.n - 1):
        below[tree.parent[i]] |= below[i]
    half = list(below[min(range(tree.nl, tree.n - 1), key=lambda i: abs(len(below[i]) - tree.nl / 2))])
    n = 48
    leaves = np.empty((n, tree.nl), np.uint8)
    for c in range(n):
        x = rng.integers(64)
        leaves[c] = x
        leaves[c, half] = x ^ sum(int(rng.integers(1, 4)) << s for s in (0, 2, 4))
    e = P.Engine(tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision="fp32b")
    f = P.Engine(tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision="fp64")
    e.set_exact_threshold(0)
    offs = np.arange(n + 1)
    b, b64 = e.batch(offs, leaves), f.batch(offs, leaves)
    for model, pi in enumerate((ps.pi_c, ps.pi_n)):
        for rho in (0.01, 0.1, 1.0):
            l, _, st = e.lpr(b, model, rho)
            l64, _, st64 = f.lpr(b64, model, rho)
            assert (st == 0).all() and (st64 == 0).all()
            Pt, _ = f.pt(model, tree.branch[:tree.n - 1] * rho)
            tol = _error_bound(tree, pi / pi.sum(), Pt, leaves) + 2.0 ** -51 * np.abs(l64)
            assert np.all(np.abs(l - l64) <= tol), (rho, np.max(np.abs(l - l64) / tol), np.abs(l - l64).max())
