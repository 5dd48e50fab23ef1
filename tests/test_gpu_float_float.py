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
