"""The tensor-core search kernel on trees and lengths at the edges of its tiles, operands and stack,
against the FP64 engine at a given rho, for P(t) formed either way and for both grid shapes.

Tolerance: the documented bound of the split TF32 kernel (2e-6 of |lpr|) plus 1e-5 for an lpr near
zero (a column whose leaves are all missing: |log z| up to ~1e-7 per node)."""
import numpy as np
import pytest

import phylocsf_gb300 as P
from phylocsf_gb300 import engine as E
from phylocsf_gb300 import synth
from tests.test_gpu_float_float import _balanced, _caterpillar

pytestmark = pytest.mark.gpu


# 2 leaves: no contraction; 3: one; caterpillars: nothing waits; balanced: the stack past its top entry
@pytest.mark.parametrize("shape,nl", [("balanced", 2), ("balanced", 3), ("balanced", 64), ("balanced", 90),
                                      ("caterpillar", 9), ("caterpillar", 130)])
@pytest.mark.parametrize("pt64", [False, True])
def test_trees(shape, nl, pt64, monkeypatch):
    rng = np.random.default_rng(nl)
    tree = P.Tree.from_newick((_balanced if shape == "balanced" else _caterpillar)(nl, rng))
    ps = synth.load_params("12flies")
    par = synth.ParamSet("t", tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n)
    lengths = np.array([1, 127, 128, 129, 0, 300])
    gf = synth.gap_fractions(rng, len(lengths), nl, 0.0, 0.4, 0.2)
    offs, leaves = synth.simulate(par, lengths, (np.arange(len(lengths)) % 2).astype(np.int32), gf, 7)
    leaves[offs[1]:offs[1] + 5] = 64                      # columns with nothing known
    monkeypatch.setitem(E.PREC, "direct_pt64", E.PREC["tf32x3_direct"] | (1 << 19))      # PCSF_PT_FP64
    e = P.Engine(tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision="direct_pt64" if pt64 else "tf32x3_direct")
    f = P.Engine(tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision="fp64")
    b, b64 = e.batch(offs, leaves), f.batch(offs, leaves)
    for rho in (0.1, 1.0, 3.3):
        e.set_tc_shape(0)
        l, el, st = e.lpr(b, 0, rho)
        l64, el64, st64 = f.lpr(b64, 0, rho)
        assert (st == 0).all() and (st64 == 0).all()
        assert np.all(np.abs(l - l64) <= 2e-6 * np.abs(l64) + 1e-5), (rho, l - l64)
        e.set_tc_shape(1)
        l1, el1, _ = e.lpr(b, 0, rho)
        assert l1.tobytes() == l.tobytes() and el1.tobytes() == el.tobytes()
