"""Per-node rescaling where some columns of a warp have no normal maximum: on zero-length branches a
column whose leaves disagree has likelihood 0 (every partial zero), one whose leaves agree the prior
of its state.  A region with both has lpr = -inf and, as its zero columns add nothing to elpr, the
elpr of the others.

Tolerance on elpr, against the FP64 engine: 1e-6 relative for FP32 (a few roundings of 6e-8 a
column), the documented 2e-6 and 1e-3 for split and single TF32."""
import numpy as np
import pytest

import phylocsf_gb300 as P
from phylocsf_gb300 import synth

pytestmark = pytest.mark.gpu


# one region: the small tiles of short launches; 700: the long launches' tiles
@pytest.mark.parametrize("precision,tol", [("fp32b", 1e-6), ("fp32", 1e-6), ("tf32x3_direct", 2e-6), ("tf32_direct", 1e-3)])
@pytest.mark.parametrize("nreg", [1, 700])
def test_zero_columns_beside_others(precision, tol, nreg):
    tree = P.Tree.from_newick("(((a:0,b:0):0,(c:0,d:0):0):0,e:0)")
    ps = synth.load_params("12flies")
    rng = np.random.default_rng(3)
    n = 100
    leaves = np.repeat(rng.integers(0, 64, n * nreg).astype(np.uint8)[:, None], 5, 1)
    zero = rng.random(n * nreg) < 0.3
    zero[::n] = True                                                  # every region has one
    leaf = rng.integers(0, 5, zero.sum())
    leaves[np.flatnonzero(zero), leaf] ^= 1                           # one leaf disagrees
    offs = np.arange(nreg + 1, dtype=np.int64) * n
    out = []
    for prec in (precision, "fp64"):
        e = P.Engine(tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision=prec)
        l, el, st = e.lpr(e.batch(offs, leaves), 0, 1.0)
        assert (st == 0).all() and np.all(np.isneginf(l))
        out.append(el)
    assert np.all(np.isfinite(out[1])) and np.all(out[1] < 0)
    assert np.all(np.abs(out[0] - out[1]) <= tol * np.abs(out[1])), np.max(np.abs(out[0] / out[1] - 1))
