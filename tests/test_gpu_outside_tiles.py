"""Expected counts, their log-likelihoods and node posteriors depend on the region alone: the same bits
whatever else the call holds and wherever its launches end."""
import numpy as np
import pytest

import phylocsf_gb300 as P
from phylocsf_gb300 import synth

pytestmark = pytest.mark.gpu


def _region(name, length, seed=5):
    ps = synth.load_params(name)
    gf = synth.gap_fractions(np.random.default_rng(seed), 1, ps.tree.nl, 0.05, 0.4, 0.2)
    _, leaves = synth.simulate(ps, np.array([length]), np.zeros(1, np.int32), gf, seed)
    return ps, leaves


# copies of one region of 10 or 96 tiles (32 columns): alone; a few; enough for several waves of CTAs;
# and past the tiles of one launch (at most 2 GiB of their counts: 5,957 tiles of 12 leaves in FP32, 2,978
# in FP64), so that a launch ends inside a copy
@pytest.mark.parametrize("prec,length,copies", [("fp32b", 32 * 9 + 5, (1, 5, 121, 500)), ("fp32b", 3050, (1, 65)),
                                                ("fp64", 32 * 9 + 5, (1, 4, 40)), ("fp64", 3050, (1, 33))])
def test_same_bits_in_any_call(prec, length, copies):
    ps, leaves = _region("12flies", length)
    eng = P.Engine(ps.tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision=prec)
    nodes = [0, ps.tree.nl, ps.tree.n - 1]
    one = None
    for n in copies:
        # empty regions at both ends and in the middle
        offs = np.concatenate([[0, 0], np.arange(1, n + 1) * length, [n * length]])
        offs = np.insert(offs, 2, length if n > 1 else 0)
        b = eng.batch(offs, np.tile(leaves, (n, 1)))
        full = np.flatnonzero(np.diff(offs))
        counts, lpr, st = eng.branch_counts(b, 0, 0.7)
        assert (st == 0).all() and len(full) == n
        for r in np.flatnonzero(np.diff(offs) == 0):
            assert not counts[r].any() and lpr[r] == 0
        if one is None:
            one = counts[full[0]], lpr[full[0]]
            # every branch's counts add up to the columns: FP64 sums of terms that carry FP32 rounding
            tol = 1e-9 if prec == "fp64" else 2e-5
            assert np.abs(one[0].sum((1, 2)) - length).max() <= tol * length
        for r in full:
            assert np.array_equal(counts[r], one[0]) and lpr[r] == one[1], (n, r)
        if n <= 5:
            post, _ = eng.node_posteriors(b, 0, 0.7, nodes)
            alone, _ = eng.node_posteriors(eng.batch([0, length], leaves), 0, 0.7, nodes)
            assert np.array_equal(post, np.tile(alone, (1, n, 1)))
    eng.close()


@pytest.mark.parametrize("name,prec,length", [("120mammals", "fp32b", 15000), ("58mammals", "fp64", 20000)])
def test_workspace_bound(name, prec, length):
    """One long region on a large tree: P(t) and the counts of one region, and for CTAs and tiles 2 GiB at
    most (64 MiB beside them for the small arrays and the allocator's granularity)."""
    import threading
    import torch

    ps, leaves = _region(name, length)
    eng = P.Engine(ps.tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision=prec)
    b = eng.batch([0, length], leaves)
    short = eng.batch([0, 40], leaves[:40])
    eng.branch_counts(short, 0, 0.7)
    free = torch.cuda.mem_get_info()[0]
    low, done = [free], threading.Event()

    def watch():
        while not done.is_set():
            low[0] = min(low[0], torch.cuda.mem_get_info()[0])

    t = threading.Thread(target=watch)
    t.start()
    try:
        _, _, st = eng.branch_counts(b, 0, 0.7)
    finally:
        done.set()
        t.join()
    assert (st == 0).all()
    matrices = (ps.tree.n - 1) * 4096 * (8 + (8 if prec == "fp64" else 4))
    assert 0 < free - low[0] <= (2 << 30) + matrices + (64 << 20)
    eng.close()
