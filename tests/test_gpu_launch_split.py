"""Values do not depend on how a launch is split over the GPU: a region alone, in a short list
and in a list long enough for the unsplit forms gives the same bits (every split keeps the
arithmetic of each matrix and column, so the tolerance is zero)."""
import numpy as np
import pytest

import phylocsf_gb300 as P
from phylocsf_gb300 import synth

pytestmark = pytest.mark.gpu


def _regions(name, lengths, seed=5):
    ps = synth.load_params(name)
    rng = np.random.default_rng(seed)
    gf = synth.gap_fractions(rng, len(lengths), ps.tree.nl, 0.05, 0.4, 0.2)
    offs, leaves = synth.simulate(ps, np.asarray(lengths), (np.arange(len(lengths)) % 2).astype(np.int32), gf, seed)
    return ps, offs, leaves


# 12 leaves: 22 branches = 11 pairs, a multiple of neither the pairs nor the branches of a CTA;
# 2,000 P sets are past the unsplit bounds, 1 / 28 / 300 on both sides of the split ones
@pytest.mark.parametrize("prec", ["tf32x3_direct", "fp32b", "fp64"])
@pytest.mark.parametrize("name,counts", [("12flies", (1, 28, 300, 2000)), ("29mammals", (1, 33))])
def test_p_sets_split_over_ctas(name, counts, prec):
    ps, offs, leaves = _regions(name, [33])
    eng = P.Engine(ps.tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision=prec)
    rho = np.exp(np.random.default_rng(1).uniform(np.log(0.02), np.log(9.0), size=max(counts)))
    got = {}
    for n in counts:
        if prec == "fp64" and n > 300:
            continue
        b = eng.batch(np.arange(n + 1) * 33, np.tile(leaves, (n, 1)))
        got[n] = eng.lpr(b, 1, rho[:n])
        assert (got[n][2] == 0).all()
    for n, (lpr, elpr, _) in got.items():
        big = got[max(got)]
        assert np.array_equal(lpr, big[0][:n]) and np.array_equal(elpr, big[1][:n]), n


# eigensolver clusters of 16, 8, 4, 2 and 1 CTAs per matrix (1 / 10 / 20 / 50 / 90 rate matrices)
@pytest.mark.parametrize("prec", ["fp64", "fp32b"])
def test_rate_matrices_split_over_clusters(prec):
    ps, offs, leaves = _regions("12flies", [41])
    eng = P.Engine.for_tree(ps.tree, precision=prec)
    rng = np.random.default_rng(2)
    kappa, omega, rho = rng.uniform(1.2, 6, 90), rng.uniform(0.05, 2, 90), rng.uniform(0.3, 3, 90)
    got = {}
    for n in (1, 10, 20, 50, 90):
        b = eng.batch(np.arange(n + 1) * 41, np.tile(leaves, (n, 1)))
        got[n] = eng.omega_grad(b, kappa[:n], omega[:n], rho[:n])
        assert (got[n]["status"] == 0).all()
    for n in got:
        for k in ("lpr", "d_branch", "d_rho", "d_kappa", "d_omega"):
            assert np.array_equal(got[n][k], got[90][k][:n]), (n, k)


# one region in one part (a call of many tiles) and split into parts of one tile each (alone):
# counts and lpr differ by the FP64 rounding of their sums alone (a few hundred terms), node
# posteriors not at all
@pytest.mark.parametrize("prec", ["fp32b", "fp64"])
def test_outside_parts(prec):
    ps, offs, leaves = _regions("12flies", [32 * 9 + 5])
    eng = P.Engine(ps.tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision=prec)
    n = 120 if prec == "fp32b" else 3
    L = int(offs[-1])
    one = eng.batch(offs, leaves)
    many = eng.batch(np.arange(n + 2) * L, np.tile(leaves, (n + 1, 1)))
    empty = eng.batch([0, 0, L], leaves)
    c1, l1, st = eng.branch_counts(one, 0, 0.7)
    assert (st == 0).all()
    for b in (many, empty):
        c, l, st = eng.branch_counts(b, 0, 0.7)
        assert (st == 0).all()
        if b is empty:
            assert (c[0] == 0).all() and l[0] == 0
            c, l = c[1:], l[1:]
        assert np.abs(c - c1).max() <= 1e-12 * np.abs(c1).max() and np.abs(l - l1).max() <= 1e-12 * np.abs(l1).max()
    p1, _ = eng.node_posteriors(one, 0, 0.7, [0, ps.tree.nl, ps.tree.n - 1])
    pm, _ = eng.node_posteriors(many, 0, 0.7, [0, ps.tree.nl, ps.tree.n - 1])
    assert np.array_equal(p1, pm[:, :L]) and np.array_equal(p1, pm[:, -L:])


# pruning tiles of 8 columns (a region alone) and of 32 or 64 (in a long launch): the same bits
@pytest.mark.parametrize("name,prec", [("12flies", "fp32b"), ("12flies", "fp32c"), ("12flies", "fp64"), ("120mammals", "fp32b")])
def test_small_pruning_tiles(name, prec):
    lengths = [1, 7, 8, 9, 31, 32, 33, 63, 64, 65, 0, 128, 200]
    ps, offs, leaves = _regions(name, lengths)
    eng = P.Engine(ps.tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision=prec)
    n, L = len(lengths), int(offs[-1])
    reps = 40                                              # 25,600 columns: past the small tiles (FP64: 19,456)
    big = eng.batch(np.concatenate([[0]] + [offs[1:] + k * L for k in range(reps)]), np.tile(leaves, (reps, 1)))
    few = eng.batch(offs, leaves)
    for rho in (0.3, 2.0):
        lpr, elpr, st = eng.lpr(big, 1, rho)
        one = eng.lpr(few, 1, rho)
        assert (st == 0).all()
        assert np.array_equal(one[0], lpr[:n]) and np.array_equal(one[1], elpr[:n])
        assert np.array_equal(one[0], lpr[-n:])


# the eigensolver's rotations come from corrected approximations of quotients and roots: an
# eigensystem (branch lengths put P(t) at both ends of its range) against numpy's in FP64.  The sums
# behind P(t) have 64 terms of at most 1 in size with a few ulp each: 1e-13
def test_eigensystem_against_numpy():
    for name in ("12flies", "29mammals"):
        ps = synth.load_params(name)
        eng = P.Engine(ps.tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision="fp64")
        for m, (S, pi) in enumerate(((ps.S_c, ps.pi_c), (ps.S_n, ps.pi_n))):
            U, lam = eng.eigensystem(m)
            Q = synth.q_matrix(S, pi)
            A = np.sqrt(pi)[:, None] * Q / np.sqrt(pi)[None, :]
            A = 0.5 * (A + A.T)
            assert np.abs((U * lam) @ U.T - A).max() <= 1e-13 * np.abs(A).max() * 64
            assert np.abs(U.T @ U - np.eye(64)).max() <= 1e-13
            assert np.abs(np.sort(lam) - np.linalg.eigvalsh(A)).max() <= 1e-13 * np.abs(lam).max() * 64


# the sums of a short launch's columns are formed 1,024 at a time: lengths at that edge, alone (small
# tiles) and in a batch long enough for the long launches' tiles (64 or 32 columns)
@pytest.mark.parametrize("name,prec", [("12flies", "fp32b"), ("12flies", "fp64"), ("120mammals", "fp32b")])
@pytest.mark.parametrize("length", [1023, 1024, 1025, 1057, 2049])
def test_sums_of_small_tiles(name, prec, length):
    ps, offs, leaves = _regions(name, [length])
    eng = P.Engine(ps.tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision=prec)
    eng.set_exact_threshold(1 << 60)                     # the SIMT kernel for every length
    one = eng.lpr(eng.batch(offs, leaves), 0, 1.3)
    n = 40
    many = eng.lpr(eng.batch(np.arange(n + 1) * length, np.tile(leaves, (n, 1))), 0, 1.3)
    assert (one[2] == 0).all() and (many[2] == 0).all()
    assert np.array_equal(np.repeat(one[0], n), many[0]) and np.array_equal(np.repeat(one[1], n), many[1])
