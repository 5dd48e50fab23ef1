"""pcsf_score_batch (regions in host buffers, one call): invalid leaf codes are refused early, with
pcsf_batch_create's message and before anything else is reported or written, and the leaf buffer that
the engine keeps does not show in the results."""
import ctypes

import numpy as np
import pytest

import phylocsf_gb300 as P
from phylocsf_gb300 import engine as E
from phylocsf_gb300 import synth

pytestmark = pytest.mark.gpu


def _engine(name="12flies", prec="tf32x3b"):
    ps = synth.load_params(name)
    return ps, P.Engine(ps.tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision=prec)


def _regions(ps, lengths, seed=3):
    rng = np.random.default_rng(seed)
    gf = synth.gap_fractions(rng, len(lengths), ps.tree.nl, 0.05, 0.4, 0.2)
    return synth.simulate(ps, np.asarray(lengths), (np.arange(len(lengths)) % 2).astype(np.int32), gf, seed)


def _call(e, offs, leaves, strategy, out):
    """The C call itself: (status, message)."""
    offs, leaves = np.ascontiguousarray(offs, np.int64), np.ascontiguousarray(leaves, np.uint8)
    rc = e.lib.pcsf_score_batch(e.handle, len(offs) - 1, E._p(offs, ctypes.c_int64), E._p(leaves, ctypes.c_uint8),
                                strategy, out.ctypes.data_as(ctypes.POINTER(E.Result)))
    return rc, e.lib.pcsf_last_error(e.handle).decode()


# 60,000 bytes of leaves: refused with the first evaluation; 2,400,000: before any
@pytest.mark.parametrize("prec", ["tf32x3b", "fp64", "bf16x3b"])
@pytest.mark.parametrize("columns,rounds", [(5000, 1), (200000, 0)])
@pytest.mark.parametrize("code", [65, 255])
def test_invalid_code(prec, columns, rounds, code):
    if prec == "fp64" and rounds == 0:
        columns = 100000
    ps, e = _engine(prec=prec)
    offs, leaves = _regions(ps, [columns // 10] * 10)
    good = e.score_batch(offs[:3], leaves[:offs[2]], P.MLE).tobytes()
    bad = leaves.copy()
    bad[columns - 7, 5] = code
    with pytest.raises(P.EngineError) as refused:
        e.batch(offs, bad)
    for strategy in (P.MLE, P.FIXED, 17):                   # a wrong strategy is not what is reported
        out = np.full(10 * E.RESULT_DTYPE.itemsize, 0xA5, np.uint8)
        e.reset_stats()
        rc, msg = _call(e, offs, bad, strategy, out)
        assert rc == refused.value.status and "%s (status %d)" % (msg, rc) == str(refused.value)
        assert (out == 0xA5).all()
        assert e.stats()["rounds"] <= rounds
    rc, msg = _call(e, offs, leaves, 17, np.zeros(10, E.RESULT_DTYPE))
    assert rc != 0 and "strategy" in msg
    assert e.score_batch(offs[:3], leaves[:offs[2]], P.MLE).tobytes() == good
    e.close()


def test_kept_leaf_buffer():
    """Growing and shrinking calls, empty ones, one past the kept size (64 MiB) and failed ones between
    them: the values of a batch of the caller's own."""
    ps, e = _engine(prec="fp32b")
    big = 6_000_000                                         # 72 MB of leaves
    offs, leaves = _regions(ps, [300, 41, 0, 1, 900])
    L = int(offs[-1])
    for n in (5, 1, 3, big, 2, 0, 5):
        if n == big:
            k = big // L + 1
            o, lv = np.arange(k + 1) * L, np.tile(leaves, (k, 1))
        else:
            o, lv = offs[:n + 1], leaves[:offs[n]]
        got = e.score_batch(o, lv, P.FIXED)
        assert (got["status"] == 0).all()
        assert got.tobytes() == e.score(e.batch(o, lv), P.FIXED).tobytes()
        wrong = lv.copy()
        if len(wrong):
            wrong[-1, -1] = 99
            assert _call(e, o, wrong, P.FIXED, np.zeros(len(o) - 1, E.RESULT_DTYPE))[0] != 0
        assert _call(e, np.array([0, 2, 1]), leaves, P.FIXED, np.zeros(2, E.RESULT_DTYPE))[0] != 0
    e.close()
