"""Distinct engines on distinct threads (the header allows it): their launches of one kernel differ in
shared memory, by tree and by the length of a launch, and must not disturb one another.  Values are those
of the engine alone, bit for bit."""
import threading

import numpy as np
import pytest

import phylocsf_gb300 as P
from phylocsf_gb300 import synth

pytestmark = pytest.mark.gpu


def _work(name, prec, regions, strategy):
    ps = synth.load_params(name)
    rng = np.random.default_rng(2)
    gf = synth.gap_fractions(rng, regions, ps.tree.nl, 0.05, 0.4, 0.2)
    offs, leaves = synth.simulate(ps, np.full(regions, 30), (np.arange(regions) % 2).astype(np.int32), gf, 2)
    e = P.Engine(ps.tree, ps.S_c, ps.pi_c, ps.S_n, ps.pi_n, precision=prec)
    b = e.batch(offs, leaves)
    rho = np.linspace(0.5, 2.0, regions)

    def once():
        l, el, st = e.lpr(b, 1, rho)
        return l.tobytes() + el.tobytes() + st.tobytes() + e.score_batch(offs, leaves, strategy).tobytes()

    return once


@pytest.mark.parametrize("prec", ["fp32b", "tf32x3b"])
def test_engines_on_threads(prec):
    # one to a few P sets a launch, and enough for two branches per CTA of the P(t) kernel
    jobs = [_work("12flies", prec, 1, P.FIXED), _work("120mammals", prec, 2, P.FIXED),
            _work("29mammals", prec, 40, P.MLE), _work("58mammals", prec, 1, P.MLE)]
    want = [j() for j in jobs]
    failures = []

    def loop(k):
        try:
            for _ in range(150):
                if jobs[k]() != want[k]:
                    failures.append((k, "values"))
                    return
        except Exception as x:      # noqa: BLE001
            failures.append((k, str(x)))

    threads = [threading.Thread(target=loop, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
