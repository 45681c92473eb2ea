"""Threads that share a model: HMM-banded and truncated calls take no workspace,
so each call's results must be its own."""
import threading

import numpy as np
import pytest

from infernox_b200 import _native as N
from infernox_b200.hb import TrInputs, hb_scan_batch, tr_qdb_scan_batch, tr_scan_hb_batch
from infernox_b200.scan import Scanner

from hb_helpers import ragged_bands, rect_bands, tr_tables, tr_valid
from helpers import frame, models, planted_seq

pytestmark = pytest.mark.gpu


def test_calls_of_several_threads_on_one_model():
    cm, _, l = models("mb3")
    sc = Scanner(l)
    tt = tr_tables(cm, l, 4, True)
    tri = TrInputs(tt["lmesc"], tt["rmesc"], tt["pty"], tt["lpos"], tt["rpos"], tt["clen"], True,
                   tt["ilmesc"], tt["irmesc"], tt["ipty"])
    w = min(l.W, 90)

    def calls(q):
        """Three calls of thread q, of sizes and data of its own."""
        seq = frame(planted_seq(cm, 300 + 90 * q, 0.5, 2, seed=q, degenerate=0.01))
        env = [(0, 1 + 7 * k, w - k + 7 * k, -5.0, -20.0,
                (rect_bands if k % 2 else ragged_bands)(l, 1 + 7 * k, w - k + 7 * k, k)) for k in range(3 + 4 * q)]
        valid = [e + (tr_valid(l.M, k, 4, True),) for k, e in enumerate(env)]
        wins = np.array([(0, 1 + 5 * k, 60 + 30 * q + 5 * k) for k in range(2 + 3 * q)], N.WINDOW_DTYPE)
        return (lambda: hb_scan_batch(sc, N.INSIDE_F32, True, True, seq, env),
                lambda: tr_scan_hb_batch(sc, N.CYK_F32, tri, 4, True, seq, valid),
                lambda: tr_qdb_scan_batch(sc, N.CYK_F32 if q % 2 else N.INSIDE_I32, N.NOQDB, tri, 4, True, seq, wins,
                                          -12.0))

    work = [calls(q) for q in range(4)]
    want = [[c() for c in cs] for cs in work]
    wrong = []

    def run(q):
        try:
            for r in range(6):
                for k, c in enumerate(work[q]):
                    if c() != want[q][k]:
                        wrong.append((q, r, k))
        except Exception as e:  # noqa: BLE001 -- reported by the assertion
            wrong.append((q, repr(e)))

    ts = [threading.Thread(target=run, args=(q,)) for q in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not wrong
    sc.close()
