"""The two kernels of the truncated QDB scan against the oracle: the column
wavefront, asked for and where the model leaves no other, over passes, band
sets, semirings and window lengths; which kernel ran; and the wavefront after
a call of its own whose wait ran out."""
import dataclasses

import numpy as np
import pytest

import oracle
from infernox_b200 import _native as N
from infernox_b200.hb import (TRQ_AUTO, TRQ_DIAG, TRQ_WAVEFRONT, TrInputs, ref_itr_inside_scan, ref_tr_cyk_scan,
                              tr_qdb_kernel, tr_qdb_scan_batch, tr_qdb_set_kernel)
from infernox_b200.scan import Scanner

from hb_helpers import tr_tables, truncated_window
from helpers import frame, models, planted_seq

pytestmark = pytest.mark.gpu

SCANS = ((False, ref_tr_cyk_scan), (True, ref_itr_inside_scan))


def bits(x):
    return np.float32(x).tobytes()


def flat(r):
    return [(i, j, bits(s), bits(b), m, v) for i, j, s, b, m, v in r[0]], bits(r[1]), r[2], bits(r[3])


def tri_of(tt, loc):
    return TrInputs(tt["lmesc"], tt["rmesc"], tt["pty"], tt["lpos"], tt["rpos"], tt["clen"], loc,
                    tt["ilmesc"], tt["irmesc"], tt["ipty"])


def check(cfg, sc, loc, f, i0, j0, qdb, pass_idx, cutoff, kernel, scans=SCANS):
    tt = tr_tables(cfg_cm(cfg), cfg, pass_idx, loc)
    for inside, fn in scans:
        ro = oracle.trq_scan(cfg, inside, tt, f, i0, j0, cutoff, True, qdb, pass_idx, loc)
        go = fn(sc, tri_of(tt, loc), f, i0, j0, cutoff, qdb, True, pass_idx)
        assert tr_qdb_kernel(sc) == kernel
        assert flat(go) == flat(ro), (inside, qdb, pass_idx, i0, j0)


def cfg_cm(cfg):
    return models(cfg.name)[0]


@pytest.mark.parametrize("name,loc,pass_idx,qdb", [("trna", True, 4, N.NOQDB), ("trna", False, 2, N.QDB1),
                                                   ("small0", True, 5, N.QDB2), ("small2", True, 3, N.QDB1),
                                                   ("mb3", True, 4, N.QDB2), ("mb3", False, 4, N.NOQDB)])
def test_wavefront_matches_oracle(name, loc, pass_idx, qdb):
    cm, g, l = models(name)
    cfg = l if loc else g
    sc = Scanner(cfg)
    tr_qdb_set_kernel(sc, TRQ_WAVEFRONT)
    f, i0, j0 = truncated_window(cm, cfg, pass_idx, 77)
    check(cfg, sc, loc, f, i0, j0, qdb, pass_idx, -10.0, TRQ_WAVEFRONT)
    f = frame(planted_seq(cm, 400, 0.45, 2, seed=5, degenerate=0.05))
    for i0, j0 in ((1, cfg.W), (50, 50), (50, 51), (9, 9 + cfg.W // 2), (20, 370)):
        check(cfg, sc, loc, f, i0, j0, qdb, pass_idx, -20.0, TRQ_WAVEFRONT)
    tr_qdb_set_kernel(sc, TRQ_AUTO)
    check(cfg, sc, loc, f, 20, 370, qdb, pass_idx, -20.0, TRQ_DIAG)
    sc.close()


def test_wavefront_batch_matches_oracle():
    cm, _, l = models("mb3")
    sc = Scanner(l)
    tr_qdb_set_kernel(sc, TRQ_WAVEFRONT)
    tt = tr_tables(cm, l, 4, True)
    f = frame(planted_seq(cm, 900, 0.45, 4, seed=6, degenerate=0.02))
    wins = [(0, 1, 60), (0, 100, 99), (0, 200, 420), (0, 500, 500), (0, 640, 900)]
    for semiring, inside in ((N.CYK_F32, False), (N.INSIDE_I32, True)):
        res = tr_qdb_scan_batch(sc, semiring, N.QDB1, tri_of(tt, True), 4, True, f, np.array(wins, N.WINDOW_DTYPE),
                                -12.0)
        assert tr_qdb_kernel(sc) == TRQ_WAVEFRONT
        for r, (_, i0, j0) in zip(res, wins):
            if j0 >= i0:
                assert flat(r) == flat(oracle.trq_scan(l, inside, tt, f, i0, j0, -12.0, True, N.QDB1, 4, True))
    sc.close()


# models that the diagonal kernel does not take: a score of -0 (CYK), an
# integer score whose sums pass a float's whole numbers (Inside)
@pytest.mark.parametrize("inside", [False, True])
@pytest.mark.parametrize("qdb", [N.NOQDB, N.QDB2])
def test_auto_takes_the_wavefront_for_other_scores(inside, qdb):
    cm, _, l = models("trna")
    if inside:
        esc = l.ioesc.copy()
        esc[np.nonzero(l.sttype == 2)[0][3], 1] = 200000
        cfg = dataclasses.replace(l, ioesc=esc, _struct=None)
    else:
        esc = l.oesc.copy()
        esc[np.nonzero(l.sttype == 2)[0][3], 1] = -0.0
        cfg = dataclasses.replace(l, oesc=esc, _struct=None)
    sc = Scanner(cfg)
    f = frame(planted_seq(cm, 300, 0.45, 2, seed=8, degenerate=0.02))
    for i0, j0 in ((1, 80), (40, 290)):
        check(cfg, sc, True, f, i0, j0, qdb, 4, -10.0, TRQ_WAVEFRONT, [SCANS[inside]])
    sc.close()


def test_wavefront_after_a_timeout():
    cm, _, l = models("small2")
    sc = Scanner(l)
    tr_qdb_set_kernel(sc, TRQ_WAVEFRONT)
    f, i0, j0 = truncated_window(cm, l, 4, 77, max_len=l.W + 10, flank=60)
    tt = tr_tables(cm, l, 4, True)
    N.check(N.lib().cmgpu_tr_qdb_inject_stall(sc._model, 3))
    with pytest.raises(N.CmgpuError, match="timed out") as ei:
        ref_tr_cyk_scan(sc, tri_of(tt, True), f, i0, j0, -5.0, N.NOQDB, True, 4)
    assert ei.value.rc == N.CMGPU_ETIMEOUT and tr_qdb_kernel(sc) == TRQ_WAVEFRONT
    check(l, sc, True, f, i0, j0, N.NOQDB, 4, -5.0, TRQ_WAVEFRONT)
    sc.close()


def test_kernel_choice_is_checked():
    sc = Scanner(models("small0")[2])
    for bad in (TRQ_DIAG, 3, -1):
        with pytest.raises(N.CmgpuError):
            tr_qdb_set_kernel(sc, bad)
    assert tr_qdb_kernel(sc) == 0
    sc.close()
