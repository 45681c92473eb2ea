"""The kernel forms that the sizes of a call choose, where they meet:

* truncated scans of windows of one, two and three column groups, and at the
  borders of a warp and of a group, against the oracle;
* HMM-banded scans with so many envelopes that a CTA shrinks to 128 and then
  to 32 threads, each envelope against the same envelope in a small call
  (whose results other tests hold against the oracle);
* hit lists long enough for the overlap rule to order them piece by piece,
  against the oracle.
"""
import numpy as np
import pytest
import torch

import oracle
from infernox_b200 import _native as N
from infernox_b200 import model, synth
from infernox_b200.hb import (Bands, TrInputs, hb_scan_batch, ref_itr_inside_scan, ref_tr_cyk_scan, tr_scan_hb_batch)
from infernox_b200.scan import CYK_F32, INSIDE_I32, NOQDB, QDB1, QDB2, Scanner

from hb_helpers import as_tuple, ragged_bands, rect_bands, tr_tables, tr_valid, truncated_window
from helpers import frame, models, oracle_cfg, planted_seq

pytestmark = pytest.mark.gpu


def bits(x):
    return np.float32(x).tobytes()


def tri_of(tt, loc):
    return TrInputs(tt["lmesc"], tt["rmesc"], tt["pty"], tt["lpos"], tt["rpos"], tt["clen"], loc,
                    tt["ilmesc"], tt["irmesc"], tt["ipty"])


@pytest.mark.parametrize("n", [31, 32, 33, 255, 256, 257, 513, 700])
@pytest.mark.parametrize("name,loc,qdb", [("small0", True, NOQDB), ("mb3", True, NOQDB), ("mb3", False, QDB2)])
def test_truncated_scan_column_groups(name, loc, qdb, n):
    cm, g, l = models(name)
    cfg = l if loc else g
    sc = Scanner(cfg)
    tt = tr_tables(cm, cfg, 4, loc)
    f = frame(planted_seq(cm, n + 20, 0.45, 2, seed=n, degenerate=0.02) if n >= 100
              else np.random.default_rng(n).integers(0, 4, n + 20).astype(np.uint8))
    for inside, fn in ((False, ref_tr_cyk_scan), (True, ref_itr_inside_scan)):
        for i0 in (1, 9):
            j0 = i0 + n - 1
            ro = oracle.trq_scan(cfg, inside, tt, f, i0, j0, -12.0, True, qdb, 4, loc)
            go = fn(sc, tri_of(tt, loc), f, i0, j0, -12.0, qdb, True, 4)
            assert bits(go[1]) == bits(ro[1]) and go[2] == ro[2] and bits(go[3]) == bits(ro[3])
            assert [(a, b, bits(s), bits(e), m, r) for a, b, s, e, m, r in go[0]] == \
                   [(a, b, bits(s), bits(e), m, r) for a, b, s, e, m, r in ro[0]]


def envelope_counts():
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return [sms, sms + 1, 2 * sms + 1, 10 * sms, 10 * sms + 1]


def same(a, b):
    """Two envelopes' results, hits included, bit for bit."""
    def flat(x):
        if isinstance(x, (list, tuple)):
            return tuple(flat(y) for y in x)
        return bits(x) if isinstance(x, (float, np.floating)) else x
    return flat(a) == flat(b)


@pytest.mark.parametrize("semiring", [N.CYK_F32, N.INSIDE_F32])
@pytest.mark.parametrize("name", ["trna", "mb3"])
def test_hmm_banded_envelope_counts(name, semiring):
    _, _, l = models(name)
    cm = models(name)[0]
    sc = Scanner(l)
    seq = frame(planted_seq(cm, 400, 0.5, 3, seed=8, degenerate=0.01))
    w = min(l.W, 130)
    base = [(0, i0, i0 + w - 1 - q, -1e30, -20.0, (rect_bands if q % 2 else ragged_bands)(l, i0, i0 + w - 1 - q, q))
            for q, i0 in enumerate((1, 40, 97, 160, 200))]
    ref = hb_scan_batch(sc, semiring, True, True, seq, base)
    assert any(len(r[3]) for r in ref)
    for n in envelope_counts():
        got = hb_scan_batch(sc, semiring, True, True, seq, [base[q % 5] for q in range(n)])
        assert all(same(got[q], ref[q % 5]) for q in range(n)), n
    sc.close()


@pytest.mark.parametrize("semiring", [N.CYK_F32, N.INSIDE_F32])
def test_truncated_hmm_banded_envelope_counts(semiring):
    cm, _, l = models("mb3")
    sc = Scanner(l)
    tt = tr_tables(cm, l, 4, True)
    tri = TrInputs(tt["lmesc"], tt["rmesc"], tt["pty"], tt["lpos"], tt["rpos"], tt["clen"], True)
    seq = frame(planted_seq(cm, 400, 0.5, 3, seed=18, degenerate=0.01))
    w = min(l.W, 90)
    base = [(0, i0, i0 + w - 1 - q, -5.0, -20.0, (rect_bands if q % 2 else ragged_bands)(l, i0, i0 + w - 1 - q, q),
             tr_valid(l.M, q, 4, q % 3 != 0)) for q, i0 in enumerate((1, 40, 97, 160, 200))]
    ref = tr_scan_hb_batch(sc, semiring, tri, 4, True, seq, base)
    for n in envelope_counts():
        got = tr_scan_hb_batch(sc, semiring, tri, 4, True, seq, [base[q % 5] for q in range(n)])
        assert all(same(got[q], ref[q % 5]) for q in range(n)), n
    sc.close()


@pytest.mark.parametrize("sr,band", [(CYK_F32, QDB1), (INSIDE_I32, QDB2)])
def test_long_hit_lists_match_oracle(sr, band):
    cm, _, l = models("small0")
    n = 9000
    dsq = frame(planted_seq(cm, n, 0.5, 6, seed=3, degenerate=0.01))
    ref, _, _, _ = oracle.qdb_scan(oracle_cfg("small0", True), sr, band, dsq, 1, n, -60.0, True)
    got = Scanner(l).generic_scan(sr, band, dsq, 1, n, -60.0, True)
    assert [(h[0], h[1], bits(h[2]), bits(h[3])) for h in got] == [(h[0], h[1], bits(h[2]), bits(h[3])) for h in ref]
    assert len(ref) > 0


# Models of three and five nodes with W of 5 and 10 to 12: a group of columns
# takes fewer phases than eight warps, so the launch takes fewer.
@pytest.mark.parametrize("ss", ["..", "....", "(...)"])
@pytest.mark.parametrize("loc", [False, True])
@pytest.mark.parametrize("qdb", [NOQDB, QDB2])
def test_truncated_scan_of_tiny_models(ss, loc, qdb):
    cm = synth.synth_cm(ss, 1, name="tiny", ins_open=0.005, ins_self=0.1)
    cfg = model.configure(cm, local=loc)
    assert cfg.W <= 15
    sc = Scanner(cfg)
    tt = tr_tables(cm, cfg, 4, loc)
    for n in (200, 257, 700, 1100):
        f = frame(planted_seq(cm, n, 0.5, 12, seed=n, degenerate=0.02))
        for inside, fn in ((False, ref_tr_cyk_scan), (True, ref_itr_inside_scan)):
            ro = oracle.trq_scan(cfg, inside, tt, f, 1, n, -6.0, True, qdb, 4, loc)
            go = fn(sc, tri_of(tt, loc), f, 1, n, -6.0, qdb, True, 4)
            assert len(ro[0]) > 0
            assert bits(go[1]) == bits(ro[1]) and go[2] == ro[2] and bits(go[3]) == bits(ro[3])
            assert [(a, b, bits(s), bits(e), m, r) for a, b, s, e, m, r in go[0]] == \
                   [(a, b, bits(s), bits(e), m, r) for a, b, s, e, m, r in ro[0]]
    sc.close()


# One row of 31,000 spans among 70,000 rows of one: 70,000 x 31,000 cell numbers
# of a state do not fit 32 bits.  (200: sixteen numbers a cell and more.)
@pytest.mark.parametrize("truncated", [False, True])
@pytest.mark.parametrize("rows,wide", [(700, 200), (70000, 31000)])
def test_hmm_banded_one_wide_row(rows, wide, truncated):
    cm, _, l = models("small0")
    sc = Scanner(l)
    rng = np.random.default_rng(rows)
    dsq = frame(rng.integers(0, 4, rows).astype(np.uint8))
    mins, maxs = [], []
    for v in range(l.M):
        lo = np.full(rows if v < 12 else 100, 0 if l.sttype[v] == 7 else 1, np.int32)  # v < 12: the first nodes
        hi = lo.copy()
        if l.sttype[v] != 7:
            hi[1:] = 2
            if v < 12 and l.sttype[v] != 5:  # (an IR state's diagonals would pass every row)
                hi[wide + 100] = wide
        mins.append(lo)
        maxs.append(hi)
    bands = Bands.from_rows(np.full(l.M, 1), np.array([len(x) for x in mins]), mins, maxs)
    if truncated:
        tt = tr_tables(cm, l, 4, True)
        valid = tr_valid(l.M, 1, 4, True)
        ro = oracle.tr_hb_scan(l, False, tt, valid, as_tuple(bands), dsq, 1, rows, -6.0, True, 4, -1e30, True)
        go = tr_scan_hb_batch(sc, N.CYK_F32, TrInputs(tt["lmesc"], tt["rmesc"], tt["pty"], tt["lpos"], tt["rpos"],
                                                      tt["clen"], True), 4, True, dsq,
                              [(0, 1, rows, -1e30, -6.0, bands, valid)])[0]
    else:
        ro = oracle.hb_scan(l, False, as_tuple(bands), dsq, 1, rows, -1e30, True, -6.0, True)
        go = hb_scan_batch(sc, N.CYK_F32, True, True, dsq, [(0, 1, rows, -1e30, -6.0, bands)])[0]
    assert same(go, ro)
    sc.close()
