"""Scans on a device whose memory others hold: fewer CTAs or the level kernel,
and the same cells."""
import dataclasses

import numpy as np
import pytest
import torch

from infernox_b200 import _native as N
from infernox_b200 import model, scan, synth
from infernox_b200.hb import TrInputs, tr_qdb_scan_batch
from infernox_b200.scan import CYK_F32, INSIDE_I32, KERNEL_LEVEL, NOQDB

from hb_helpers import tr_tables
from helpers import frame, models, planted_seq

pytestmark = pytest.mark.gpu

DIAG = 3  # CMGPU_KERNEL_DIAG in the statistics


# W = 6,000: one region of the diagonal kernel is 670 MB, a deck of the level
# kernel 450 MB (both hold W x W per bifurcation; the level kernel takes a deck
# per item, so it gets one item, the diagonal kernel three).
@pytest.mark.parametrize("leave_mb,chunk,kernel", [(560, 0, KERNEL_LEVEL), (1500, 100, DIAG)])
def test_scan_with_little_device_memory(leave_mb, chunk, kernel):
    cm, _, l = models("mb3")
    c = dataclasses.replace(l, W=6000, _struct=None)
    dsq = frame(planted_seq(cm, 300, 0.5, 1, seed=4))
    a = scan.Scanner(c)
    a.set_shape(0, 0, chunk, 0)
    want = a.scan_cells(INSIDE_I32, NOQDB, dsq, 1, 300, -30.0)
    assert a.stats()["kernel"] == DIAG and len(want) > 0
    a.close()
    torch.cuda.empty_cache()
    b = scan.Scanner(c)
    b.set_shape(0, 0, chunk, 0)
    held = torch.empty(torch.cuda.mem_get_info()[0] - (leave_mb << 20), dtype=torch.uint8, device="cuda")
    try:
        got = b.scan_cells(INSIDE_I32, NOQDB, dsq, 1, 300, -30.0)
        assert b.stats()["kernel"] == kernel
    finally:
        del held
        torch.cuda.empty_cache()
    assert got == want
    b.close()


# 16 reportable cells per column of a 4,000,000-column window would take 1.9 GB.
def test_truncated_scan_with_little_device_memory():
    cm = synth.synth_cm("(...)", 1, name="tiny", ins_open=0.005, ins_self=0.1)
    c = model.configure(cm, local=True)
    tt = tr_tables(cm, c, 4, True)
    tri = TrInputs(tt["lmesc"], tt["rmesc"], tt["pty"], tt["lpos"], tt["rpos"], tt["clen"], True,
                   tt["ilmesc"], tt["irmesc"], tt["ipty"])
    n = 4000000
    dsq = frame(synth.random_dsq(n, 0.5, np.random.default_rng(3)))
    w = np.array([(0, 1, n)], N.WINDOW_DTYPE)
    res = []
    for leave_mb in (None, 1200):
        sc = scan.Scanner(c)
        held = None
        if leave_mb:
            held = torch.empty(torch.cuda.mem_get_info()[0] - (leave_mb << 20), dtype=torch.uint8, device="cuda")
        try:
            res.append(tr_qdb_scan_batch(sc, CYK_F32, NOQDB, tri, 4, True, dsq, w, 3.0))
        finally:
            del held
            torch.cuda.empty_cache()
        sc.close()
    assert len(res[0][0][0]) > 0 and res[0] == res[1]
