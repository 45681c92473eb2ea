"""Scans on a device whose memory others hold: fewer CTAs or the level kernel,
and the same cells."""
import dataclasses

import pytest
import torch

from infernox_b200 import scan
from infernox_b200.scan import INSIDE_I32, KERNEL_LEVEL, NOQDB

from helpers import frame, models, planted_seq

pytestmark = pytest.mark.gpu

DIAG = 3  # CMGPU_KERNEL_DIAG in the statistics


# W = 6,000: one region of the diagonal kernel is 670 MB, a deck of the level
# kernel 450 MB (both hold W x W per bifurcation; the level kernel takes a deck
# per item, so it gets one item, the diagonal kernel three).
@pytest.mark.parametrize("leave_mb,chunk,kernel", [(560, 0, KERNEL_LEVEL), (1500, 100, DIAG)])
def test_scan_with_little_device_memory(leave_mb, chunk, kernel):
    cm, _, l = models("mb3")
    c = dataclasses.replace(l, W=6000)
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
