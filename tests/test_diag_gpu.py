"""The diagonal scan kernel (what KERNEL_AUTO runs) at the sizes where its
tiling can go wrong: a warp's 32 columns, a CTA's group of columns, the last
partial group, windows shorter than W, forced pieces -- against the oracle
bit for bit, and every ROOT cell against the level kernel over all semirings,
band sets and configurations."""
import dataclasses
import time

import numpy as np
import pytest

import oracle
from infernox_b200 import _native as N
from infernox_b200 import model, scan, synth
from infernox_b200.scan import CYK_F32, INSIDE_I32, KERNEL_LEVEL, NOQDB, QDB1, QDB2

from helpers import frame, models, oracle_cfg, planted_seq

pytestmark = pytest.mark.gpu

DIAG = 3  # CMGPU_KERNEL_DIAG in the statistics


def seq_of(cm, n, seed):
    if n < 100:
        return np.random.default_rng(seed).integers(0, 4, n).astype(np.uint8)
    return planted_seq(cm, n, 0.5, 1 + n // 1000, seed=seed, degenerate=0.01)


def bits(hits):
    return [(h[0], h[1], np.float32(h[2]).tobytes(), np.float32(h[3]).tobytes()) for h in hits]


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 256, 257, 511, 512, 513, 1100])
@pytest.mark.parametrize("name", ["small0", "mb3"])
@pytest.mark.parametrize("sr,band", [(CYK_F32, QDB1), (INSIDE_I32, QDB2), (INSIDE_I32, NOQDB)])
def test_edges_match_oracle(name, n, sr, band):
    cm, _, l = models(name)
    dsq = frame(seq_of(cm, n, 100 + n))
    ref, _, _, _ = oracle.qdb_scan(oracle_cfg(name, True), sr, band, dsq, 1, n, -20.0, True)
    s = scan.Scanner(l)
    got = s.generic_scan(sr, band, dsq, 1, n, -20.0, True)
    assert s.stats()["kernel"] == DIAG
    assert bits(got) == bits(ref)


@pytest.mark.parametrize("name", ["small0", "trna", "small2", "mb3", "cfg2"])
@pytest.mark.parametrize("local", [False, True])
@pytest.mark.parametrize("sr", [CYK_F32, INSIDE_I32])
@pytest.mark.parametrize("band", [NOQDB, QDB1, QDB2])
def test_every_root_cell_matches_level_kernel(name, local, sr, band):
    cm, g, l = models(name)
    a, b = scan.Scanner(l if local else g), scan.Scanner(l if local else g)
    b.set_kernel(KERNEL_LEVEL)
    for n, chunk in ((40, 0), (700, 0), (1500, 130)):
        dsq = frame(seq_of(cm, n, n))
        a.set_shape(0, 0, chunk, 0)
        ca, cb = a.scan_cells(sr, band, dsq, 1, n, -30.0), b.scan_cells(sr, band, dsq, 1, n, -30.0)
        assert (a.stats()["kernel"], b.stats()["kernel"]) == (DIAG, KERNEL_LEVEL)
        assert ca == cb


@pytest.mark.parametrize("sr", [CYK_F32, INSIDE_I32])
@pytest.mark.parametrize("null3", [False, True])
def test_calibration_scan_matches_level_kernel(sr, null3):
    cm, g, l = models("trna")
    buf = frame(seq_of(cm, 1500, 9))
    w = np.array([(0, 1, 1500), (0, 500, 1200), (0, 1, 40), (0, 900, 899)], N.WINDOW_DTYPE)
    for c in (g, l):
        a, b = scan.Scanner(c), scan.Scanner(c)
        b.set_kernel(KERNEL_LEVEL)
        x = a.calibrate_scan_batch(sr, QDB2, buf, w, null3)
        y = b.calibrate_scan_batch(sr, QDB2, buf, w, null3)
        assert len(x) > 0 and x.tobytes() == y.tobytes()


# (chunk: residues reported per item, which adds W-1 columns before them; a
# group of columns holds 512 at most, so 1,152 takes three groups and 500 two.
# small2 has 44 nodes that own a buffer, two more than a multiple of three, and
# a ROOT of five steps of sixteen spans.)
@pytest.mark.parametrize("chunk,n", [(500, 1400), (1152, 3000)])
@pytest.mark.parametrize("name", ["small0", "trna", "small2", "mb3"])
@pytest.mark.parametrize("sr,band", [(CYK_F32, QDB1), (INSIDE_I32, QDB2), (INSIDE_I32, NOQDB)])
def test_glocal_column_groups_match_level_kernel(name, sr, band, chunk, n):
    cm, g, _ = models(name)
    a, b = scan.Scanner(g), scan.Scanner(g)
    b.set_kernel(KERNEL_LEVEL)
    a.set_shape(0, 0, chunk, 0)
    dsq = frame(seq_of(cm, n, n))
    ca, cb = a.scan_cells(sr, band, dsq, 1, n, -500.0), b.scan_cells(sr, band, dsq, 1, n, -500.0)
    assert a.stats()["kernel"] == DIAG and len(ca) > n
    assert ca == cb


# Local begins start from an empty row in every group of columns: the row of
# the group before it must be gone when the first node reads it.
@pytest.mark.parametrize("chunk,n", [(500, 1400), (1152, 3000)])
@pytest.mark.parametrize("name", ["small0", "small2", "mb3"])
@pytest.mark.parametrize("sr,band", [(CYK_F32, QDB1), (INSIDE_I32, NOQDB)])
def test_local_begins_of_column_groups_match_level_kernel(name, sr, band, chunk, n):
    cm, _, l = models(name)
    a, b = scan.Scanner(l), scan.Scanner(l)
    b.set_kernel(KERNEL_LEVEL)
    a.set_shape(0, 0, chunk, 0)
    dsq = frame(seq_of(cm, n, 7 * n))
    ca, cb = a.scan_cells(sr, band, dsq, 1, n, -500.0), b.scan_cells(sr, band, dsq, 1, n, -500.0)
    assert a.stats()["kernel"] == DIAG and len(ca) > n
    assert ca == cb


# Bands that begin at span 5 in every state: the first node of a group then
# starts with residues of the warps on its left.
@pytest.mark.parametrize("name", ["small0", "mb3"])
@pytest.mark.parametrize("sr,band", [(CYK_F32, QDB1), (INSIDE_I32, QDB2)])
def test_bands_without_short_spans_match_oracle(name, sr, band):
    cm, _, _ = models(name)
    ref = oracle_cfg(name, True)
    up = {k: np.where(np.asarray(ref.sttype) == 7, getattr(ref, k), np.maximum(getattr(ref, k), 5)).astype(np.int32)
          for k in ("dmin1", "dmin2")}
    up.update({k: np.maximum(getattr(ref, k), up["dmin" + k[-1]]).astype(np.int32) for k in ("dmax1", "dmax2")})
    c = dataclasses.replace(ref, **up, _struct=None)
    s = scan.Scanner(c)
    for n in (40, 700):
        dsq = frame(seq_of(cm, n, 3 * n))
        want, _, _, _ = oracle.qdb_scan(c, sr, band, dsq, 1, n, -60.0, True)
        got = s.generic_scan(sr, band, dsq, 1, n, -60.0, True)
        assert s.stats()["kernel"] == DIAG
        assert len(want) > 0 and bits(got) == bits(want)


# Models of three and five nodes: a group of columns takes fewer steps than a
# warp may be ahead of its right neighbour.
@pytest.mark.parametrize("ss", ["..", "....", "(...)"])
@pytest.mark.parametrize("local", [False, True])
@pytest.mark.parametrize("sr,band", [(CYK_F32, QDB1), (INSIDE_I32, QDB2), (INSIDE_I32, NOQDB)])
def test_tiny_models_match_level_kernel(ss, local, sr, band):
    cm = synth.synth_cm(ss, 1, name="tiny", ins_open=0.005, ins_self=0.1)
    c = model.configure(cm, local=local)
    a, b = scan.Scanner(c), scan.Scanner(c)
    b.set_kernel(KERNEL_LEVEL)
    for n, chunk in ((257, 0), (3000, 0), (3000, 1152)):
        a.set_shape(0, 0, chunk, 0)
        dsq = frame(seq_of(cm, n, n))
        ca, cb = a.scan_cells(sr, band, dsq, 1, n, -500.0), b.scan_cells(sr, band, dsq, 1, n, -500.0)
        assert (a.stats()["kernel"], b.stats()["kernel"]) == (DIAG, KERNEL_LEVEL)
        assert len(ca) > n and ca == cb


# Failure detection without a GPU fault: a warp waits for a step that its
# neighbour never reaches, gives up, and so does every other wait; the same
# workspace then scans correctly.
@pytest.mark.parametrize("n", [100, 3000])
@pytest.mark.parametrize("sr,band", [(CYK_F32, QDB1), (INSIDE_I32, NOQDB)])
def test_waits_of_the_diagonal_scan_run_out(sr, band, n):
    cm, _, l = models("small2")
    s = scan.Scanner(l)
    s.set_shape(0, 0, 1152, 0)
    dsq = frame(seq_of(cm, n, 70 + n))
    want, _, _, _ = oracle.qdb_scan(oracle_cfg("small2", True), sr, band, dsq, 1, n, -20.0, True)
    for _ in range(2):
        N.check(N.lib().cmgpu_workspace_inject_stall(s._ws))
        t0 = time.perf_counter()
        with pytest.raises(N.CmgpuError, match="timed out") as ei:
            s.generic_scan(sr, band, dsq, 1, n, -20.0, True)
        assert ei.value.rc == N.CMGPU_ETIMEOUT and time.perf_counter() - t0 < 30
        assert bits(s.generic_scan(sr, band, dsq, 1, n, -20.0, True)) == bits(want)
        assert s.stats()["kernel"] == DIAG


def test_autotune_tries_what_acts():
    cm, _, l = models("small2")
    dsq = frame(seq_of(cm, 2000, 5))
    w = np.array([(0, 1, 2000), (0, 300, 900)], N.WINDOW_DTYPE)
    s = scan.Scanner(l)
    t = s.autotune(INSIDE_I32, NOQDB, dsq, w, 5.0, chunks_w=(0, 4))
    assert s.stats()["kernel"] == DIAG and s.stats()["lanes"] == 1  # work items per CTA
    assert [x["chunk"] for x in t["trials"]] == [0, 4 * l.W]
    s.set_kernel(KERNEL_LEVEL)
    t = s.autotune(INSIDE_I32, NOQDB, dsq, w, 5.0, lanes=(1, 2), chunks_w=(0, 4))
    assert len(t["trials"]) == 4
