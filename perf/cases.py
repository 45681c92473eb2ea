"""The work a search program has this library do, as cases that can be timed.

listed() names twelve of them, draw() gives more of the same ranges,
prepare() makes what a program holds before the call (residues, windows,
bands, and the uploaded model or filter it keeps from call to call), run()
makes one pass through the public entry points, work() counts the bytes and
operations the pass cannot do without, and exact() gives what run() returns
in 64 bits where the result is a real number (the Forward and bias scores).

The other results have no 64-bit counterpart: hit lists are chosen by a
greedy report on scores defined in scaled integers (Inside), in quantised
bytes and words (SSV, Viterbi) or in single precision with a fixed operand
order (CYK, HMM-banded scans), so exact() returns None for them.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from infernox_b200 import _native as N
from infernox_b200 import calibrate, hb, model, p7, scan, synth

# Consensus structures the repository's own workloads use: the 72-column
# tRNA-like model, the 120-column model of the uneven-window search, and the
# 1,500-column model with 25 bifurcations; other lengths are drawn like the
# models of a cmscan library (30-60% paired, at most one bifurcation per 40
# columns).
OPS_PER_TERM = {scan.CYK_F32: 2.0, scan.INSIDE_I32: 7.0, N.INSIDE_F32: 9.0}
F1, F3, F3B = 0.35, 0.02, 0.02  # filter thresholds of a small database


@functools.lru_cache(maxsize=16)
def _cm(clen, paired, nbif):
    if clen == 72:
        return synth.synth_cm(synth.trna_like(), 11, name="trna")
    return synth.synth_cm(synth.structure(clen, paired, nbif, 31 if clen == 1500 else 5), 23, name="cm%d" % clen)


@functools.lru_cache(maxsize=16)
def _cfg(clen, paired, nbif):
    return model.configure(_cm(clen, paired, nbif), local=True)


def _spec(case):
    return int(case["clen"]), float(case["paired"]), int(case["nbif"])


@functools.lru_cache(maxsize=4)
def _scanner(spec):
    """The uploaded model and its workspace: a search program keeps one per model."""
    return scan.Scanner(_cfg(*spec))


@functools.lru_cache(maxsize=8)
def _tr_inputs(spec):
    return hb.tr_inputs(_cm(*spec), _cfg(*spec), 4, True)


@functools.lru_cache(maxsize=8)
def _profile(m):
    return p7.synthetic_profile(m, 77, 0.6)


@functools.lru_cache(maxsize=4)
def _filters(m):
    prof, _ = _profile(m)
    return (p7.MsvFilter(prof, int(1.25 * m), -8.0, 0.693), p7.VitFilter(prof),
            p7.FwdFilter(prof, p7.mean_composition(prof), -6.0, 0.69))


def listed():
    trna = dict(clen=72, paired=0.5, nbif=2)
    cm120 = dict(clen=120, paired=0.5, nbif=3)
    cm1500 = dict(clen=1500, paired=0.6, nbif=25)
    return [
        # one short window rescored by itself, as the last stage of a search
        # does for a single surviving envelope: latency
        dict(name="window-inside", op="window", n=300, inside=True, band=2, **trna),
        # one window through the Forward filter alone: the smallest call
        dict(name="forward-one", op="forward", m=120, windows=1, length=300),
        # --nohmm search of one 100 kb chunk: QDB1 CYK filter, then QDB2
        # Inside over the envelopes it leaves
        dict(name="nohmm-chunk", op="chunk", n=100000, **trna),
        # --max search: every window of uneven sequences, both strands,
        # non-banded Inside
        dict(name="batch-inside-max", op="batch", seqs=60, median=1500, sigma=0.78, inside=True, band=0, **cm120),
        # a bifurcation-heavy rRNA-sized model over 1 kb windows, CYK filter
        dict(name="batch-cyk-large", op="batch", seqs=1, median=1000, sigma=0.0, inside=False, band=1, **cm1500),
        # cmcalibrate on a short random sample: glocal/local, CYK/Inside scans
        # with cutoff -inf and the tail fits
        dict(name="calibrate", op="calibrate", kb=50, **trna),
        # the default pipeline's first pass over a bacterial genome, both
        # strands: SSV windows, Forward and bias filters, merge
        dict(name="cascade-genome", op="cascade", m=120, total=4600000, chunk=100000),
        # the Viterbi stage of a large database: many odd-length windows
        dict(name="viterbi-windows", op="viterbi", m=151, windows=9001, length=377),
        # the Forward stage: many windows of twice the model's length
        dict(name="forward-windows", op="forward", m=120, windows=13334, length=300),
        # the final stage of the default pipeline: HMM-banded Inside, each
        # envelope with its own bands
        dict(name="hb-inside", op="hb", envelopes=500, slack=20, inside=True, **cm120),
        # its truncated sibling at sequence ends (5' and 3' truncation)
        dict(name="hb-truncated-cyk", op="hbtr", envelopes=200, slack=20, inside=False, **cm120),
        # truncated non-banded Inside of short cut sequences (--max pass)
        dict(name="truncated-inside", op="trq", windows=200, inside=True, band=0, **cm120),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above; none larger than the largest listed."""
    op = rng.choice(["window", "chunk", "batch", "calibrate", "cascade", "viterbi", "forward", "hb", "hbtr", "trq"])
    clen = _log(rng, 40, 400)
    if clen == 72:
        clen = 73
    cm = dict(clen=clen, paired=round(rng.uniform(0.3, 0.6), 3), nbif=rng.randint(0, min(6, clen // 40)))
    inside = rng.random() < 0.5
    small = max(1.0, (clen / 120.0) ** 2)  # larger models: fewer residues
    if op == "window":
        return dict(op=op, n=_log(rng, 100, 2000), inside=inside, band=rng.choice([0, 1, 2]), **cm)
    if op == "chunk":
        return dict(op=op, n=_log(rng, 2000, max(3000, 60000 / small)), **cm)
    if op == "batch":
        return dict(op=op, seqs=_log(rng, 2, max(4, 60 / small)), median=_log(rng, 300, 1500),
                    sigma=round(rng.uniform(0.0, 0.78), 3), inside=inside, band=rng.choice([0, 1, 2]), **cm)
    if op == "calibrate":
        cm = dict(clen=rng.randint(40, 90), paired=0.5, nbif=rng.randint(0, 1))
        return dict(op=op, kb=10 * rng.randint(2, 5), **cm)
    if op == "cascade":
        return dict(op=op, m=_log(rng, 40, 400), total=_log(rng, 50000, 4600000), chunk=rng.choice([100000, 40001]))
    if op in ("viterbi", "forward"):
        m = _log(rng, 20, 400)
        return dict(op=op, m=m, windows=_log(rng, 1, 13334), length=min(2 * int(1.25 * m) + rng.randint(0, 9), 600))
    if op == "hb":
        return dict(op=op, envelopes=_log(rng, 1, max(2, 500 / small)), slack=rng.randint(4, 20), inside=inside, **cm)
    if op == "hbtr":
        return dict(op=op, envelopes=_log(rng, 1, max(2, 200 / small)), slack=rng.randint(4, 20), inside=inside, **cm)
    return dict(op="trq", windows=_log(rng, 1, max(2, 200 / small)), inside=inside, band=rng.choice([0, 1, 2]), **cm)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _frames(seqs):
    """Window frames [255, residues, 255] back to back, and their windows."""
    parts, wins, off = [], [], 0
    for s in seqs:
        parts.append(np.concatenate([[255], s, [255]]).astype(np.uint8))
        wins.append((off, 1, len(s)))
        off += len(s) + 2
    return np.concatenate(parts), np.array(wins, N.WINDOW_DTYPE)


def _plant(seq, cm, rng):
    h = synth.emit(cm, rng)[: len(seq)]
    if len(h):
        q = int(rng.integers(0, len(seq) - len(h) + 1))
        seq[q:q + len(h)] = h
    return seq


def _lengths(case):
    """Sequence lengths of a batch: log-normal quantiles, clipped to 200 nt - 20 kb."""
    n = int(case["seqs"])
    u = torch.tensor([(k + 0.5) / n for k in range(n)], dtype=torch.float64)
    z = torch.erfinv(2 * u - 1).numpy() * math.sqrt(2.0)
    return np.clip(case["median"] * np.exp(case["sigma"] * z), 200, 20000).astype(int)


def _bands(cfg, rects):
    """ij2d_bands of one envelope's per-state rectangles, all rows at once."""
    im, ix, jm, jx = (np.asarray(r, np.int64) for r in rects)
    n = np.maximum(0, jx - jm + 1)
    off = np.concatenate([[0], np.cumsum(n)[:-1]])
    v = np.repeat(np.arange(len(n)), n)
    j = np.arange(int(n.sum())) - off[v] + jm[v]
    st = np.asarray(cfg.sttype)[v]
    sd = np.where(st == 1, 2, np.where((st >= 2) & (st <= 5), 1, 0))
    lo, hi = j - ix[v] + 1, j - im[v] + 1
    empty = hi < sd
    mn = np.where(st == 7, 0, np.where(empty, -1, np.maximum(lo, sd)))
    mx = np.where(st == 7, 0, np.where(empty, -2, hi))
    c = lambda a: np.ascontiguousarray(a, np.int32)  # noqa: E731
    return hb.Bands(c(jm), c(jx), c(off), c(mn), c(mx))


def _envelopes(case, rng):
    """Envelopes of W residues, one homolog each, with CP9-shaped bands."""
    spec = _spec(case)
    cm, cfg = _cm(*spec), _cfg(*spec)
    seqs, tasks, off = [], [], 0
    for _ in range(int(case["envelopes"])):
        h = synth.emit(cm, rng)
        n = cfg.W + 40
        s = synth.random_dsq(n, 0.45, rng)
        q = int(rng.integers(10, max(11, n - len(h) - 10)))
        s[q - 1:q - 1 + len(h)] = h[: n - q + 1]
        i0, j0 = 5, 5 + cfg.W - 1
        rects = synth.hb_band_rects(cm.st, q, i0, j0, int(case["slack"]), rng)
        tasks.append((off, i0, j0, 0.0, 0.0, _bands(cfg, rects)))
        seqs.append(s)
        off += n + 2
    return _frames(seqs)[0], tasks


def _chunked(total, chunk, cons, rng):
    top = p7.planted_residues(total, cons, max(1, total // 115000), int(rng.integers(1 << 30)), gc=0.508)
    return _frames([s[a:a + chunk] for s in (top, synth.revcomp(top)) for a in range(0, total, chunk)])


def prepare(case, seed):
    rng = np.random.default_rng(int(seed))
    op = case["op"]
    st = {"op": op, "case": case, "seed": int(seed)}
    if op in ("window", "chunk", "batch", "hb", "hbtr", "trq"):
        spec = _spec(case)
        cm = _cm(*spec)
        st["scanner"] = _scanner(spec)
    if op in ("window", "chunk"):
        s = synth.random_dsq(int(case["n"]), 0.5, rng)
        for _ in range(1 + int(case["n"]) // 10000):
            _plant(s, cm, rng)
        st["dsq"] = _frames([s])[0]
    elif op == "batch":
        seqs = []
        for k, n in enumerate(_lengths(case)):
            s = synth.random_dsq(int(n), 0.45, rng)
            if k % 10 == 0:
                _plant(s, cm, rng)
            seqs += [s, synth.revcomp(s)]
        st["buf"], st["wins"] = _frames(seqs)
    elif op == "calibrate":
        st["cm"], st["W"] = _cm(*_spec(case)), _cfg(*_spec(case)).W
    elif op in ("cascade", "viterbi", "forward"):
        m = int(case["m"])
        _, cons = _profile(m)
        st["filters"] = _filters(m)
        if op == "cascade":
            st["buf"], st["wins"] = _chunked(int(case["total"]), int(case["chunk"]), cons, rng)
        else:
            n, ln = int(case["windows"]), int(case["length"])
            s = p7.planted_residues(n * ln, cons, max(1, n // 100), int(rng.integers(1 << 30)), gc=0.508)
            buf = np.full((n, ln + 2), 255, np.uint8)
            buf[:, 1:-1] = s.reshape(n, ln)
            st["buf"] = buf.reshape(-1)
            st["wins"] = np.zeros(n, N.WINDOW_DTYPE)
            st["wins"]["dsq_offset"] = np.arange(n) * (ln + 2)
            st["wins"]["i0"], st["wins"]["j0"] = 1, ln
    elif op in ("hb", "hbtr"):
        st["buf"], st["tasks"] = _envelopes(case, rng)
        if op == "hbtr":
            ones = np.ones(_cfg(*spec).M, np.uint8)
            st["tasks"] = [t + ((ones, ones, ones, ones),) for t in st["tasks"]]
            st["tri"] = _tr_inputs(spec)
    elif op == "trq":
        seqs = []
        for _ in range(int(case["windows"])):
            h = synth.emit(cm, rng)
            seqs.append(np.concatenate([synth.random_dsq(20, 0.45, rng), h[len(h) // 4:len(h) - len(h) // 5],
                                        synth.random_dsq(20, 0.45, rng)]))
        st["buf"], st["wins"] = _frames(seqs)
        st["tri"] = _tr_inputs(spec)
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _columns(a, room):
    """The fields of a hit list, in arrays of `room` entries (zeros after the last hit)."""
    out = {k: np.zeros(room, a.dtype[k]) for k in a.dtype.names}
    for k in out:
        out[k][:len(a)] = a[k]
    return out


def _rows(rows, width, room, dtype=np.float64):
    """A hit list as a table of `room` rows (zeros after the last hit)."""
    out = np.zeros((room, width), dtype)
    if len(rows):
        out[:len(rows)] = rows
    return out


def run(st):
    op, case = st["op"], st["case"]
    if op == "window":
        sr = scan.INSIDE_I32 if case["inside"] else scan.CYK_F32
        return _rows(st["scanner"].generic_scan(sr, case["band"], st["dsq"], 1, case["n"], 10.0, True), 4, case["n"])
    if op == "chunk":
        sc = st["scanner"]
        envs = sc.cyk_seq_filter(st["dsq"], case["n"], 12.0, True)
        return {"envelopes": _rows(envs, 2, case["n"] // 4 + 1, np.int64),
                "hits": _rows(sc.final_stage_inside(st["dsq"], envs, 15.0, True), 4, case["n"] // 4 + 1)}
    if op == "batch":
        sr = scan.INSIDE_I32 if case["inside"] else scan.CYK_F32
        hits = st["scanner"].scan_batch(sr, case["band"], st["buf"], st["wins"], 15.0, True)
        return _columns(hits, 64 + 16 * len(st["wins"]))
    if op == "calibrate":
        cfg = calibrate.CalibrateConfig(seed=1 + st["seed"] % 100000, l_mb=case["kb"] / 1000.0)
        r = calibrate.calibrate_cm(st["cm"], cfg, W=st["W"])
        return {"exp": [[e[k] for k in ("lambda_", "mu", "mu_orig", "tailp", "nrandhits")] for e in r["exp"]],
                "nhits": r["nhits"]}
    if op == "cascade":
        mf, vf, ff = st["filters"]
        w, acct = p7.f3_filter_batch(ff, st["buf"], st["wins"], F1, F3, F3B, int(case["m"] * 1.25), mf=mf)
        return {"windows": _columns(w, 1024 + case["total"] // 16), "accounting": acct}
    if op == "viterbi":
        return list(st["filters"][1].score_batch(st["buf"], st["wins"]))
    if op == "forward":
        return list(st["filters"][2].score_batch(st["buf"], st["wins"]))
    if op == "hb":
        sr = N.INSIDE_F32 if case["inside"] else N.CYK_F32
        r = hb.hb_scan_batch(st["scanner"], sr, True, True, st["buf"], st["tasks"])
        return {"vsc": np.array([x[0] for x in r], np.float32), "env": np.array([x[1:3] for x in r], np.int64),
                "nhits": np.array([len(x[3]) for x in r]), "hits": _rows([h for x in r for h in x[3]], 4, 64 * len(r))}
    if op == "hbtr":
        sr = N.INSIDE_F32 if case["inside"] else N.CYK_F32
        r = hb.tr_scan_hb_batch(st["scanner"], sr, st["tri"], 4, True, st["buf"], st["tasks"])
        return {"vsc": np.array([x[1] for x in r], np.float32), "mode": np.array([x[2] for x in r]),
                "env": np.array([x[3:5] for x in r], np.int64), "nhits": np.array([len(x[0]) for x in r]),
                "hits": _rows([h for x in r for h in x[0]], 6, 64 * len(r))}
    sr = N.INSIDE_I32 if case["inside"] else N.CYK_F32
    r = hb.tr_qdb_scan_batch(st["scanner"], sr, case["band"], st["tri"], 4, True, st["buf"], st["wins"], 0.0)
    return {"vsc": np.array([x[1] for x in r], np.float32), "mode": np.array([x[2] for x in r]),
            "full": np.array([x[3] for x in r], np.float32), "nhits": np.array([len(x[0]) for x in r]),
            "hits": _rows([h for x in r for h in x[0]], 6, 64 * len(r))}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _scan_flops(cfg, sr, band, lengths):
    f = 0.0
    for n in lengths:
        c, t = cfg.count_work(sr, band, int(n))
        f += t * OPS_PER_TERM[sr] + 2.0 * c
    return f


def _model_bytes(cfg):
    return sum(a.nbytes for a in (cfg.tsc, cfg.oesc, cfg.endsc, cfg.beginsc, cfg.dmin1, cfg.dmax1))


def work(case):
    """Residues and model tables read once, results written once; operations:
    two per child relaxation in max-plus, seven in integer log-sum (nine in
    the float one) and two per cell, as the repository's benchmark counts."""
    op = case["op"]
    if op in ("window", "chunk", "batch", "calibrate"):
        cfg = _cfg(*_spec(case))
        sr = scan.INSIDE_I32 if case.get("inside") else scan.CYK_F32
        if op == "window":
            return {"bytes": case["n"] + _model_bytes(cfg), "flops": _scan_flops(cfg, sr, case["band"], [case["n"]])}
        if op == "chunk":
            # the Inside stage sees only the envelopes of the few planted homologs
            env = [3 * cfg.W] * (1 + case["n"] // 10000)
            return {"bytes": case["n"] + _model_bytes(cfg),
                    "flops": _scan_flops(cfg, scan.CYK_F32, 1, [case["n"]])
                    + _scan_flops(cfg, scan.INSIDE_I32, 2, env)}
        if op == "batch":
            ln = _lengths(case)
            return {"bytes": 2 * int(ln.sum()) + _model_bytes(cfg),
                    "flops": 2 * _scan_flops(cfg, sr, case["band"], ln)}
        n = calibrate.n_sequences(calibrate.CalibrateConfig(l_mb=case["kb"] / 1000.0))
        ln = [calibrate.EXPTAIL_CHUNKLEN] * n
        return {"bytes": 10000 * n + _model_bytes(cfg),
                "flops": 2 * (_scan_flops(cfg, scan.CYK_F32, 2, ln[:1]) + _scan_flops(cfg, scan.INSIDE_I32, 2, ln[:1])) * n}
    if op == "cascade":
        return {"bytes": 2 * case["total"], "flops": 4.0 * 2 * case["total"] * case["m"]}
    if op in ("viterbi", "forward"):
        n = case["windows"] * case["length"]
        return {"bytes": n + 8 * case["windows"], "flops": (14.0 if op == "viterbi" else 16.0) * n * case["m"]}
    cfg = _cfg(*_spec(case))
    live = int(np.sum(~np.isin(np.asarray(cfg.sttype), (7,))))
    if op in ("hb", "hbtr"):
        # a state's rectangle is about slack x slack cells around its place
        cells = case["envelopes"] * live * (case["slack"] + 1.0) ** 2
        rows = case["envelopes"] * live * (case["slack"] + 1.0)
        per = 3.0 * OPS_PER_TERM[N.INSIDE_F32 if case["inside"] else N.CYK_F32] + 2.0
        return {"bytes": 8.0 * rows + case["envelopes"] * (cfg.W + 40), "flops": cells * per * (3 if op == "hbtr" else 1)}
    n = int(0.55 * cfg.clen) + 40
    c, t = cfg.count_work(scan.CYK_F32, case["band"], n)
    per = OPS_PER_TERM[scan.INSIDE_I32 if case["inside"] else scan.CYK_F32]
    return {"bytes": case["windows"] * n + _model_bytes(cfg), "flops": 3.0 * case["windows"] * (t * per + 2.0 * c)}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def exact(case, seed):
    """Forward and bias-filter scores (nats) of each window from the profile's
    probabilities, in float64: the local multihit Forward recurrence in odds
    space over a uniform null, uniform local entries weighted by match
    occupancy, and the two-state composition null."""
    if case["op"] != "forward":
        return None
    st = prepare(case, seed)
    prof, _ = _profile(int(case["m"]))
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
    m, n, ln = int(case["m"]), int(case["windows"]), int(case["length"])
    dsq = torch.as_tensor(st["buf"].reshape(n, ln + 2)[:, 1:-1].astype(np.int64), device=dev)
    odds = f64(prof.mat)[1:] / 0.25                       # [m, 4]
    t = np.asarray(prof.trans, np.float64)
    occ = np.zeros(m + 1)
    occ[1] = t[0, 0] + t[0, 1]
    for k in range(2, m + 1):
        occ[k] = occ[k - 1] * (t[k - 1, 0] + t[k - 1, 1]) + (1.0 - occ[k - 1]) * t[k - 1, 5]
    z = sum(occ[k] * (m - k + 1) for k in range(1, m + 1))
    tbm = f64(occ[1:] / z)
    mm, im, dm = f64(t[:m, 0]), f64(t[:m, 3]), f64(t[:m, 5])   # into k = 1..m from k-1
    mi, ii = t[1:, 1].copy(), t[1:, 4].copy()
    md, dd = t[1:, 2].copy(), t[1:, 6].copy()
    mi[-1] = ii[-1] = md[-1] = dd[-1] = 0.0
    mi, ii = f64(mi), f64(ii)
    chain = np.zeros((m, m))                                # D(k) from M(k'), k' < k
    for a in range(m):
        x = md[a]
        for k in range(a + 1, m):
            chain[a, k] = x
            x *= dd[k]
    chain = f64(chain)
    shift = lambda a: torch.nn.functional.pad(a[:, :-1], (1, 0))  # noqa: E731
    M = torch.zeros(n, m, dtype=torch.float64, device=dev)
    I, D = M.clone(), M.clone()
    move = 3.0 / (ln + 3.0)
    loop = 1.0 - move
    one = torch.ones(n, 1, dtype=torch.float64, device=dev)
    xn, xj, xc, xb, tot = one, 0 * one, 0 * one, move * one, 0 * one
    for i in range(ln):
        M2 = (xb * tbm + shift(M) * mm + shift(I) * im + shift(D) * dm) * odds[:, dsq[:, i]].T
        I2 = M * mi + I * ii
        D2 = M2 @ chain
        xe = (M2 + D2).sum(1, keepdim=True)
        xn = xn * loop
        xc, xj = xc * loop + 0.5 * xe, xj * loop + 0.5 * xe
        xb = (xj + xn) * move
        s = torch.where(xe > 1e4, xe, one)
        M, I, D, xn, xc, xj, xb, tot = M2 / s, I2 / s, D2 / s, xn / s, xc / s, xj / s, xb / s, tot + s.log()
    fwd = (tot + (xc * move).log()).squeeze(1)
    # bias null: background state against the model's mean composition, which
    # lasts m/8 residues on average and is entered once in a thousand
    comp = f64(p7.mean_composition(prof))
    stay = m / 8.0
    p1 = ln / (ln + 1.0)
    t1 = (1.0 / (stay + 1.0), stay / (stay + 1.0))
    e1 = comp / 0.25
    f0, g0 = 0.999 * torch.ones(n, dtype=torch.float64, device=dev), 0.001 * e1[dsq[:, 0]]
    sc = torch.zeros(n, dtype=torch.float64, device=dev)
    for i in range(1, ln):
        s = f0 + g0
        sc = sc + s.log()
        f0, g0 = f0 / s, g0 / s
        f0, g0 = f0 * p1 + g0 * t1[0], (f0 * (1 - p1) + g0 * t1[1]) * e1[dsq[:, i]]
    bias = sc + (f0 + g0).log() + ln * math.log(p1) + math.log(1.0 - p1)
    return [fwd.cpu().numpy(), bias.cpu().numpy()]
