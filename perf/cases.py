"""Performance cases of the Hallen solver: what a user's program asks of it,
over the range of sizes, structures and precisions it is used with.

Each case names the structure, its size and the precision; prepare() builds
the geometry from a seed and plans it (HallenBatch, Server) or lays out the
host arrays of a single call; run() is one pass through the public entry
points, from the host inputs to the host results that a report prints.

Structures:
  dipole  one centre-fed wire along z
  array   parallel wires along z, the second (or only) one driven
  uneven  random antennas of 1-8 straight wires of 11-101 segments in a 20 m
          cube, one frequency each, free space or perfect ground
  mesh    junctioned wire grid over perfect ground, 2 segments per edge
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "fnec-rust_b200"))

import nec_accel as acc  # noqa: E402

C0 = 299792458.0
F0 = 14.2e6
ETA0 = 4.0 * math.pi * 1e-7 * C0
RHS_SCALE = 2.0 * math.pi / ETA0


def listed():
    return [
        # the smallest whole job: a centre-fed dipole and its elevation cut,
        # as an interactive user runs it; latency and launches
        {"name": "dipole_cut", "kind": "solve", "family": "dipole", "precision": "fp64", "wires": 1, "segments": 51,
         "freqs": 1, "ground": 0, "n_theta": 181, "n_phi": 1},
        # one frequency of a Yagi-sized array through the call that replaces
        # the reference's single-solve accelerator entry
        {"name": "array_call", "kind": "call", "family": "array", "precision": "fp64", "wires": 5, "segments": 51,
         "ground": 0},
        # an ordinary sweep with a coarse pattern per frequency, plain form
        {"name": "array_sweep_plain", "kind": "solve", "family": "array", "precision": "fp64", "wires": 5,
         "segments": 51, "freqs": 41, "ground": 0, "n_theta": 37, "n_phi": 73},
        # the full sweep: 201 frequencies, 1 degree hemisphere each, mixed form
        {"name": "array_sweep_mixed", "kind": "solve", "family": "array", "precision": "mixed", "wires": 5,
         "segments": 51, "freqs": 201, "ground": 0, "n_theta": 91, "n_phi": 361},
        # a population of candidate antennas (an optimiser's generation),
        # plain form
        {"name": "uneven_plain", "kind": "solve", "family": "uneven", "precision": "fp64", "antennas": 512},
        # the largest batch, mixed form
        {"name": "uneven_mixed", "kind": "solve", "family": "uneven", "precision": "mixed", "antennas": 4096},
        # a junctioned grid over ground in each form, the mixed one at the
        # largest size in use (S = 12,972 unknowns)
        {"name": "mesh_plain", "kind": "solve", "family": "mesh", "precision": "fp64", "cells": 20},
        {"name": "mesh_mixed", "kind": "solve", "family": "mesh", "precision": "mixed", "cells": 46},
        # a receiving array: every incidence direction a right-hand side
        {"name": "receive_sweep", "kind": "receive", "wires": 5, "segments": 51, "freqs": 3, "n_theta": 37,
         "n_phi": 72},
        # near fields over a plane beside the array
        {"name": "near_plane", "kind": "near", "wires": 5, "segments": 51, "nx": 64, "ny": 64},
        # a far-field pattern of given currents in one call
        {"name": "pattern_call", "kind": "pattern", "wires": 5, "segments": 51, "ground": 1, "n_theta": 19,
         "n_phi": 73},
        # a burst of independent requests through the server
        {"name": "serve_burst", "kind": "serve", "precision": "mixed", "requests": 256},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _odd(rng, lo, hi):
    return 2 * (_log_int(rng, lo, hi) // 2) + 1


def draw(rng):
    while True:
        kind = rng.choice(["dipole", "call", "sweep", "sweep", "uneven", "uneven", "mesh", "mesh", "receive", "near",
                           "pattern", "serve"])
        precision = rng.choice(["fp64", "mixed"])
        mixed = precision == "mixed"
        step = rng.choice([1, 2, 3, 5, 10])
        ground = rng.randint(0, 1)
        n_theta, n_phi = (90 if ground else 180) // step + 1, rng.choice([1, 2, 360 // step + 1])
        if kind == "dipole":
            c = {"kind": "solve", "family": "dipole", "precision": precision, "wires": 1,
                 "segments": _odd(rng, 11, 301), "freqs": 1, "ground": ground, "n_theta": n_theta, "n_phi": n_phi}
        elif kind == "call":
            c = {"kind": "call", "family": "array", "precision": precision, "wires": rng.randint(1, 6),
                 "segments": _odd(rng, 11, 101), "ground": ground}
        elif kind == "sweep":
            c = {"kind": "solve", "family": "array", "precision": precision, "wires": rng.randint(1, 6),
                 "segments": _odd(rng, 11, 101), "freqs": _log_int(rng, 3, 201 if mixed else 61), "ground": ground,
                 "n_theta": n_theta, "n_phi": n_phi}
        elif kind == "uneven":
            c = {"kind": "solve", "family": "uneven", "precision": precision,
                 "antennas": _log_int(rng, 8, 4096 if mixed else 512)}
        elif kind == "mesh":
            c = {"kind": "solve", "family": "mesh", "precision": precision,
                 "cells": _log_int(rng, 4, 46 if mixed else 20)}
        elif kind == "receive":
            c = {"kind": "receive", "wires": rng.randint(1, 6), "segments": _odd(rng, 11, 81),
                 "freqs": rng.randint(1, 5), "n_theta": _log_int(rng, 3, 37), "n_phi": _log_int(rng, 3, 72)}
        elif kind == "near":
            c = {"kind": "near", "wires": rng.randint(1, 6), "segments": _odd(rng, 11, 101),
                 "nx": _log_int(rng, 4, 128), "ny": _log_int(rng, 4, 128)}
        elif kind == "pattern":
            c = {"kind": "pattern", "wires": rng.randint(1, 6), "segments": _odd(rng, 11, 101), "ground": ground,
                 "n_theta": n_theta, "n_phi": n_phi}
        else:
            c = {"kind": "serve", "precision": precision, "requests": _log_int(rng, 8, 256)}
        # patterns no larger than the listed sweep's
        if c.get("n_theta", 1) * c.get("n_phi", 1) * c.get("freqs", 1) <= 3_000_000:
            return c


# ---------------------------------------------------------------------------
# geometry, from the seed
# ---------------------------------------------------------------------------
def _wires(starts, ends, segments, radius):
    w = np.zeros(len(starts), acc.WIRE_DTYPE)
    w["tag"] = np.arange(1, len(starts) + 1)
    w["segments"], w["start"], w["end"], w["radius"] = segments, starts, ends, radius
    return w


def _array(case, rng):
    """Parallel wires along z, lengths 0.9-1.1 half waves at 14.2 MHz, spaced
    0.15-0.25 wavelengths; over ground their lower ends sit above z = 0."""
    lam, nw = C0 / F0, case["wires"]
    length = rng.uniform(0.9, 1.1, nw) * lam / 2
    x = np.concatenate([[0.0], np.cumsum(rng.uniform(0.15, 0.25, nw - 1) * lam)])
    lift = rng.uniform(0.3, 0.5) * lam if case.get("ground") else 0.0
    a, b = np.zeros((nw, 3)), np.zeros((nw, 3))
    a[:, 0] = b[:, 0] = x
    a[:, 2], b[:, 2] = lift - length / 2, lift + length / 2
    return _wires(a, b, case["segments"], 1e-3), [(min(2, nw), (case["segments"] + 1) // 2, 1.0)]


def _random_antenna(rng, counts):
    """Straight wires with random end points in a 20 m cube above z = 0,
    radius log-uniform 0.5-5 mm, no segment shorter than its diameter."""
    nw = len(counts)
    rad = np.exp(rng.uniform(math.log(0.5e-3), math.log(5e-3), nw))
    ends = rng.uniform([-10.0, -10.0, 0.0], [10.0, 10.0, 20.0], (2, nw, 3))
    while True:
        short = np.linalg.norm(ends[1] - ends[0], axis=1) < 2.0 * rad * counts
        if not short.any():
            return _wires(ends[0], ends[1], counts, rad)
        ends[:, short] = rng.uniform([-10.0, -10.0, 0.0], [10.0, 10.0, 20.0], (2, int(short.sum()), 3))


def _frequency(rng):
    return float(np.exp(rng.uniform(math.log(3e6), math.log(30e6))))


def _mesh(case, rng):
    """Square grid of cells of 0.05 wavelengths at z = 0.25 wavelengths, nodes
    jittered by 1 % of the pitch; the centre row edge is driven."""
    cells, lam = case["cells"], C0 / F0
    pitch, nn = 0.05 * lam, cells + 1
    grid = np.stack(np.meshgrid(np.arange(nn), np.arange(nn), indexing="ij"), axis=-1) * pitch
    node = np.full((nn, nn, 3), 0.25 * lam)
    node[..., :2] = grid + rng.uniform(-0.01, 0.01, (nn, nn, 2)) * pitch
    rows_a, rows_b = node[:-1].swapaxes(0, 1).reshape(-1, 3), node[1:].swapaxes(0, 1).reshape(-1, 3)
    cols_a, cols_b = node[:, :-1].reshape(-1, 3), node[:, 1:].reshape(-1, 3)
    centre = (nn // 2) * cells + cells // 2 + 1
    return _wires(np.concatenate([rows_a, cols_a]), np.concatenate([rows_b, cols_b]), 2, 1e-3), [(centre, 1, 1.0)]


def _jobs(case, seed):
    """The case's antennas as dicts: wires, sources, freqs, ground, rp,
    separate (each source a right-hand side of its own)."""
    rng = np.random.default_rng(seed)
    size = np.random.default_rng(case.get("antennas", case.get("requests", 0)))  # sizes are the case's, not the seed's
    job = {"ground": case.get("ground", 0), "rp": None, "separate": False}
    if case["kind"] == "serve":
        out = []
        for _ in range(case["requests"]):
            # total segments lognormal (median 150), 1-4 source positions,
            # half of the requests with a 5 degree pattern
            n = int(min(1200, max(11, round(float(np.exp(size.normal(math.log(150.0), 0.75)))))))
            nw = max(1, min(int(size.integers(1, 9)), n // 3))
            counts = np.maximum(3, np.round(n * size.dirichlet(np.ones(nw)))).astype(int) | 1
            src = {(1, (int(counts[0]) + 1) // 2): None}
            for _ in range(int(size.integers(0, 4))):
                t = int(size.integers(0, nw))
                src[(t + 1, int(size.integers(1, counts[t] + 1)))] = None
            rp = (19, 73, 0.0, 0.0, 5.0, 5.0) if size.random() < 0.5 else None
            out.append(dict(job, wires=_random_antenna(rng, counts), sources=[(t, s, 1.0) for t, s in src],
                            freqs=[_frequency(rng)], ground=int(size.integers(0, 2)), rp=rp, separate=True))
        return out
    if case.get("family") == "uneven":
        out = []
        for _ in range(case["antennas"]):
            w = _random_antenna(rng, 2 * size.integers(5, 51, int(size.integers(1, 9))) + 1)
            out.append(dict(job, wires=w, sources=[(1, (int(w["segments"][0]) + 1) // 2, 1.0)],
                            freqs=[_frequency(rng)], ground=int(size.integers(0, 2))))
        return out
    if case.get("family") == "mesh":
        w, src = _mesh(case, rng)
        return [dict(job, wires=w, sources=src, freqs=[F0], ground=1)]
    w, src = _array(case, rng)
    nf = case.get("freqs", 1)
    freqs = [F0] if nf == 1 else [13.0e6 + i * 2.5e6 / (nf - 1) for i in range(nf)]
    rp = None
    if case["kind"] == "solve":
        nt, nph = case["n_theta"], case["n_phi"]
        rp = (nt, nph, 0.0, 0.0, (90.0 if case["ground"] or nt == 91 else 180.0) / max(nt - 1, 1),
              360.0 / max(nph - 1, 1) if nph > 2 else 90.0)
    return [dict(job, wires=w, sources=src, freqs=freqs, rp=rp)]


def _antenna(j, plane_wave=None):
    return acc.Antenna(j["wires"], acc.sources_array(j["sources"] if plane_wave is None else []), j["freqs"],
                       j["ground"], j["rp"], separate_sources=j["separate"], plane_wave=plane_wave)


def _precision(case):
    return acc.PRECISION_MIXED if case["precision"] == "mixed" else acc.PRECISION_FP64


def _card(case):
    """EX 2 card: right elliptic, axial ratio 0.5, eta 20 degrees; directions
    over the sphere (off its poles, where wires along z receive nothing)."""
    nt, nph = case["n_theta"], case["n_phi"]
    return acc.plane_wave(2, 90.0 / nt, 0.0, 20.0, nt, nph, 180.0 / nt, 360.0 / nph, 0.5)


def _points(case):
    """(theta, phi) of a pattern call, phi outer."""
    nt, nph = case["n_theta"], case["n_phi"]
    th = np.arange(nt) * ((90.0 if case["ground"] else 180.0) / max(nt - 1, 1))
    ph = np.arange(nph) * (360.0 / max(nph - 1, 1) if nph > 2 else 90.0)
    return np.stack([np.tile(th, nph), np.repeat(ph, nt)], axis=1)


def _plane(case):
    """Points of a plane 0.3 wavelengths beside the wires."""
    lam = C0 / F0
    x = np.linspace(-0.5 * lam, 1.5 * lam, case["nx"])
    z = np.linspace(-0.6 * lam, 0.6 * lam, case["ny"])
    p = np.zeros((case["nx"], case["ny"], 3))
    p[..., 0], p[..., 1], p[..., 2] = x[:, None], 0.3 * lam, z[None, :]
    return p.reshape(-1, 3)


def _currents(seg, rng):
    """Standing-wave currents of plausible size: a half sine per wire with a
    random complex amplitude."""
    amp = rng.normal(0, 5e-3, seg["wire"].max() + 1) + 1j * rng.normal(0, 5e-3, seg["wire"].max() + 1)
    t = np.zeros(len(seg["wire"]))
    for q in range(seg["wire"].max() + 1):
        m = seg["wire"] == q
        t[m] = (np.arange(m.sum()) + 0.5) / m.sum()
    return amp[seg["wire"]] * np.sin(math.pi * t)


# ---------------------------------------------------------------------------
# the call and what it is given
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    jobs = _jobs(case, seed)
    st = {"kind": kind}
    if kind == "solve":
        st["batch"] = acc.HallenBatch([_antenna(j) for j in jobs], precision=_precision(case))
        st["pattern"] = jobs[0]["rp"] is not None
    elif kind == "receive":
        st["batch"] = acc.HallenBatch([_antenna(jobs[0], _card(case))], precision=acc.PRECISION_FP64)
    elif kind == "serve":
        st["server"] = acc.Server(precision=_precision(case), lanes=4, hbm_budget_bytes=8 << 30, max_batch=256)
        st["antennas"] = [_antenna(j) for j in jobs]
    else:
        j = jobs[0]
        seg = _segments(j["wires"])
        st["segments"] = acc.build_geometry(j["wires"])
        st["freq"], st["ground"] = j["freqs"][0], j["ground"]
        if kind == "call":
            st["rhs"], st["cos"] = _rhs(seg, j["sources"], 2.0 * math.pi * st["freq"] / C0)
            st["rhs"] = st["rhs"][:, 0]
            st["endpoints"], st["precision"] = seg["ends"], _precision(case)
        else:
            st["segments"] = acc.gpu_segments_from(st["segments"])
            st["currents"] = _currents(seg, np.random.default_rng(seed + 1))
            st["points"] = _plane(case) if kind == "near" else _points(case)
    return st


def run(st):
    kind = st["kind"]
    if kind == "solve":
        b = st["batch"]
        b.upload()
        if st["pattern"]:
            b.run_report()
            cur, feeds, pattern, status = b.read_report(pattern=False)
            return {"currents": cur, "feeds": feeds, "pattern": pattern, "status": status}
        b.run()
        cur, feeds, _, status, _ = b.read_raw(pattern=False)
        return {"currents": cur, "feeds": feeds, "status": status}
    if kind == "receive":
        b = st["batch"]
        b.upload()
        b.run()
        return {"receive": b.read_receive()}
    if kind == "serve":
        reqs = [st["server"].submit(a, copy_out=True) for a in st["antennas"]]
        for r in reqs:
            st["server"].wait(r)
        for r in reqs:
            r.release()
        return {"currents": np.concatenate([r.currents.reshape(-1) for r in reqs]),
                "feeds": np.concatenate([r.feeds for r in reqs]),
                "pattern": np.concatenate([r.pattern.reshape(-1, 6) for r in reqs if r.pattern is not None] +
                                          [np.zeros((0, 6))]),
                "status": np.concatenate([r.status for r in reqs])}
    if kind == "call":
        return {"x": acc.solve_hallen_gpu_resident(st["segments"], st["rhs"], st["cos"], st["endpoints"], [],
                                                   st["freq"], st["ground"], st["precision"])}
    if kind == "near":
        e, h = acc.near_field(st["segments"], st["currents"], st["freq"], st["points"])
        return {"e": e, "h": h}
    out, total = acc.compute_radiation_pattern(st["segments"], st["currents"], st["freq"], st["points"], st["ground"])
    return {"pattern": out, "total": total}


def _directions(case_ground, points):
    """Far-field directions of one pattern: the power integral's and the points'."""
    return (90 if case_ground else 180) * 360 + points


def work(case):
    kind = case["kind"]
    seg = case.get("wires", 1) * case.get("segments", 1)
    if kind == "near":
        pts = case["nx"] * case["ny"]
        return {"bytes": 72 * seg + 24 * pts + 192 * pts, "flops": 150 * seg * pts}
    if kind == "pattern":
        pts = case["n_theta"] * case["n_phi"]
        return {"bytes": 72 * seg + 48 * pts, "flops": 8 * seg * (1 + case["ground"]) * _directions(case["ground"], pts)}
    # per system: the fill's G(R) samples (60 operations each), the Hermitian
    # normal equations, their triangular factor, two substitutions per right-hand side
    nbytes = flops = 0

    def add(n, s, ground, rhs, systems, points, out=None):
        nonlocal nbytes, flops
        flops += systems * (60 * 8 * n * n * (1 + ground) + 4 * n * n * (n + 1) + 4 * s ** 3 / 3 + 8 * s * s * rhs +
                            rhs * (8 * n * _directions(ground, points) if points else 0))
        nbytes += 128 * n + systems * rhs * (out or 16 * n + 56 + 32 * points)

    if kind == "receive":
        add(seg, seg + 2 * case["wires"], 0, case["n_theta"] * case["n_phi"], case["freqs"], 0, out=24)
    elif kind == "call":
        add(seg, seg + case["wires"], case["ground"], 1, 1, 0)
    elif kind == "serve" or case["family"] == "uneven":
        for j in _jobs(case, 1):
            n = int(j["wires"]["segments"].sum())
            add(n, n + len(j["wires"]), j["ground"], len(j["sources"]) if j["separate"] else 1, 1,
                j["rp"][0] * j["rp"][1] if j["rp"] else 0)
    elif case["family"] == "mesh":
        edges = 2 * case["cells"] * (case["cells"] + 1)
        add(2 * edges, 3 * edges, 1, 1, 1, 0)
    else:
        add(seg, seg + case["wires"], case["ground"], 1, case["freqs"], case["n_theta"] * case["n_phi"])
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same results in 64 bits, from the equations
# ---------------------------------------------------------------------------
# Gauss-Legendre abscissae and weights, rounded to the digits the method is defined with
GL4 = (np.array([-0.861136311594953, -0.339981043584856, 0.339981043584856, 0.861136311594953]),
       np.array([0.347854845137454, 0.652145154862626, 0.652145154862626, 0.347854845137454]))
GL8 = (np.array([-0.960289856497536, -0.796666477413627, -0.525532409916329, -0.183434642495650,
                 0.183434642495650, 0.525532409916329, 0.796666477413627, 0.960289856497536]),
       np.array([0.101228536290376, 0.222381034453374, 0.313706645877887, 0.362683783378362,
                 0.362683783378362, 0.313706645877887, 0.222381034453374, 0.101228536290376]))
REG = 1e-8  # the normal equations' Tikhonov term


def _segments(w):
    """Segments of straight wires: midpoint, direction, length, radius, the
    wire of each and (first, last) segment of each wire."""
    cnt = w["segments"].astype(np.int64)
    first = np.concatenate([[0], np.cumsum(cnt)[:-1]])
    wire = np.repeat(np.arange(len(w)), cnt)
    i = np.arange(len(wire)) - first[wire]
    d = w["end"] - w["start"]
    length = np.linalg.norm(d, axis=1)
    t = (i / cnt[wire] + (i + 1.0) / cnt[wire]) * 0.5
    return {"mid": w["start"][wire] + d[wire] * t[:, None], "dir": (d / length[:, None])[wire],
            "len": (length / cnt)[wire], "rad": w["radius"][wire], "wire": wire, "s": (t - 0.5) * length[wire],
            "ends": np.stack([first, first + cnt - 1], axis=1)}


def _rhs(seg, sources, k, separate=False):
    """The Hallen right-hand sides (n, r) and cos(k s) of voltage sources; one
    source per wire at most unless they are separate."""
    y = np.zeros((len(seg["s"]), len(sources) if separate else 1), np.complex128)
    for q, (tag, s, v) in enumerate(sources):
        f = seg["ends"][tag - 1, 0] + s - 1
        on = seg["wire"] == tag - 1
        y[on, q if separate else 0] += -1j * RHS_SCALE * np.sin(k * np.abs(seg["s"][on] - seg["s"][f])) * v
    return y, np.cos(k * seg["s"])


def _constraints(w, seg):
    """Rows on the currents beside the integral equation: I = 0 at free wire
    ends, and I_a + sign I_b = 0 for every pair of wire ends that meet."""
    node, rows = {}, []
    for q in range(len(w)):
        for e, p in ((0, w["start"][q]), (1, w["end"][q])):
            node.setdefault(tuple(np.round(p / 1e-4).astype(np.int64)), []).append((int(seg["ends"][q, e]), e))
    for ends in node.values():
        if len(ends) == 1:
            rows.append((ends[0][0], -1, 0.0))
        for a in range(len(ends)):
            for b in range(a + 1, len(ends)):
                rows.append((ends[a][0], ends[b][0], 1.0 if ends[a][1] == ends[b][1] else -1.0))
    return rows


def _green(r, k):
    return torch.polar(1.0 / r, -k * r)


def _z_block(o, s, k, dev):
    """Z of one system: the 8-point rule over each source segment, the self
    term with its static part in closed form, PEC images added."""
    t = {q: torch.as_tensor(s[q], device=dev) for q in ("mid", "dir", "len", "rad")}
    n = len(s["len"])
    z = torch.empty((n, n), dtype=torch.complex128, device=dev)
    flip = torch.tensor([1.0, 1.0, -1.0], dtype=torch.float64, device=dev)
    half = t["len"] * 0.5
    for r0 in range(0, n, 2048):
        om, od = t["mid"][r0:r0 + 2048], t["dir"][r0:r0 + 2048]
        acc_ = 0
        for image in (False, True) if o["ground"] else (False,):
            sm, sd = (t["mid"] * flip, -t["dir"] * flip) if image else (t["mid"], t["dir"])
            total = 0
            for x, wt in zip(*GL8):
                p = sm + (x * half)[:, None] * sd
                r2 = sum((om[:, None, c] - p[None, :, c]) ** 2 for c in range(3))
                total = total + wt * _green(torch.sqrt(r2 + t["rad"] ** 2), k)
            total = total * half
            if not image:
                x4, w4 = (torch.as_tensor(v, device=dev) for v in GL4)
                r = torch.sqrt((x4[:, None] * half) ** 2 + t["rad"] ** 2)
                own = (w4[:, None] * (_green(r, k) - 1.0 / r)).sum(0) * half
                own = own + 2.0 * torch.log((half + torch.sqrt(half ** 2 + t["rad"] ** 2)) / t["rad"])
                i = torch.arange(len(om), device=dev)
                total[i, r0 + i] = own[r0:r0 + 2048]
            acc_ = acc_ + total * (od @ sd.T)
        z[r0:r0 + 2048] = acc_
    return z


def _solve(z, homog, wire, rows, y):
    """min |M x - y|^2 + REG |x|^2 with M = [Z | -homogeneous columns] over the
    constraint rows; Cholesky of the normal equations, refined with residuals
    formed from M.  homog: (n, h) columns of each wire's own rows."""
    dev, n, h = z.device, len(z), homog.shape[1]
    nw = int(wire.max()) + 1
    s = n + h * nw
    m = torch.zeros((n + len(rows), s), dtype=torch.complex128, device=dev)
    m[:n, :n] = z
    i, wi = torch.arange(n, device=dev), torch.as_tensor(wire, device=dev)
    for q in range(h):
        m[i, n + h * wi + q] = -torch.as_tensor(homog[:, q], device=dev).to(torch.complex128)
    r = np.array(rows)
    a, b = r[:, 0].astype(np.int64), r[:, 1].astype(np.int64)
    at = n + np.arange(len(rows))
    m[at, a] = 1.0
    two = b >= 0
    m[at[two], b[two]] = torch.as_tensor(r[two, 2], device=dev).to(torch.complex128)
    full = torch.zeros((len(m), y.shape[1]), dtype=torch.complex128, device=dev)
    full[:n] = torch.as_tensor(y, device=dev)
    aty = m.mH @ full
    g = m.mH @ m
    g.diagonal().add_(REG)
    low = torch.linalg.cholesky(g)
    del g
    x = torch.cholesky_solve(aty, low)
    for _ in range(4):
        x = x + torch.cholesky_solve(m.mH @ (full - m @ x) - REG * x, low)
    return x


def _far(seg, cur, k, pts, ground, dev):
    """(F_theta, F_phi) at (theta, phi) points in degrees."""
    th, ph = (torch.as_tensor(np.deg2rad(pts[:, c]), device=dev) for c in (0, 1))
    st, ct, sp, cp = torch.sin(th), torch.cos(th), torch.sin(ph), torch.cos(ph)
    rh = torch.stack([st * cp, st * sp, ct], 1)
    tv, pv = torch.stack([ct * cp, ct * sp, -st], 1), torch.stack([-sp, cp, 0 * sp], 1)
    flip = torch.tensor([1.0, 1.0, -1.0], dtype=torch.float64, device=dev)
    mid, d, il = (torch.as_tensor(v, device=dev) for v in (seg["mid"], seg["dir"], cur * seg["len"]))
    out = torch.zeros((2, len(th)), dtype=torch.complex128, device=dev)
    for p0 in range(0, len(th), 16384):
        q = slice(p0, p0 + 16384)
        for sm, sd in ((mid, d), (mid * flip, -d * flip))[: 2 if ground else 1]:
            wave = torch.polar(torch.ones((), dtype=torch.float64, device=dev), k * (rh[q] @ sm.T)) * il
            out[0, q] += (wave * (tv[q] @ sd.T)).sum(1)
            out[1, q] += (wave * (pv[q] @ sd.T)).sum(1)
    return out


def _pattern(seg, cur, k, pts, ground, dev):
    """Gains (total, theta, phi) in dBi, axial ratio, U_theta, U_phi at the
    points, and the total radiated power they are normalised by."""
    nt = 91 if ground else 181
    th = np.arange(1, nt) if ground else np.arange(1, nt - 1)
    grid = np.stack([np.repeat(th, 360), np.tile(np.arange(360), len(th))], 1).astype(np.float64)
    u = (_far(seg, cur, k, grid, ground, dev).abs() ** 2).sum(0)
    wt = np.where(grid[:, 0] == nt - 1, 0.5, 1.0) * np.sin(np.deg2rad(grid[:, 0])) * (math.pi / 180.0) ** 2
    total = float((u * torch.as_tensor(wt, device=dev)).sum())
    et, ep = _far(seg, cur, k, pts, ground, dev)
    ut, up = et.abs() ** 2, ep.abs() ** 2
    below = torch.as_tensor(pts[:, 0] > 90.0, device=dev) & bool(ground)
    cols = []
    for v in (ut + up, ut, up):
        g = v * (4.0 * math.pi / total if total > 0 else 0.0)
        g = torch.where(g > 1e-20, 10.0 * torch.log10(g.clamp_min(1e-300)), torch.full_like(g, -999.99))
        cols.append(torch.where(below, torch.full_like(g, -999.99), g))
    s0 = ut + up
    s3 = 2.0 * (et * ep.conj()).imag
    ar = torch.tan(0.5 * torch.asin((s3 / s0.clamp_min(1e-300)).clamp(-1.0, 1.0)))
    cols += [torch.where((s0 <= 1e-30) | below, 0 * ar, ar)] + [torch.where(below, 0 * v, v) for v in (ut, up)]
    return torch.stack(cols, 1).cpu().numpy(), total


def _rp_points(rp):
    nt, nph, t0, p0, dt, dp = rp
    return np.stack([np.tile(t0 + np.arange(nt) * dt, nph), np.repeat(p0 + np.arange(nph) * dp, nt)], 1)


def _exact_receive(case, j, dev):
    seg = _segments(j["wires"])
    _, nt, nph, th0, ph0, eta, dth, dph, ar = _card(case)
    t = np.deg2rad(np.repeat(th0 + np.arange(nt) * dth, nph))
    p = np.deg2rad(np.tile(ph0 + np.arange(nph) * dph, nt))
    rh = np.stack([np.sin(t) * np.cos(p), np.sin(t) * np.sin(p), np.cos(t)], 1)
    thv = np.stack([np.cos(t) * np.cos(p), np.cos(t) * np.sin(p), -np.sin(t)], 1)
    phv = np.stack([-np.sin(p), np.cos(p), 0 * p], 1)
    ce, se = math.cos(math.radians(eta)), math.sin(math.radians(eta))
    pol = ce * thv + se * phv + 1j * ar * (-se * thv + ce * phv)
    out = []
    for f in j["freqs"]:
        k = 2.0 * math.pi * f / C0
        e = (seg["dir"] @ pol.T) * np.exp(1j * k * (seg["mid"] @ rh.T))
        kern = np.sin(k * np.abs(seg["s"][:, None] - seg["s"][None, :])) * (seg["wire"][:, None] == seg["wire"][None, :])
        y = -1j * RHS_SCALE * ((kern * seg["len"]) @ e)
        homog = np.stack([np.cos(k * seg["s"]), np.sin(k * seg["s"])], 1)
        rows = [(int(v), -1, 0.0) for v in seg["ends"].reshape(-1)]
        x = _solve(_z_block(j, seg, k, dev), homog, seg["wire"], rows, y)
        peak = x[: len(seg["s"])].abs().amax(0).cpu().numpy()
        out.append(np.stack([np.rad2deg(t), np.rad2deg(p), 20.0 * np.log10(peak / peak.max())], 1))
    return {"receive": np.concatenate(out)}


def _exact_near(seg, cur, k, pts):
    r = pts[:, None, :] - seg["mid"]
    dist = np.linalg.norm(r, axis=2)
    rh, u = r / dist[..., None], seg["dir"]
    jkr = 1j * k * dist
    ph = np.exp(-jkr) * (cur * seg["len"])
    c = (rh * u).sum(2)
    rad = 2.0 * c / dist ** 2 * (1 + 1 / jkr)
    th = jkr / dist ** 2 * (1 + 1 / jkr - 1 / (k * dist) ** 2)
    pe = ph * ETA0 / (4.0 * math.pi)
    e = ((pe * rad)[..., None] * rh + (pe * th)[..., None] * (c[..., None] * rh - u)).sum(1)
    h = ((ph / (4.0 * math.pi) * jkr / dist ** 2 * (1 + 1 / jkr))[..., None] * np.cross(u, rh)).sum(1)
    return {"e": e, "h": h}


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    jobs = _jobs(case, seed)
    if kind == "solve" and len(jobs) > 1024:
        return None  # one dense 64-bit solve per antenna would take too long
    if kind == "receive":
        return _exact_receive(case, jobs[0], dev)
    if kind in ("near", "pattern"):
        j = jobs[0]
        seg, k = _segments(j["wires"]), 2.0 * math.pi * j["freqs"][0] / C0
        cur = _currents(seg, np.random.default_rng(seed + 1))
        if kind == "near":
            return _exact_near(seg, cur, k, _plane(case))
        pat, total = _pattern(seg, cur, k, _points(case), j["ground"], dev)
        return {"pattern": pat[:, :4], "total": total}
    currents, feeds, pattern = [], [], []
    for j in jobs:
        seg = _segments(j["wires"])
        rows = _constraints(j["wires"], seg)
        for f in j["freqs"]:
            k = 2.0 * math.pi * f / C0
            y, cosv = _rhs(seg, j["sources"], k, j["separate"])
            x = _solve(_z_block(j, seg, k, dev), cosv[:, None], seg["wire"], rows, y).cpu().numpy()
            if kind == "call":
                return {"x": x[:, 0]}
            n = len(seg["s"])
            for q in range(y.shape[1]):
                cur = x[:n, q]
                currents.append(cur)
                for tag, s, v in [j["sources"][q]] if j["separate"] else j["sources"]:
                    at = int(seg["ends"][tag - 1, 0]) + s - 1
                    zin = v / cur[at]
                    feeds.append([at, complex(v).real, complex(v).imag, cur[at].real, cur[at].imag, zin.real,
                                  zin.imag])
                if j["rp"]:
                    pattern.append(_pattern(seg, cur, k, _rp_points(j["rp"]), j["ground"], dev)[0])
    out = {"currents": np.concatenate(currents), "feeds": np.array(feeds), "status": None}
    if kind == "serve":
        out["pattern"] = np.concatenate(pattern + [np.zeros((0, 6))])
    elif jobs[0]["rp"] is not None:
        out["pattern"] = np.concatenate(pattern)[:, :4]
    return out
