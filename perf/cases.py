"""Performance cases: the calls a user of this framework makes, over the real range of sizes.

A case is a dict of plain values; ``kind`` says which call sequence it stands for:

  tti    a detector pool serving one transmission interval: its resident detectors (dictionaries
         full) get a few new pilots each (``append``, 0 for none) and detect a short block of
         data, all host buffers, one ``DetectorPool.run`` call
  frame  the reference CLI's frame: one ``NomaDetector`` (one or several users of a cell), reset,
         train on the pilots and detect the data, host arrays
  train  training of a large model and the snapshot of it that a user keeps
         (``train`` then ``get_state``)
  large  detection of a long recording on device buffers with a large trained model, in the
         exact form or a tensor-core form (``detect_device``)
  batch  many detectors of different sizes in one pool batch on device buffers: fresh training
         and detection of every detector, or detection alone (``run_prepared``)

Frames are synthetic: Gray-mapped QAM users behind a Rapp power amplifier (p = 2, 3 dB back-off),
a flat Rayleigh channel per cell and white noise.  ``exact`` evaluates the model in 64 bits.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import libapsm_b200 as L

# The algorithm's defaults that a case does not set (the reference's own).
DEFAULTS = {"windowSize": 20, "gaussianKernelVariance": 0.05, "eB": 0.001, "gaussianKernelWeight": 0.5,
            "dictionarySize": 685}
CLASSES = (4, 8, 16, 32)  # antennas of a pool's detectors


def listed() -> list[dict]:
    return [
        # the smallest call: one resident detector detects one short block (latency, launches)
        dict(name="tti_detect", kind="tti", detectors=1, antennas=8, dictionary=2000, append=0, symbols=500,
             window=80, variance=0.05, eB=0.001, form="balanced"),
        # one served interval: 16 detectors of mixed antenna counts append pilots and detect
        dict(name="tti_append", kind="tti", detectors=16, antennas=0, dictionary=2000, append=64, symbols=4000,
             window=80, variance=0.05, eB=0.001, form="balanced"),
        # a single QPSK user, 8 antennas, 600 pilots, 1800 data symbols
        dict(name="frame_qpsk", kind="frame", otype="APSM", antennas=8, users=1, pilots=600, symbols=1800, bits=2,
             window=80, variance=0.5, eB=0.01, dictionary=685),
        # all eight 16QAM users of a cell, 16 antennas, 1000 pilots, 8000 data symbols
        dict(name="frame_users", kind="frame", otype="APSM", antennas=16, users=8, pilots=1000, symbols=8000, bits=4,
             window=80, variance=0.5, eB=0.01, dictionary=1000),
        # the testbed recording's size with the algorithm's defaults: 16 antennas, six users,
        # 685 pilots, 3840 symbols, window 20 (odd sizes)
        dict(name="frame_testbed", kind="frame", otype="APSM", antennas=16, users=6, pilots=685, symbols=3840, bits=2,
             window=20, variance=0.05, eB=0.001, dictionary=685),
        # the linear least-squares detector on the eight-user frame
        dict(name="frame_lls", kind="frame", otype="LLS", antennas=16, users=8, pilots=1000, symbols=8000, bits=4,
             window=0, variance=0.0, eB=0.0, dictionary=0),
        # a large model: 64 antennas, 16 users, 8192 pilots into a dictionary of 8192
        dict(name="train_large", kind="train", antennas=64, users=16, pilots=8192, window=80, variance=0.5, eB=0.01,
             dictionary=8192, bits=4),
        # 65536 symbols with that model in the exact FP32 form and in two tensor-core forms
        dict(name="large_exact", kind="large", antennas=64, users=16, dictionary=8192, symbols=65536,
             form="balanced", window=80, variance=0.05, eB=0.01, bits=4),
        dict(name="large_tf32x3", kind="large", antennas=64, users=16, dictionary=8192, symbols=65536,
             form="gram_tf32x3", window=80, variance=0.05, eB=0.01, bits=4),
        dict(name="large_bf16", kind="large", antennas=64, users=16, dictionary=8192, symbols=65536,
             form="gram_bf16", window=80, variance=0.5, eB=0.01, bits=4),
        # 512 detectors (4 to 32 antennas, 200 to 2000 pilots, 1000 to 16000 symbols), fresh
        # training and tensor-core detection of each
        dict(name="batch_frames", kind="batch", detectors=512, train=True, form="gram_tf32x3", pilots=2000,
             symbols=16000, window=80, variance=0.05, eB=0.001, dictionary=2000, mix=0),
        # the same detectors, trained before, detecting in the FP32 form
        dict(name="batch_detect", kind="batch", detectors=512, train=False, form="balanced", pilots=2000,
             symbols=16000, window=80, variance=0.05, eB=0.001, dictionary=2000, mix=0),
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(("tti", "frame", "frame", "train", "large", "batch"))
    if kind == "tti":
        return dict(kind=kind, detectors=_log_int(rng, 1, 24), antennas=rng.choice((0, 3, 4, 8, 12, 16, 32)),
                    dictionary=_log_int(rng, 200, 2000), append=rng.choice((0, rng.randint(16, 64))),
                    symbols=_log_int(rng, 500, 4000), window=rng.choice((20, 40, 80)),
                    variance=rng.choice((0.05, 0.5)), eB=rng.choice((0.001, 0.01)),
                    form=rng.choice(("balanced", "balanced", "gram_bf16")))
    if kind == "frame":
        pilots = _log_int(rng, 64, 2000)
        return dict(kind=kind, otype=rng.choice(("APSM", "APSM", "APSM", "LLS")), antennas=rng.randint(2, 32),
                    users=rng.choice((1, 2, 6, 8)), pilots=pilots, symbols=_log_int(rng, 200, 16000),
                    bits=rng.choice((2, 4)), window=rng.choice((20, 40, 80, 100)), variance=rng.choice((0.05, 0.5)),
                    eB=rng.choice((0.001, 0.01)), dictionary=max(300, rng.choice((pilots, pilots * 3 // 4))))
    if kind == "train":
        pilots = _log_int(rng, 1000, 6000)
        return dict(kind=kind, antennas=rng.choice((8, 16, 31, 64)), users=rng.randint(1, 16), pilots=pilots,
                    window=rng.choice((40, 80)), variance=rng.choice((0.05, 0.5)), eB=rng.choice((0.001, 0.01)),
                    dictionary=pilots, bits=4)
    if kind == "large":
        return dict(kind=kind, antennas=rng.choice((8, 16, 24, 32, 64)), users=rng.randint(1, 16),
                    dictionary=_log_int(rng, 500, 4000), symbols=_log_int(rng, 5000, 65536),
                    form=rng.choice(("balanced", "gram_bf16", "gram_bf16x3", "gram_tf32", "gram_tf32x3")), window=80,
                    variance=rng.choice((0.05, 0.5)), eB=0.01, bits=4)
    return dict(kind=kind, detectors=_log_int(rng, 8, 300), train=rng.random() < 0.6,
                form=rng.choice(("balanced", "gram_tf32x3", "gram_tf32x3", "gram_bf16x3")),
                pilots=_log_int(rng, 300, 2000), symbols=_log_int(rng, 1500, 16000),
                window=rng.choice((20, 40, 80)), variance=rng.choice((0.05, 0.5)), eB=rng.choice((0.001, 0.01)),
                dictionary=2000, mix=rng.randint(1, 1000))


# ------------------------------------------------------------------ sizes --

def _sizes(case: dict) -> list[tuple[int, int, int]]:
    """(antennas, pilots, symbols) of every detector of a tti or batch case."""
    if case["kind"] == "tti":
        return [(case["antennas"] or CLASSES[i % 4], case["dictionary"],
                 case["symbols"] if case["detectors"] == 1 else max(64, case["symbols"] * (i + 2) // (case["detectors"] + 1)))
                for i in range(case["detectors"])]
    rng = random.Random(7919 * case["mix"] + case["detectors"])
    return [(rng.choice(CLASSES), rng.randint(min(200, case["pilots"]), case["pilots"]),
             rng.randint(min(1000, case["symbols"]), case["symbols"])) for _ in range(case["detectors"])]


def _append(case: dict, i: int) -> int:
    """Pilots that detector i of a tti case appends."""
    return max(1, case["append"] - 3 * (i % 16)) if case["append"] else 0


# ----------------------------------------------------------------- inputs --

def _frame(gen: torch.Generator, users: int, antennas: int, length: int, bits: int, snr_db: float):
    """Received samples (antennas, length) and sent symbols (users, length) on the GPU, complex64."""
    dev = gen.device
    side = 1 << (bits // 2)
    scale = math.sqrt(3.0 / (2.0 * (side * side - 1)))
    grid = torch.randint(0, side, (2, users, length), generator=gen, device=dev).double() * 2 - (side - 1)
    tx = torch.complex(grid[0], grid[1]) * scale
    drive = tx * 10.0 ** (-3.0 / 20.0)
    sent = drive / (1.0 + drive.abs() ** 4) ** 0.25
    h = torch.randn((antennas, users), generator=gen, device=dev, dtype=torch.complex128)
    clean = h @ sent
    noise = torch.randn((antennas, length), generator=gen, device=dev, dtype=torch.complex128)
    power = clean.abs().square().mean() * 10.0 ** (-snr_db / 10.0)
    rx = clean + noise * power.sqrt()
    return rx.to(torch.complex64), tx.to(torch.complex64)


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(1_000_003 * (int(seed) + 1))


def _cells(case: dict, seed: int):
    """Per detector of a tti or batch case: rx and tx of its pilots, of the appended pilots, and its data."""
    gen = _generator(seed)
    out = []
    for i, (n, p, s) in enumerate(_sizes(case)):
        extra = _append(case, i) if case["kind"] == "tti" else 0
        rx, tx = _frame(gen, 4, n, p + extra + s, 2 if i % 2 else 4, 10.0 + 15.0 * ((i * 37) % 16) / 15.0)
        out.append((rx[:, :p].contiguous(), tx[0, :p].contiguous(), rx[:, p:p + extra].contiguous(),
                    tx[0, p:p + extra].contiguous(), rx[:, p + extra:].contiguous()))
    return out


def _cell(case: dict, seed: int):
    """rx, tx of the pilots and the data rx of a frame, train or large case."""
    pilots = case.get("pilots", case["dictionary"])
    rx, tx = _frame(_generator(seed), case["users"], case["antennas"], pilots + case.get("symbols", 0), case["bits"],
                    20.0 if case["kind"] == "frame" else 15.0)
    return rx[:, :pilots].contiguous(), tx[:, :pilots].contiguous(), rx[:, pilots:].contiguous()


def _config(case: dict) -> dict:
    if case.get("otype") == "LLS":
        return {"otype": "LLS"}
    return {"otype": "APSM", "windowSize": case["window"], "gaussianKernelVariance": case["variance"], "eB": case["eB"],
            "dictionarySize": case["dictionary"], "detectVersion": case.get("form", "balanced")}


# ----------------------------------------------------------- prepare, run --

def prepare(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("tti", "batch"):
        pool = L.DetectorPool(_config(case))
        cells = _cells(case, seed)
        ids = [pool.add(c[0].shape[0]) for c in cells]
        training = [L.PoolJob(d, c[0], c[1], fresh=True) for d, c in zip(ids, cells)]
        if kind == "batch":
            total = sum(c[4].shape[1] for c in cells)
            est = torch.zeros(total, dtype=torch.complex64, device="cuda")
            parts = torch.split(est, [c[4].shape[1] for c in cells])
            detection = [L.PoolJob(d, c[4], est=e) for d, c, e in zip(ids, cells, parts)]
            torch.cuda.synchronize()
            if not case["train"]:
                pool.run_device(training)
                pool.wait()
                training = []
            return {"kind": kind, "pool": pool, "cells": cells, "est": est,
                    "jobs": pool.prepare(training + detection, device=True)}
        torch.cuda.synchronize()
        pool.run_device(training)
        pool.wait()
        jobs = [L.PoolJob(d, c[2].cpu().numpy(), c[3].cpu().numpy()) for d, c in zip(ids, cells) if case["append"]]
        jobs += [L.PoolJob(d, c[4].cpu().numpy()) for d, c in zip(ids, cells)]
        return {"kind": kind, "pool": pool, "jobs": jobs}
    det = L.NomaDetectorFactory.build(_config(case), case["antennas"], num_users=case["users"])
    rx, tx, data = _cell(case, seed)
    state = {"kind": kind, "det": det}
    if kind == "large":
        torch.cuda.synchronize()
        det.train_device(rx, tx)
        det.synchronize()
        state.update(data=data, est=torch.zeros((case["users"], case["symbols"]), dtype=torch.complex64, device="cuda"))
        return state
    state.update(rx=rx.cpu().numpy(), tx=tx.cpu().numpy(), data=data.cpu().numpy())
    return state


def run(state):
    kind = state["kind"]
    if kind == "tti":
        return [e for e in state["pool"].run(state["jobs"]) if e is not None]
    if kind == "batch":
        state["pool"].run_prepared(state["jobs"], mode=1)
        return state["est"]
    det = state["det"]
    if kind == "large":
        det.detect_device(state["data"], state["est"])
        return state["est"]
    det.reset_state()
    det.train(state["rx"], state["tx"])
    if kind == "train":
        return det.get_state()
    return det.detect(state["data"])[0]


# ------------------------------------------------------------------- work --

def _train_work(pilots: int, before: int, antennas: int, users: int, window: int, capacity: int) -> float:
    """Operations of one training call: each distinct kernel value once (pair form: one complex
    product and three exponentials per two samples), and per step and user the projection of the
    window, its rows' update by the window kernel and the new rows' sums over the dictionary."""
    flops = 0.0
    for t in range(pilots):
        seen = min(before + t + 1, capacity)
        w = min(window, seen)
        flops += seen * (8.0 * antennas + 3.0) + users * (8.0 * w * w + 8.0 * seen + 8.0 * w)
    return flops


def _detect_work(symbols: int, entries: int, antennas: int, users: int) -> float:
    return float(symbols) * (entries * (8.0 * antennas + 3.0 + 8.0 * users) + 8.0 * antennas * users)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("tti", "batch"):
        nbytes = flops = 0.0
        for i, (n, p, s) in enumerate(_sizes(case)):
            capacity = case["dictionary"]
            new = _append(case, i) if kind == "tti" else (p if case["train"] else 0)
            entries = min(p, capacity)
            # samples and targets in, estimates out; the dictionary (samples, coefficients) read or written
            nbytes += 8.0 * (n + 1) * (new + s) + 8.0 * (n + 1) * entries
            flops += _train_work(new, p if kind == "tti" else 0, n, 1, case["window"], capacity)
            flops += _detect_work(s, entries, n, 1)
        return {"bytes": nbytes, "flops": flops}
    n, u, s = case["antennas"], case["users"], case.get("symbols", 0)
    if case.get("otype") == "LLS":
        p = case["pilots"]
        return {"bytes": 8.0 * (n + u) * (p + s),
                "flops": 2.0 * 2 * p * 2 * n * (2 * n + u) + 2.0 * (2 * n) ** 3 / 3 + 8.0 * s * n * u}
    if kind == "large":
        m = case["dictionary"]
        return {"bytes": 8.0 * (n + u) * (s + m), "flops": _detect_work(s, m, n, u)}
    p, capacity = case["pilots"], case["dictionary"]
    m = min(p, capacity)
    return {"bytes": 8.0 * (n + u) * (p + s) + 8.0 * (n + u) * m,
            "flops": _train_work(p, 0, n, u, case["window"], capacity) + _detect_work(s, m, n, u)}


# ------------------------------------------------------------------ exact --

def _rows(rx: torch.Tensor) -> torch.Tensor:
    """Real rows of complex samples (antennas, n): [Re; Im] and [Im; -Re] of each, float64 (2n, 2 antennas)."""
    y = rx.to(torch.complex128).transpose(-1, -2)
    even = torch.cat([y.real, y.imag], -1)
    odd = torch.cat([y.imag, -y.real], -1)
    return torch.stack([even, odd], -2).flatten(-3, -2)


def _targets(tx: torch.Tensor) -> torch.Tensor:
    """(users, n) complex -> (users, 2n) float64, real and imaginary parts in turn."""
    return torch.view_as_real(tx.to(torch.complex128)).flatten(-2)


def _kernel(x: torch.Tensor, z: torch.Tensor, ew: float, wg: float) -> torch.Tensor:
    d2 = x.square().sum(-1)[..., :, None] + z.square().sum(-1)[..., None, :] - 2.0 * x @ z.transpose(-1, -2)
    return d2.clamp_(min=0.0).mul_(ew).exp_().mul_(wg)


def _sweep(x, y, lengths, window: int, capacity: int, eb: float, ew: float, wg: float, calls):
    """The training sweep of a batch of models in 64 bits.  x (B, R, D) rows, y (B, U, R) targets,
    lengths (B,) rows in use, calls: end row of each training call.  Returns a (B, U, R), w (B, U, D)."""
    b, r, _ = x.shape
    wl, cap, q2 = 1.0 - wg, 2 * capacity, 2 * window
    k = _kernel(x, x, ew, wg)
    norms = wl * x.square().sum(-1) + wg
    a = torch.zeros_like(y)
    w = torch.zeros((b, y.shape[1], x.shape[2]), dtype=torch.float64, device=x.device)
    start = 0
    for end in calls:
        for hi in range(start + 2, end + 1, 2):
            lo, w0 = max(0, hi - cap), max(0, hi - min(q2, cap))
            f = wl * w @ x[:, w0:hi].transpose(1, 2) + a[:, :, lo:hi] @ k[:, lo:hi, w0:hi]
            e = y[:, :, w0:hi] - f
            c = e.sign() * (e.abs() - eb).clamp_(min=0.0) / (hi - w0) / norms[:, None, w0:hi]
            if lengths is not None:
                c = torch.where((lengths >= hi)[:, None, None], c, 0.0)
            a[:, :, w0:hi] += c
            w += c @ x[:, w0:hi]
        start = end
    return a, w


def _soft(z, x, a, w, ew: float, wg: float) -> torch.Tensor:
    """Soft outputs of data rows z (S2, D) with models a (U, M) over rows x (M, D), w (U, D): (U, S) complex128."""
    out = []
    step = max(2, (1 << 27) // max(1, x.shape[0]) // 2 * 2)
    for s in range(0, z.shape[0], step):
        part = z[s:s + step]
        out.append((1.0 - wg) * w @ part.T + a @ _kernel(x, part, ew, wg))
    f = torch.cat(out, 1)
    return torch.complex(f[:, 0::2], f[:, 1::2])


def _exact_cells(case: dict, seed: int):
    cells = _cells(case, seed)
    wg, window, capacity = DEFAULTS["gaussianKernelWeight"], case["window"], case["dictionary"]
    eb = float(np.float32(case["eB"]))
    out: list = [None] * len(cells)
    order = sorted(range(len(cells)), key=lambda i: (cells[i][0].shape[0], cells[i][0].shape[1]))
    while order:
        n = cells[order[0]][0].shape[0]
        group = [i for i in order if cells[i][0].shape[0] == n]
        group = group[-64:]
        order = [i for i in order if i not in set(group)]
        ew = -0.5 / (float(np.float32(case["variance"])) * n * n)
        rows = [_rows(torch.cat([cells[i][0], cells[i][2]], 1)) for i in group]
        tx = [_targets(torch.cat([cells[i][1], cells[i][3]])[None]) for i in group]
        most = max(v.shape[0] for v in rows)
        x = torch.stack([torch.nn.functional.pad(v, (0, 0, 0, most - v.shape[0])) for v in rows])
        y = torch.stack([torch.nn.functional.pad(v, (0, most - v.shape[1])) for v in tx])
        lengths = torch.tensor([v.shape[0] for v in rows], device=x.device)
        calls = [most]
        if case["kind"] == "tti" and case["append"]:
            calls = [2 * case["dictionary"], most]
        a, w = _sweep(x, y, lengths, window, capacity, eb, ew, wg, calls)
        for j, i in enumerate(group):
            end = rows[j].shape[0]
            lo = max(0, end - 2 * capacity)
            out[i] = _soft(_rows(cells[i][4]), x[j, lo:end], a[j, :, lo:end], w[j], ew, wg)[0]
    return torch.cat(out) if case["kind"] == "batch" else [v.cpu().numpy() for v in out]


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("tti", "batch"):
        return _exact_cells(case, seed)
    rx, tx, data = _cell(case, seed)
    x, y = _rows(rx), _targets(tx)
    if case.get("otype") == "LLS":
        w = torch.linalg.lstsq(x, y.T).solution.T
        f = w @ _rows(data).T
        f = torch.complex(f[:, 0::2], f[:, 1::2]).cpu().numpy()
        return f[0] if case["users"] == 1 else f
    wg, capacity = DEFAULTS["gaussianKernelWeight"], case["dictionary"]
    ew = -0.5 / (float(np.float32(case["variance"])) * case["antennas"] ** 2)
    a, w = _sweep(x[None], y[None], None, case["window"], capacity, float(np.float32(case["eB"])), ew, wg, [x.shape[0]])
    lo = max(0, x.shape[0] - 2 * capacity)
    if kind == "train":
        return {"dictionary": x[lo:].cpu().numpy(), "a": a[0, :, lo:].cpu().numpy(), "w": w[0].cpu().numpy()}
    f = _soft(_rows(data), x[lo:], a[0, :, lo:], w[0], ew, wg)
    if kind == "large":
        return f
    f = f.cpu().numpy()
    return f[0] if case["users"] == 1 else f
