"""Performance cases of the FRU hot path: what programs built on the library
have it do, from one Dormand-Prince attempt of a 250-FRU cell to ensembles of
full-size cells, each through the public entry points.

Kinds of case:
  attempt   The five FRU stages of one Dormand-Prince attempt after a
            rollback (send_resume_state, then distrib_simFRU over the
            tableau's five intervals), and the per-FRU properties a program
            writes (Cell.resume, Cell.stage, gw_download_range).
  cell      One cell from a host-held state: Cell.upload, Cell.run over a few
            output steps with all traces, Cell.download.
  cells     Many cells from host-held states: upload, one concurrent run
            (streams, lockstep batch, device integrator or persistent
            kernel), the final FRU properties of every cell.
  serve     A Server taking a burst of requests that start from rest.

Synthetic states: `rest` is the rest state with a little scatter; `peak` and
`late` follow the distributions of the bench cell's FRUs at 30 ms (release at
its peak) and at 110 ms (plateau, most RyRs adapted) of a paced beat.
"""
import numpy as np

import greenstein2002_gb300 as G

# ---- the cases --------------------------------------------------------------


def listed():
    return [
        # the smallest configuration (250 FRUs, FP64): latency of a stage call
        {"name": "attempt_250_fp64", "kind": "attempt", "nfru": 250, "precision": "fp64", "phase": "peak", "step": 0.1},
        # a serving-size cell in mixed precision, odd FRU count, plateau
        {"name": "attempt_1251_mixed", "kind": "attempt", "nfru": 1251, "precision": "mixed", "phase": "late",
         "step": 0.1},
        # a full-size cell at the peak of release, both precisions
        {"name": "attempt_12500_fp64", "kind": "attempt", "nfru": 12500, "precision": "fp64", "phase": "peak",
         "step": 0.1},
        {"name": "attempt_12500_mixed", "kind": "attempt", "nfru": 12500, "precision": "mixed", "phase": "peak",
         "step": 0.1},
        # diastole: few substeps per stage, most of a paced cycle's stages; ragged count
        {"name": "attempt_12497_fp64_rest", "kind": "attempt", "nfru": 12497, "precision": "fp64", "phase": "rest",
         "step": 0.1},
        # whole calls on one cell: the plain method's 250-FRU cell, the full-size cell, and a
        # voltage clamp of a mid-size cell in mixed precision
        {"name": "cell_250_fp64", "kind": "cell", "nfru": 250, "precision": "fp64", "phase": "peak", "ms": 3,
         "clamp": False},
        {"name": "cell_12500_fp64", "kind": "cell", "nfru": 12500, "precision": "fp64", "phase": "late", "ms": 4,
         "clamp": False},
        {"name": "cell_5000_mixed_clamp", "kind": "cell", "nfru": 5000, "precision": "mixed", "phase": "rest", "ms": 12,
         "clamp": True},
        # the ensemble throughput runs: 16 full-size cells, one stream each, packed launches
        {"name": "ensemble_16_fp64", "kind": "cells", "cells": 16, "nfru": 12500, "uneven": False, "precision": "fp64",
         "phase": "peak", "ms": 2, "mode": "streams", "packed": 4},
        {"name": "ensemble_16_mixed", "kind": "cells", "cells": 16, "nfru": 12500, "uneven": False,
         "precision": "mixed", "phase": "peak", "ms": 10, "mode": "streams", "packed": 4},
        # uneven cells with their own pacing, PCa and GKr in one persistent launch
        {"name": "batch_24_mixed", "kind": "cells", "cells": 24, "nfru": 12500, "uneven": True, "precision": "mixed",
         "phase": "late", "ms": 10, "mode": "persistent", "packed": 0},
        # serving: a burst of short requests of mixed sizes and protocols from rest
        {"name": "serve_12_mixed", "kind": "serve", "requests": 12, "nfru": 5000, "precision": "mixed", "ms": 12},
    ]


def _log(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choice(["attempt", "attempt", "attempt", "cell", "cell", "cells", "cells", "serve"])
    precision = rng.choice(["fp64", "mixed"])
    phase = rng.choice(["peak", "late", "rest"])
    if kind == "attempt":
        return {"kind": kind, "nfru": _log(rng, 33, 12500), "precision": precision, "phase": phase,
                "step": round(rng.uniform(0.02, 0.1), 4)}
    if kind == "cell":
        return {"kind": kind, "nfru": _log(rng, 125, 12500), "precision": precision, "phase": phase,
                "ms": rng.randint(1, 4), "clamp": rng.random() < 0.25}
    if kind == "cells":
        return {"kind": kind, "cells": _log(rng, 2, 16), "nfru": _log(rng, 250, 12500), "uneven": rng.random() < 0.5,
                "precision": precision, "phase": phase, "ms": rng.randint(1, 3),
                "mode": rng.choice(["streams", "lockstep", "device", "persistent"]), "packed": rng.choice([0, 0, 4])}
    return {"kind": kind, "requests": _log(rng, 2, 12), "nfru": _log(rng, 500, 5000), "precision": precision,
            "ms": rng.randint(2, 6)}


# ---- states -------------------------------------------------------------------
NODES = (0.0, 1.0 / 5.0, 3.0 / 10.0, 3.0 / 5.0, 2.0 / 3.0, 1.0)  # Dormand-Prince 5(4), rk_pd54m.c
# LCC state 1..12 probabilities by phase
_LCC = {
    "peak": (.002, .031, .125, .259, .192, .0856, 0, .0002, .0106, .077, .217, .0006),
    "late": (.0005, .005, .030, .083, .103, .046, 0, .0002, .012, .130, .590, .0003),
    "rest": (.97, .024, .002, 0, 0, 0, .004, 0, 0, 0, 0, 0),
}
# RyR state 1..8 probabilities of a releasing and of a quiet cleft
_RYR = {
    "peak": ((.10, 0, .03, .50, 0, 0, .025, .345), (.95, 0, 0, 0, 0, 0, 0, .05)),
    "late": ((.15, 0, .02, .30, 0, 0, 0, .53), (.27, 0, 0, 0, 0, 0, 0, .73)),
    "rest": ((.90, 0, 0, 0, .08, .02, 0, 0), (.985, 0, 0, 0, .015, 0, 0, 0)),
}
_RELEASING = {"peak": 0.5, "late": 0.04, "rest": 0.02}
_VDI2 = {"peak": 0.91, "late": 0.70, "rest": 0.99}
_CL2 = {"peak": 0.06, "late": 0.006, "rest": 0.003}
# (V, Cai, CaNSR) and their slopes per ms during an attempt
_DEP = {"peak": ((2.7, 3.57e-4, 0.480), (0.5, 2e-6, -1e-3)), "late": ((9.2, 4.61e-4, 0.3725), (-0.2, -1e-6, 1e-4)),
        "rest": ((-95.0, 1.2e-4, 0.70), (0.05, 1e-9, 0.0))}
_T0 = {"peak": 30.0, "late": 110.0, "rest": 0.0}
# the 37 global states of the bench cell at the phase's time (V, Nai, Ki, Cai, CaNSR, ... of indices.h)
_GLOBAL = {
    "peak": (2.69532, 0.996105, 1.20649e-07, 0.00222175, 10.0019, 155.464, 0.000356873, 0.480188, 0.0149685,
              0.135433, 0.975199, 1.53455e-05, 0.000469317, 0.00527984, 0.0255316, 0.0506479, 4.21036e-09,
              1.45018e-06, 0.000267499, 0.0264254, 0.891362, 0, 4.16265e-08, 1.24176e-05, 0.00162546, 0.077376,
              -3.87198e-09, 1.15674e-06, -1.13294e-06, 0.000218973, 0.920767, 6.13368, 0.543982, 0.264352,
              0.0407713, 0.0151344, 0.13576),
    "late": (9.20662, 0.998089, 4.10958e-08, 0, 9.99595, 155.464, 0.000461151, 0.372541, 0.0546471, 0.322029,
              0.985286, 2.28701e-08, 1.24915e-06, 2.55845e-05, 0.000232882, 0.000794866, 3.78453e-10,
              2.64702e-07, 9.38291e-05, 0.0175123, 0.981339, 0, 2.93133e-10, 1.97095e-07, 4.93245e-05,
              0.00462937, -2.08013e-09, 1.13263e-06, -1.16977e-06, 0.000127529, 0.995194, 6.22659, 0.225244,
              0.183769, 0.0278954, 0.026417, 0.536674),
}
# FRU substeps per FRU and simulated ms, for work(): of an attempt from the phase's state (counted with
# exact()), and of a run (the mean over the first 200 ms of plateau of the bench cell)
_SUBSTEPS = {"peak": 880.0, "late": 165.0, "rest": 165.0}
_SUBSTEPS_RUN = 267.0
_OPS_PER_SUBSTEP = 700.0  # additions, multiplications, divisions, exponentials and comparisons of one FRU substep


def _pick(rng, p, shape):
    c = np.cumsum(np.asarray(p) / np.sum(p))
    return np.minimum(np.searchsorted(c, rng.random(shape), side="right"), len(p) - 1).astype(np.int32) + 1


def _frus(n, phase, rng):
    """A cell's FRUs in the layout of Cell.upload."""
    rel = rng.random((n, 4)) < _RELEASING[phase]
    hot, cold = _RYR[phase]
    ryr = np.where(rel[:, :, None], _pick(rng, hot, (n, 4, 5)), _pick(rng, cold, (n, 4, 5)))
    ltype = np.empty((n, 4, 2), np.int32)
    ltype[:, :, 0] = _pick(rng, _LCC[phase], (n, 4))
    ltype[:, :, 1] = 1 + (rng.random((n, 4)) < _VDI2[phase])
    ito2 = (1 + (rng.random((n, 4)) < _CL2[phase])).astype(np.int32)
    nopen = np.isin(ryr, (3, 4, 7)).sum(2)
    lcc = (ltype[:, :, 0] % 6 == 0) & (ltype[:, :, 1] == 2)
    frus = np.empty((n, 5))
    noise = np.exp(0.1 * rng.standard_normal((n, 4)))
    if phase == "rest":
        frus[:, 0] = 0.7 * np.exp(0.01 * rng.standard_normal(n))
        frus[:, 1:] = 0.12e-3 * noise
    else:
        base = 0.36e-3 if phase == "peak" else 0.46e-3
        near = np.roll(nopen, 1, 1) + np.roll(nopen, -1, 1)
        frus[:, 0] = np.clip((0.505 if phase == "peak" else 0.365) - 0.012 * nopen.sum(1) +
                             0.012 * rng.standard_normal(n), 0.24, 0.52)
        frus[:, 1:] = base * noise + (0.0052 * nopen + 0.0006 * near + 0.004 * lcc) * noise
    return {"frus": frus, "ltype": ltype, "ryr": np.ascontiguousarray(ryr, dtype=np.int32), "ito2": ito2,
            "mti": rng.integers(0, 625, n).astype(np.int32),
            "mt": rng.integers(0, 1 << 32, (n, 624), dtype=np.uint32)}


def _global_state(phase):
    if phase == "rest":
        c = G.Cell(8)
        state = c.init_rest()
        c.close()
        return state
    return np.array(_GLOBAL[phase])


def _sizes(n, nfru, uneven):
    """FRU counts of a case's cells or requests: the case's own, whatever the seed."""
    if not uneven:
        return [nfru] * n
    div = np.random.default_rng([n, nfru]).choice([1, 2, 4, 10], n, p=[.15, .15, .35, .35])
    return [max(1, nfru // int(d)) for d in div]


def _attempt_nodes(case):
    t0, h = _T0[case["phase"]], case["step"]
    dep, slope = (np.array(a) for a in _DEP[case["phase"]])
    return [(t0 + h * a, t0 + h * b, dep, dep + h * b * slope) for a, b in zip(NODES[:-1], NODES[1:])]


def _settings(case, rng, many):
    if case.get("clamp"):
        return G.settings(vclamp_flag=1, vclamp_hold=-100.0, vclamp_set=float(rng.uniform(-10.0, 10.0)),
                          vclamp_duration=200.0, vclamp_shift=_T0[case["phase"]] + 1.0, vclamp_period=100000.0)
    if many and case["uneven"]:
        return G.settings(period=float(rng.uniform(400.0, 2000.0)), scale_GKr=float(np.exp(rng.normal(0.0, 0.2))))
    return G.settings(shift=1.0 if case["phase"] == "rest" else 10.0)


def prepare(case, seed):
    rng = np.random.default_rng([int(seed), 2002])
    kind = case["kind"]
    if kind == "attempt":
        cell = G.Cell(case["nfru"], precision=case["precision"])
        cell.upload(_frus(case["nfru"], case["phase"], rng))
        cell.save()
        return {"case": case, "cell": cell, "nodes": _attempt_nodes(case)}
    if kind == "cell":
        cell = G.Cell(case["nfru"], precision=case["precision"])
        return {"case": case, "cell": cell, "frus": _frus(case["nfru"], case["phase"], rng),
                "set": _settings(case, rng, False), "state": _global_state(case["phase"])}
    if kind == "cells":
        cells, frus, sets = [], [], []
        for n in _sizes(case["cells"], case["nfru"], case["uneven"]):
            pca = float(np.exp(rng.normal(0.0, 0.2))) if case["uneven"] else None
            cell = G.Cell(n, precision=case["precision"], pca_scale=pca)
            if case["packed"] and case["mode"] == "streams":
                cell.set_stage_packing(((n + 7) // 8 + case["packed"] - 1) // case["packed"])
            cells.append(cell)
            frus.append(_frus(n, case["phase"], rng))
            sets.append(_settings(case, rng, True))
        return {"case": case, "cells": cells, "frus": frus, "sets": sets, "state": _global_state(case["phase"]),
                "batch": G.Batch(case["precision"])}
    reqs = []
    for i, n in enumerate(_sizes(case["requests"], case["nfru"], True)):
        r = G.Request()
        r.nfru = n
        if rng.random() < 0.5:
            r.set = G.settings(shift=1.0, period=float(rng.uniform(400.0, 2000.0)))
        else:
            r.set = G.settings(vclamp_flag=1, vclamp_hold=-100.0, vclamp_set=float(rng.uniform(-40.0, 40.0)),
                               vclamp_duration=200.0, vclamp_shift=1.0, vclamp_period=100000.0)
        r.seed_scheme = G.SEED_BASE
        r.seed = 5489 + 1000003 * i + 7919 * int(seed)
        r.pca_scale = 1.0
        r.duration_ms = float(case["ms"])
        reqs.append(r)
    srv = G.Server(case["precision"], slots=16, mem_budget_bytes=8 << 30)
    for n in sorted(set(r.nfru for r in reqs)):
        srv.reserve(n, sum(1 for r in reqs if r.nfru == n))
    return {"case": case, "server": srv, "requests": reqs}


# ---- one pass -----------------------------------------------------------------


def _props(cell):
    """Every FRU's Ca and channel states (what write_fru_props reads at an output step)."""
    n = cell.nfru
    frus, ltype, ryr, ito2 = (np.empty((n, 5)), np.empty((n, 4, 2), np.int32), np.empty((n, 4, 5), np.int32),
                              np.empty((n, 4), np.int32))
    L = G.load()
    if L.gw_download_range(cell._h, 0, n, frus.reshape(-1), ltype.reshape(-1), ryr.reshape(-1), ito2.reshape(-1)):
        raise G.GWError((L.gw_last_error() or b"").decode())
    return {"frus": frus, "ltype": ltype, "ryr": ryr, "ito2": ito2}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "attempt":
        cell = s["cell"]
        cell.resume()
        flux, sums = [], []
        for t0, tf, dep0, depf in s["nodes"]:
            out, num = cell.stage(t0, tf, dep0, depf)
            flux.append(out)
            sums.append(num)
        return {"flux": np.array(flux), "sums": np.array(sums), "frus": _props(cell)}
    if kind == "cell":
        cell, state = s["cell"], s["state"].copy()
        cell.upload(s["frus"])
        t, states, other, currents = cell.run(state, _T0[case["phase"]], case["ms"], set_=s["set"])
        frus = cell.download()
        frus["mt"] = frus["mt"].view(np.int32)
        return {"t": t, "state": state, "states": states, "other": other, "currents": currents,
                "oldstep": cell.oldstep, "frus": frus}
    if kind == "cells":
        cells = s["cells"]
        n = len(cells)
        for c, f in zip(cells, s["frus"]):
            c.upload(f)
        t = np.full(n, _T0[case["phase"]])
        states = np.tile(s["state"], (n, 1))
        old = np.full(n, 0.1)
        if case["mode"] in ("device", "persistent"):
            tr = G.run_device(cells, s["sets"], t, states, old, case["ms"], traces=True,
                              persistent=case["mode"] == "persistent")
        else:
            tr = s["batch"].run(cells, s["sets"], t, states, old, case["ms"], traces=True,
                                lockstep=case["mode"] == "lockstep")
        props = [_props(c) for c in cells]
        return {"t": t, "states": states, "oldsteps": old, "traces": list(tr),
                **{k: np.concatenate([p[k] for p in props]) for k in ("frus", "ltype", "ryr", "ito2")}}
    srv, out = s["server"], []
    for r in s["requests"]:
        v, final = np.zeros(case["ms"]), np.zeros(G.NSTATE)
        srv.submit(r, v, final)
        out.append((v, final))
    srv.wait()
    for r in s["requests"]:
        if r.status:
            raise G.GWError(r.message.decode())
    return {"v": np.array([v for v, _ in out]), "final": np.array([f for _, f in out])}


# ---- the work of a pass --------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind == "attempt":
        n, ms = case["nfru"], case["step"]
    elif kind == "cell":
        n, ms = case["nfru"], case["ms"]
    elif kind == "cells":
        n, ms = sum(_sizes(case["cells"], case["nfru"], case["uneven"])), case["ms"]
    else:
        n, ms = sum(_sizes(case["requests"], case["nfru"], True)), case["ms"]
    subs = n * ms * (_SUBSTEPS[case["phase"]] if kind == "attempt" else _SUBSTEPS_RUN)
    # FRU state read and written once (40 B Ca, 16 B channel words, 4 B position), its
    # channel states handed out, and the 32 MT19937 words of every substep
    return {"bytes": 2 * 60.0 * n + 168.0 * n + subs * 128.0, "flops": subs * _OPS_PER_SUBSTEP}


# ---- an attempt in 64 bits, in numpy -------------------------------------------
_FARADAY, _RTF = 96.5, 8.314 * 310.0 / 96.5
_VSS = 0.5 * 0.2 * 2.03e-12
_VJSR = 4.0 * 0.53 * 0.5 * 0.2 * 1.05e-10
_PCA, _PCL = 1.5 / 2.8 * 0.2 * 0.9 * 0.9468e-11, 2.65e-15
_CAO, _CLO, _CLI, _ACAP = 2.0, 150.0, 20.0, 1.534e-4
_OMEGA, _BL, _AL = 0.83 * 2.0 * 1.3 * 0.01, 1.9356, 2.0


def _twist(m):
    m = m.copy()

    def mix(k, nxt, far):
        y = (m[:, k] & np.uint32(0x80000000)) | (nxt & np.uint32(0x7fffffff))
        m[:, k] = far ^ (y >> np.uint32(1)) ^ np.where(y & np.uint32(1), np.uint32(0x9908b0df), np.uint32(0))

    # a block of words depends only on words that are old or in an earlier block
    for a, b in ((0, 227), (227, 454), (454, 623)):
        k = np.arange(a, b)
        mix(k, m[:, k + 1], m[:, k + 397] if a == 0 else m[:, k - 227])
    mix(623, m[:, 0], m[:, 396])
    return m


def _temper(y):
    y = y ^ (y >> np.uint32(11))
    y = y ^ ((y << np.uint32(7)) & np.uint32(0x9d2c5680))
    y = y ^ ((y << np.uint32(15)) & np.uint32(0xefc60000))
    return y ^ (y >> np.uint32(18))


def _lcc_rows(s, a, b, g):
    """Exit rates (m, 4, 3) and destinations of LCC states s for alpha, beta, gamma."""
    ap, bp, z = a * _AL, b / _BL, 0.0 * g
    k = [_OMEGA / _BL**i for i in range(5)]
    rate, to = np.zeros(s.shape + (3,)), np.zeros(s.shape + (3,), np.int32)
    rows = {
        1: ((4 * a + z, 2), (g, 7)),
        2: ((b + z, 1), (3 * a + z, 3), (_AL * g, 8)),
        3: ((2 * b + z, 2), (2 * a + z, 4), (_AL**2 * g, 9)),
        4: ((3 * b + z, 3), (a + z, 5), (_AL**3 * g, 10)),
        5: ((4 * b + z, 4), (0.85 + z, 6), (_AL**4 * g, 11)),
        6: ((2.0 + z, 5),),
        7: ((k[0] + z, 1), (4 * ap + z, 8)),
        8: ((bp + z, 7), (k[1] + z, 2), (3 * ap + z, 9)),
        9: ((2 * bp + z, 8), (k[2] + z, 3), (2 * ap + z, 10)),
        10: ((3 * bp + z, 9), (k[3] + z, 4), (ap + z, 11)),
        11: ((4 * bp + z, 10), (k[4] + z, 5), (0.005 + z, 12)),
        12: ((7.0 + z, 11),),
    }
    for st, row in rows.items():
        at = s == st
        for j, (r, d) in enumerate(row):
            rate[..., j][at] = r[at]
            to[..., j][at] = d
    return rate, to


def _ryr_rows(s, regime, ca):
    """Exit rates (m, 4, 5, 3) and destinations of resolved RyR states."""
    sat, sat2 = np.minimum(2.0, ca * ca / 0.00127215), np.minimum(2.0, ca * ca / 3.4188)
    k12, k23, k34, k54, k25, k56 = (3000.0 * sat2, 300000.0 * sat, 1800.0 * sat, 0.1188 * sat, 3000.0 * sat,
                                    24000.0 * sat)
    k43, z = 0.07 / 0.06667 * 13.0, 0.0 * sat
    p7, p8 = k34 / (k34 + k43), 30.0 / (k56 + 30.0)
    r0, r2 = regime == 0, regime == 2
    d5, d3 = np.where(r0, 5, 8), np.where(r2, 7, 3)
    rows = {
        1: ((k12, 2),), 2: ((250.0 + z, 1), (k23, d3), (k25, d5)), 3: ((9.6 + z, 2), (k34, 4)),
        4: ((k43 + z, 3), (0.07 + z, d5)), 5: ((0.001235 + z, 2), (k54, 4), (k56, 6)), 6: ((30.0 + z, 5),),
        7: (((1.0 - p7) * 9.6, 2), (p7 * 0.07, 8)), 8: ((p8 * 0.001235, 2), (p8 * k54, np.where(r2, 7, 4))),
    }
    rate, to = np.zeros(s.shape + (3,)), np.zeros(s.shape + (3,), np.int32)
    for st, row in rows.items():
        at = s == st
        for j, (r, d) in enumerate(row):
            rate[..., j][at] = np.broadcast_to(r[..., None], s.shape)[at]
            to[..., j][at] = np.broadcast_to(np.asarray(d)[..., None] if np.ndim(d) else d, s.shape)[at]
    return rate, to


def _choose(u, dt, rate, to):
    """Next state where the channel leaves (u > 1 - dt * total): cumulative walk."""
    total = rate.sum(-1)
    acc = (1.0 - dt * total)[..., None] + np.cumsum(dt[..., None] * rate, -1)
    last = (rate > 0).sum(-1) - 1
    j = np.minimum((u[..., None] > acc).sum(-1), np.maximum(last, 0))
    return total, u > 1.0 - dt * total, np.take_along_axis(to, j[..., None], -1)[..., 0]


def _ode(y, v, cai, nsr, lopen, nopen):
    ss, jsr = y[:, 1:], y[:, 0]
    jryr = 0.6 * 1.5 * 1.1 * 3.96 * nopen * (jsr[:, None] - ss)
    jss = (ss - np.roll(ss, -1, 1)) / 0.05
    x = v / _RTF
    e2 = np.exp(2.0 * x)[:, None]
    a2 = (4.0 * _PCA * 1000.0 * _FARADAY * x / np.expm1(2.0 * x))[:, None] / (2.0 * _VSS * _FARADAY * 1000.0)
    jdh = -(ss * e2 - _CAO * 0.341) * a2 * lopen
    bss = 1.0 / (1.0 + 0.047 * 0.00087 / (ss + 0.00087) ** 2 + 1.124 * 0.0087 / (ss + 0.0087) ** 2)
    d = np.empty_like(y)
    d[:, 1:] = bss * (jdh + jryr - (ss - cai[:, None]) / 0.005 - jss + np.roll(jss, 1, 1))
    d[:, 0] = ((nsr - jsr) / 3.0 - _VSS / _VJSR * jryr.sum(1)) / (1.0 + 13.5 * 0.63 / (jsr + 0.63) ** 2)
    return d


def _stage64(f, t0, tf, dep0, depf):
    """Advance the FRUs of dict f over [t0, tf] (simfru_local.c), in place."""
    n = len(f["mti"])
    t = np.full(n, t0)
    live = np.arange(n)
    while len(live):
        y, lt, ryr, cl, mti = (f[k][live] for k in ("frus", "ltype", "ryr", "ito2", "mti"))
        tl, m = t[live], len(live)
        frac = (tl - t0) / (tf - t0)
        v = dep0[0] + frac * (depf[0] - dep0[0])
        ca = y[:, 1:]
        one = np.ones((m, 4))
        a = one * (4.0 * 1.2 * 0.416 * np.exp(0.012 * (v - 35.0)))[:, None]
        b = one * (4.0 * 0.45 * 0.049 * np.exp(-0.05 * (v - 35.0)))[:, None]
        lrate, lto = _lcc_rows(lt[:, :, 0], a, b, 0.83 * 1.9 * 1.3 * 0.31 * 7.5 * 0.09233 * ca)
        yinf = 0.4 / (1.0 + np.exp((v + 12.5) / 5.0)) + 0.6
        tau = 60.0 + 340.0 / (1.0 + np.exp((v + 30.0) / 12.0))
        vdi = np.where(lt[:, :, 1] == 2, (1.0 - yinf)[:, None], yinf[:, None]) / tau[:, None]
        regime = np.where(ca < 0.00011447933531005, 0, np.where(ca < 0.0368369379834969, 1, 2))
        # RyR pseudo-states: draws in cleft and RyR order, then the 32 uniforms of the substep
        rg = np.broadcast_to(regime[:, :, None], ryr.shape)
        extra = ((rg <= 1) & (ryr == 7)) | ((rg == 0) & (ryr == 8))
        order = np.cumsum(extra.reshape(m, 20), 1).reshape(ryr.shape) - 1
        etot = extra.sum((1, 2))
        pos = mti[:, None] + np.arange(52)[None, :]
        words = f["mt"][live[:, None], np.minimum(pos, 623)]
        cross = mti + etot + 32 > 624
        if cross.any():
            nxt = _twist(f["mt"][live[cross]])
            f["mt"][live[cross]] = nxt
            p = pos[cross]
            words[cross] = np.where(p < 624, words[cross], nxt[np.arange(len(p))[:, None], np.maximum(p - 624, 0)])
        rows = np.arange(m)[:, None]
        u = _temper(words).astype(np.float64) / 4294967296.0
        f["mti"][live] = np.where(cross, mti + etot + 32 - 624, mti + etot + 32)
        ux = u[np.arange(m)[:, None, None], np.maximum(order, 0)]
        ub = u[rows, etot[:, None] + np.arange(32)[None, :]].reshape(m, 4, 8)
        sat = np.minimum(2.0, ca * ca / 0.00127215)
        k34, k56 = (1800.0 * sat)[:, :, None], (24000.0 * sat)[:, :, None]
        r7 = np.where(ux < k34 / (k34 + 0.07 / 0.06667 * 13.0), 4, 3)
        r8 = np.where(ux < k56 / (k56 + 30.0), 6, 5)
        res = np.where((rg <= 1) & (ryr == 7), r7, ryr)
        res = np.where((rg == 0) & (ryr == 8), r8, res)
        res = np.where((rg >= 1) & ((ryr == 5) | (ryr == 6)), 8, res)
        ryr = np.where((rg == 2) & ((ryr == 3) | (ryr == 4)), 7, res)
        rrate, rto = _ryr_rows(ryr, regime, ca)
        clr = np.where(cl == 1, 2.0 / 0.1502 * ca, 2.0)
        mx = np.maximum(np.maximum(lrate.sum(-1), vdi), np.maximum(rrate.sum(-1).max(-1), clr)).max(1)
        dt = np.minimum(0.1 / mx, 10.001e-3)
        dt = np.where(ca.max(1) > 1.5e-3, np.minimum(dt, 5.001e-3), dt)
        last = dt >= tf - tl
        dt = np.where(last, tf - tl, dt)
        lopen = ((lt[:, :, 0] % 6 == 0) & (lt[:, :, 1] == 2)).astype(np.float64)
        nopen = np.isin(f["ryr"][live], (3, 4, 7)).sum(2)
        dep = [dep0[i] + frac * (depf[i] - dep0[i]) for i in range(3)]
        k1 = dt[:, None] * _ode(y, *dep, lopen, nopen)
        tl = np.where(last, tf, tl + dt)
        frac = (tl - t0) / (tf - t0)
        dep = [dep0[i] + frac * (depf[i] - dep0[i]) for i in range(3)]
        k2 = dt[:, None] * _ode(y + k1, *dep, lopen, nopen)
        f["frus"][live] = y + (k1 + k2) / 2.0
        d4 = np.broadcast_to(dt[:, None], (m, 4))
        _, go, new = _choose(ub[:, :, 0], d4, lrate, lto)
        lt[:, :, 0] = np.where(go, new, lt[:, :, 0])
        lt[:, :, 1] = np.where(ub[:, :, 1] >= 1.0 - d4 * vdi, 3 - lt[:, :, 1], lt[:, :, 1])
        _, go, new = _choose(ub[:, :, 2:7], np.broadcast_to(dt[:, None, None], (m, 4, 5)), rrate, rto)
        f["ltype"][live], f["ryr"][live] = lt, np.where(go, new, ryr)
        f["ito2"][live] = np.where(ub[:, :, 7] >= 1.0 - d4 * clr, 3 - cl, cl)
        t[live] = tl
        live = live[~last]


def _flux64(f, dep, scale):
    ca = f["frus"][:, 1:]
    lopen = (f["ltype"][:, :, 0] % 6 == 0) & (f["ltype"][:, :, 1] == 2)
    num = np.array([ca.sum(), f["frus"][:, 0].sum(), ca[lopen].sum(), lopen.sum(), (f["ito2"] == 2).sum()])
    x = dep[0] / _RTF
    vf, e1, e2 = 1000.0 * _FARADAY * x, np.exp(x), np.exp(2.0 * x)
    ica = 4.0 * _PCA * vf * (num[2] * e2 - num[3] * _CAO * 0.341) / (e2 - 1.0) / _ACAP
    ito2 = num[4] * _PCL * vf * (_CLI - _CLO * e1) / (1.0 - e1) / _ACAP
    n = len(f["mti"])
    return scale * np.array([(num[0] - 4.0 * n * dep[1]) / 0.005, (n * dep[2] - num[1]) / 3.0, ica, ito2]), num


def exact(case, seed):
    if case["kind"] != "attempt":
        return None
    f = _frus(case["nfru"], case["phase"], np.random.default_rng([int(seed), 2002]))
    flux, sums = [], []
    for t0, tf, dep0, depf in _attempt_nodes(case):
        _stage64(f, t0, tf, dep0, depf)
        out, num = _flux64(f, depf, 12500.0 / case["nfru"])
        flux.append(out)
        sums.append(num)
    return {"flux": np.array(flux), "sums": np.array(sums),
            "frus": {"frus": f["frus"], "ltype": None, "ryr": None, "ito2": None}}
