"""The work that programs have the engine do, as timed cases: networks of the
repository's own configurations, stepped through the engine's public binding
(``nestgpu._abi.Engine``, ``nestgpu.workloads``, ``nestgpu.serving`` and the
allocation-free C entry point).

A pass advances a prepared network by its simulated time, drains the recorded
spikes and reads the state back, as a script's ``Simulate(t)`` followed by
``spike_recorder.events`` and ``GetStatus`` does.  A network goes on from
where the last pass left it.  A raster is returned whole, as one ordered key
per spike, (step within the pass) * neurons + source (the order inside the
log is not defined), in a buffer of fixed length that ends in -1.

Weights of the FP64 cases are multiples of 1/8, so their ring sums do not
depend on the order of the additions; the FP32 form's fixed-point sums never
do.
"""

import copy
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "nest-simulator_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from nestgpu import _abi, serving, workloads  # noqa: E402

H = 0.1          # ms per step, everywhere
DELAY = 15       # steps: the 1.5 ms delay of the benchmark networks
FOREVER = 10**9  # steps: a serving network that never ends


def listed():
    return [
        # a controller steps a small network a few slices per tick, all memory its own
        {"name": "noalloc_tick", "kind": "noalloc", "n": 997, "k_exc": 80, "k_inh": 20, "steps": 150},
        # the deterministic balanced network of the parity tests: a notebook-sized run
        {"name": "balanced_delta", "kind": "delta", "n": 1009, "k_exc": 80, "k_inh": 20, "steps": 10000},
        # a small network with spread delays and a multimeter on ten neurons, sampled every ms
        {"name": "traced_exp", "kind": "traced", "n": 1500, "k_exc": 120, "k_inh": 30, "d_min": 10, "d_max": 25,
         "n_rec": 10, "every": 10, "steps": 2000},
        # a simulator that owns the time loop calls the engine once per slice
        {"name": "slice_calls", "kind": "calls", "n": 2503, "k_exc": 200, "k_inh": 50, "slices": 100},
        # the headline benchmark network: one simulated second
        {"name": "brunel_fp64", "kind": "brunel", "n": 12500, "k_exc": 1000, "k_inh": 250, "copies": 1,
         "precision": "fp64", "steps": 10000},
        # the same kind of network in the FP32 form, a size that fills no tile
        {"name": "brunel_fp32_odd", "kind": "brunel", "n": 9377, "k_exc": 750, "k_inh": 187, "copies": 1,
         "precision": "fp32", "steps": 10000},
        # a parameter scan: eight networks advanced together
        {"name": "batch8_fp32", "kind": "brunel", "n": 7001, "k_exc": 560, "k_inh": 140, "copies": 8,
         "precision": "fp32", "steps": 5000},
        # iaf_psc_alpha with plastic excitatory connections, learning on (weights read back)
        {"name": "hpc_stdp", "kind": "stdp", "n_exc": 3600, "n_inh": 900, "k_exc": 1800, "k_inh": 450, "steps": 2000},
        # a quarter-size cortical layer model in the plain form, spikes recorded
        {"name": "layered_quarter_fp64", "kind": "layered", "scale": 0.25, "precision": "fp64", "record": True,
         "steps": 300},
        # the full layer model in the precision form, state read at the end
        {"name": "layered_full_fp32", "kind": "layered", "scale": 1.0, "precision": "fp32", "record": False,
         "steps": 300},
        # adaptive neurons integrated with error control
        {"name": "aeif_fp64", "kind": "aeif", "n": 50000, "precision": "fp64", "steps": 600},
        # a server that admits, runs and retires networks of mixed sizes
        {"name": "serving_mix", "kind": "serving", "count": 24, "n_min": 1000, "n_max": 30000, "t_min_ms": 100.0,
         "t_max_ms": 250.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["noalloc", "delta", "traced", "calls", "brunel", "brunel", "stdp", "layered", "layered", "aeif",
                       "serving"])
    if kind in ("noalloc", "delta"):
        n = _log_int(rng, 100, 10000)
        k = max(4, min(n // 10, 500))
        return {"kind": kind, "n": n, "k_exc": k, "k_inh": max(1, k // 4),
                "steps": rng.randint(15, 300) if kind == "noalloc" else rng.randint(500, 10000)}
    if kind == "traced":
        n = _log_int(rng, 100, 10000)
        k = max(4, min(n // 10, 500))
        d_min = rng.randint(1, 20)
        every = rng.randint(1, 20)
        return {"kind": kind, "n": n, "k_exc": k, "k_inh": max(1, k // 4), "d_min": d_min,
                "d_max": d_min + rng.randint(0, 40), "n_rec": rng.randint(1, min(n, 50)), "every": every,
                "steps": every * (rng.randint(200, 2000) // every)}
    if kind == "calls":
        n = _log_int(rng, 500, 15000)
        k = max(4, min(n // 10, 1000))
        return {"kind": kind, "n": n, "k_exc": k, "k_inh": max(1, k // 4), "slices": rng.randint(20, 200)}
    if kind == "brunel":
        copies = rng.choice([1, 1, 1, 2, 5, 8])
        n = _log_int(rng, 1000, 30000 if copies == 1 else 7001)
        k = max(4, min(n // 12, 1000))
        return {"kind": kind, "n": n, "k_exc": k, "k_inh": max(1, k // 4), "copies": copies,
                "precision": rng.choice(["fp64", "fp32"]), "steps": rng.randint(1000, 8000)}
    if kind == "stdp":
        n = _log_int(rng, 500, 3600)
        k = max(4, n // 2)
        return {"kind": kind, "n_exc": n, "n_inh": max(1, n // 4), "k_exc": k, "k_inh": max(1, k // 4),
                "steps": rng.randint(200, 2000)}
    if kind == "layered":
        precision = rng.choice(["fp64", "fp32"])
        return {"kind": kind, "scale": round(math.exp(rng.uniform(math.log(0.05), math.log(0.35 if precision == "fp64"
                                                                                         else 0.9))), 3),
                "precision": precision, "record": rng.random() < 0.5, "steps": rng.randint(100, 300)}
    if kind == "aeif":
        return {"kind": kind, "n": _log_int(rng, 1200, 50000), "precision": rng.choice(["fp64", "fp32"]),
                "steps": rng.randint(150, 600)}
    return {"kind": kind, "count": rng.randint(4, 24), "n_min": 1000, "n_max": _log_int(rng, 3000, 30000),
            "t_min_ms": 50.0, "t_max_ms": float(rng.randint(60, 250))}


# ---------------------------------------------------------------------------
# networks
# ---------------------------------------------------------------------------
def _graph(rng, n, n_exc, k_exc, k_inh, w_exc, w_inh, copies=1):
    """Rows of `copies` networks of n neurons: every neuron of a network gets
    k_exc + k_inh in-edges on average (each source draws its targets)."""
    out_e = max(1, int(round(k_exc * n / n_exc)))
    out_i = max(1, int(round(k_inh * n / max(1, n - n_exc))))
    deg = np.where(np.arange(n) < n_exc, out_e, out_i).astype(np.int64)
    deg = np.tile(deg, copies)
    row = np.zeros(n * copies + 1, dtype=np.int64)
    np.cumsum(deg, out=row[1:])
    tgt = rng.integers(0, n, row[-1], dtype=np.int32)
    if copies > 1:
        per = int(row[n])
        tgt += np.repeat(np.arange(copies, dtype=np.int32) * n, per)
    w = np.repeat(np.where(np.tile(np.arange(n) < n_exc, copies), w_exc, w_inh), deg)
    return row, tgt, w


def _delta_network(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    n_exc = int(round(0.8 * n))
    row, tgt, w = _graph(rng, n, n_exc, case["k_exc"], case["k_inh"], 0.125, -0.625)
    return {"n": n, "row": row, "tgt": tgt, "w": w, "I_e": rng.uniform(300.0, 500.0, n), "V0": rng.uniform(0.0, 20.0, n),
            "C_m": 250.0, "tau_m": 20.0, "t_ref": 2.0, "V_th": 20.0, "V_reset": 10.0}


def _delta_coefficients(net):
    h = (1.0 / 1000.0) * 100
    P33 = math.exp(-h / net["tau_m"])
    return P33, 1 / net["C_m"] * (1 - P33) * net["tau_m"], int(round(net["t_ref"] / H))


def _precision(case):
    return _abi.NG_FP32 if case.get("precision") == "fp32" else _abi.NG_FP64


def _as_state(case, values):
    return values.astype(np.float32) if case.get("precision") == "fp32" else values


def _raster_buffer(n, steps, most_hz, refr=5):
    """Room for the spikes of a pass: what refractoriness allows, or a mean
    rate well above what the networks reach."""
    return np.empty(int(min(n * (steps // refr + 1), 100_000 + n * steps * H * 1e-3 * most_hz)), dtype=np.int32)


def _raster(buf, src, stamp, n, start):
    keys = ((stamp - start) * n + src).astype(np.int32)
    keys.sort()
    if len(keys) > len(buf):
        raise RuntimeError("more spikes than the raster buffer holds")
    buf[:len(keys)] = keys
    buf[len(keys):] = -1
    return buf


def _exp_engine(case, seed, n, copies, delays=None):
    """Poisson-driven iaf_psc_exp networks: J = 87.75 pA, g = 5, 8 kHz."""
    rng = np.random.default_rng(seed)
    N = n * copies
    n_exc = int(round(0.8 * n))
    J = 87.75
    scale = 1000.0 / case["k_exc"]      # smaller networks keep the summed input per neuron near the large one's
    w = J * max(1.0, min(8.0, 2.0 ** round(math.log2(scale) / 2)))
    row, tgt, wt = _graph(rng, n, n_exc, case["k_exc"], case["k_inh"], w, -5.0 * w, copies)
    d = np.full(len(tgt), DELAY, dtype=np.int32) if delays is None else rng.integers(delays[0], delays[1] + 1, len(tgt),
                                                                                   dtype=np.int32)
    lo, hi = (DELAY, DELAY) if delays is None else delays
    eng = _abi.Engine([(_abi.NG_IAF_PSC_EXP, N)], H, lo, hi, precision=_precision(case))
    eng.set_graph_slices(64)
    eng.set_var(0, "tau_syn_ex", np.full(N, 0.5))
    eng.set_var(0, "tau_syn_in", np.full(N, 0.5))
    eng.set_var(0, "V_m_rel", rng.normal(-58.0, 10.0, N) + 70.0)
    eng.set_connections(row, tgt, wt, d)
    eng.set_poisson(np.full(N, 8000.0), np.full(N, J), np.full(N, lo, dtype=np.int32), 0, 2**62, seed + 1)
    eng.set_recording(np.ones(N, dtype=np.uint8))
    return eng, rng


class NoAllocNet(ctypes.Structure):
    _fields_ = [
        ("n", ctypes.c_int64), ("min_delay", ctypes.c_int32), ("max_delay", ctypes.c_int32),
        ("start_step", ctypes.c_int64),
        ("P33", ctypes.c_void_p), ("P30", ctypes.c_void_p), ("V_th_rel", ctypes.c_void_p),
        ("V_reset_rel", ctypes.c_void_p), ("V_min_rel", ctypes.c_void_p), ("I_e", ctypes.c_void_p),
        ("refr_counts", ctypes.c_void_p), ("V_m_rel", ctypes.c_void_p), ("r", ctypes.c_void_p),
        ("row_ptr", ctypes.c_void_p), ("target", ctypes.c_void_p), ("weight", ctypes.c_void_p),
        ("delay", ctypes.c_void_p), ("out_src", ctypes.c_void_p), ("out_stamp", ctypes.c_void_p),
        ("out_cap", ctypes.c_int64), ("out_count", ctypes.c_void_p),
        ("continue_run", ctypes.c_int32), ("reserved", ctypes.c_int32), ("out_skipped", ctypes.c_void_p),
    ]


def _prepare_noalloc(case, seed):
    net = _delta_network(case, seed)
    n = net["n"]
    P33, P30, refr = _delta_coefficients(net)
    cap = n * (case["steps"] // (refr + 1) + 1)
    f64, i32 = torch.float64, torch.int32
    t = {
        "P33": torch.full((n,), P33, dtype=f64), "P30": torch.full((n,), P30, dtype=f64),
        "V_th_rel": torch.full((n,), net["V_th"], dtype=f64), "V_reset_rel": torch.full((n,), net["V_reset"], dtype=f64),
        "V_min_rel": torch.full((n,), -np.finfo(np.float64).max, dtype=f64), "I_e": torch.from_numpy(net["I_e"]),
        "refr_counts": torch.full((n,), refr, dtype=i32), "V_m_rel": torch.from_numpy(net["V0"].copy()),
        "r": torch.zeros(n, dtype=i32), "row_ptr": torch.from_numpy(net["row"]), "target": torch.from_numpy(net["tgt"]),
        "weight": torch.from_numpy(net["w"]), "delay": torch.full((len(net["tgt"]),), DELAY, dtype=i32),
        "out_src": torch.zeros(cap, dtype=i32), "out_stamp": torch.zeros(cap, dtype=torch.int64),
        "out_count": torch.zeros(1, dtype=torch.int64), "out_skipped": torch.zeros(1, dtype=torch.int64),
    }
    t = {k: v.cuda() for k, v in t.items()}
    desc = NoAllocNet(n=n, min_delay=DELAY, max_delay=DELAY, out_cap=cap, **{k: v.data_ptr() for k, v in t.items()})
    lib = _abi.load()
    lib.ng_simulate_noalloc.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p]
    lib.ng_simulate_noalloc.restype = ctypes.c_int
    return {"kind": "noalloc", "lib": lib, "desc": desc, "t": t, "steps": case["steps"]}


def _prepare_delta(case, seed):
    net = _delta_network(case, seed)
    n = net["n"]
    eng = _abi.Engine([(_abi.NG_IAF_PSC_DELTA, n)], H, DELAY, DELAY)
    eng.set_graph_slices(64)
    for name, key in (("C_m", "C_m"), ("tau_m", "tau_m"), ("t_ref", "t_ref"), ("V_th_rel", "V_th"),
                      ("V_reset_rel", "V_reset")):
        eng.set_var(0, name, np.full(n, net[key]))
    eng.set_var(0, "I_e", net["I_e"])
    eng.set_var(0, "V_m_rel", net["V0"])
    eng.set_connections(net["row"], net["tgt"], net["w"], np.full(len(net["tgt"]), DELAY, dtype=np.int32))
    eng.set_recording(np.ones(n, dtype=np.uint8))
    return {"kind": "delta", "eng": eng, "case": case, "n": n, "step": 0, "steps": case["steps"],
            "buf": _raster_buffer(n, case["steps"], 150.0)}


def _prepare_stdp(case, seed):
    rng = np.random.default_rng(seed)
    ne, ni = case["n_exc"], case["n_inh"]
    n = ne + ni
    tau_syn, tau_m, C_m = workloads.HPC_TAU_SYN, 10.0, 250.0
    JE = 0.14 * workloads.alpha_pa_per_mv(tau_m, tau_syn, C_m) * 9000.0 / (4.0 * case["k_exc"])
    rate = 1.685 * 20.0 / (tau_m / C_m * JE * math.e * tau_syn) * 1000.0
    eng = _abi.Engine([(_abi.NG_IAF_PSC_ALPHA, n)], H, DELAY, DELAY, precision=_abi.NG_FP32)
    eng.set_graph_slices(64)
    for name, v in (("C_m", C_m), ("tau_m", tau_m), ("t_ref", 0.5), ("V_th_rel", 20.0), ("V_reset_rel", 0.0),
                    ("tau_syn_ex", tau_syn), ("tau_syn_in", tau_syn), ("tau_minus", 30.0)):
        eng.set_var(0, name, np.full(n, v))
    eng.set_var(0, "V_m_rel", rng.normal(5.7, 7.2, n))
    # static: E -> I, I -> all; plastic: E -> E
    out_ei = max(1, case["k_exc"] * ni // ne)
    out_i = max(1, case["k_inh"] * n // ni)
    row = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(np.where(np.arange(n) < ne, out_ei, out_i), out=row[1:])
    tgt = np.concatenate([rng.integers(ne, n, ne * out_ei, dtype=np.int32), rng.integers(0, n, ni * out_i, dtype=np.int32)])
    w = np.concatenate([np.full(ne * out_ei, JE), np.full(ni * out_i, -5.0 * JE)])
    eng.set_connections(row, tgt, w, np.full(len(tgt), DELAY, dtype=np.int32))
    prow = np.arange(ne + 1, dtype=np.int64) * case["k_exc"]
    ptgt = rng.integers(0, ne, ne * case["k_exc"], dtype=np.int32)
    eng.set_plastic(prow, ptgt, np.full(len(ptgt), JE), np.full(len(ptgt), DELAY, dtype=np.int32), lam=0.1, alpha=0.0513,
                    mu=0.4, tau_plus=15.0)
    eng.set_poisson(np.full(n, rate), np.full(n, JE), np.full(n, DELAY, dtype=np.int32), 0, 2**62, seed + 1)
    eng.set_recording(np.ones(n, dtype=np.uint8))
    return {"kind": "stdp", "eng": eng, "case": dict(case, precision="fp32"), "n": n, "step": 0, "steps": case["steps"],
            "buf": _raster_buffer(n, case["steps"], 400.0)}


def _prepare_layered(case, seed):
    spec = workloads.layered_spec(seed=2024, scale=case["scale"])   # the configuration's probabilities
    spec["seed"] = seed                                             # graph, drive and initial state of this input
    if case["precision"] == "fp64":
        spec["J"], spec["J_sd"] = 87.75, 0.0
    if case["scale"] < 1.0:
        # the in-degree shrinks with the populations: the external drive makes up for part of it
        spec["k_ext"] = spec["k_ext"] + int(1000 * (1.0 - case["scale"]))
    eng = workloads.layered_engine(spec, case["precision"])
    nid = workloads.layered_add(eng, spec, FOREVER, record=case["record"])
    n = sum(spec["sizes"])
    return {"kind": "net", "eng": eng, "case": case, "n": n, "nid": nid, "step": 0, "steps": case["steps"],
            "buf": _raster_buffer(n, case["steps"], 500.0) if case["record"] else None,
            "vars": ("V_m_rel", "I_syn_ex", "I_syn_in")}


def _prepare_aeif(case, seed):
    n = case["n"]
    n_exc = int(round(0.8 * n))
    spec = workloads.aeif_spec(seed=seed, n_exc=n_exc, n_inh=n - n_exc)
    eng = workloads.aeif_engine(spec, case["precision"])
    nid = workloads.aeif_add(eng, spec, FOREVER, record=True)
    return {"kind": "net", "eng": eng, "case": case, "n": n, "nid": nid, "step": 0, "steps": case["steps"],
            "buf": _raster_buffer(n, case["steps"], 100.0), "vars": ("V_m", "g_ex", "g_in", "w")}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "noalloc":
        return _prepare_noalloc(case, seed)
    if kind == "delta":
        return _prepare_delta(case, seed)
    if kind == "stdp":
        return _prepare_stdp(case, seed)
    if kind == "layered":
        return _prepare_layered(case, seed)
    if kind == "aeif":
        return _prepare_aeif(case, seed)
    if kind == "serving":
        # the mix of sizes and durations is the case's, the networks themselves the input's
        reqs = serving.make_requests(count=case["count"], rate_hz=20.0, seed=2026, n_min=case["n_min"],
                                     n_max=case["n_max"], t_min_ms=case["t_min_ms"], t_max_ms=case["t_max_ms"])
        for r, s in zip(reqs, np.random.default_rng(seed).integers(1, 2**62, len(reqs))):
            r.seed = int(s)
        eng = serving.new_engine("fp32", capacity_neurons=500_000, capacity_edges=500_000_000, max_networks=64)
        return {"kind": "serving", "eng": eng, "reqs": reqs,
                "buf": np.empty(int(sum(r.n * r.steps for r in reqs) * H * 1e-3 * 200.0), dtype=np.int32)}
    n, copies = case["n"], case.get("copies", 1)
    delays = (case["d_min"], case["d_max"]) if kind == "traced" else None
    eng, rng = _exp_engine(case, seed, n, copies, delays)
    if kind == "traced":
        eng.set_trace(np.sort(rng.choice(n, case["n_rec"], replace=False)), ["V_m_rel", "I_syn_ex", "I_syn_in"],
                      case["every"])
    steps = case["slices"] * DELAY if kind == "calls" else case["steps"]
    return {"kind": kind, "eng": eng, "case": case, "n": n * copies, "step": 0, "steps": steps,
            "buf": _raster_buffer(n * copies, steps, 60.0)}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "noalloc":
        rc = state["lib"].ng_simulate_noalloc(ctypes.byref(state["desc"]), state["steps"],
                                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        _abi.check(rc)
        t = state["t"]
        return [t["V_m_rel"], t["r"], t["out_count"], t["out_skipped"]]
    eng = state["eng"]
    if kind == "serving":
        done, _ = serving.run_batched([copy.copy(r) for r in state["reqs"]], eng, realtime=False)
        # the rasters of the networks one after the other, and their lengths
        done.sort(key=lambda r: r.rid)
        buf, at = state["buf"], 0
        for r in done:
            k = len(r.spikes[0])
            if at + k > len(buf):
                raise RuntimeError("more spikes than the raster buffer holds")
            _raster(buf[at:at + k], r.spikes[0], r.spikes[1], r.n, 0)
            at += k
        buf[at:] = -1
        return [buf, np.array([len(r.spikes[0]) for r in done])]
    case, n, start, steps = state["case"], state["n"], state["step"], state["steps"]
    state["step"] += steps
    if kind == "net":
        eng.simulate(steps)
        out = [_as_state(case, eng.net_get_var(state["nid"], v, n)) for v in state["vars"]]
        if state["buf"] is not None:
            src, stamp = eng.net_spikes(state["nid"])
            out.append(_raster(state["buf"], src, stamp, n, start))
        return out
    if kind == "calls":
        for t in range(start, start + steps, DELAY):
            eng.update(t, 0, DELAY)
        eng.sync()
    else:
        eng.simulate(steps)
    src, stamp = eng.spikes()
    out = [_raster(state["buf"], src, stamp, n, start), _as_state(case, eng.get_var(0, "V_m_rel"))]
    if kind == "traced":
        out.append(eng.trace()[1])
    if kind == "stdp":
        out.append(eng.plastic_weights())
    if kind != "delta":
        out += [_as_state(case, eng.get_var(0, v)) for v in ("I_syn_ex", "I_syn_in")]
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: the state read and written once, 8 bytes per out-edge of every
    spike (edge word and weight in their 4-byte forms), the recorded spikes;
    flops: the arithmetic of the neuron steps and one add per event.  The
    mean rates are those the networks run at."""
    kind = case["kind"]
    if kind == "serving":
        mean_n = (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
        steps = 0.5 * (case["t_min_ms"] + case["t_max_ms"]) / H
        n, rate, flops, state = case["count"] * mean_n, 130.0, 20.0, 28.0
        deg = min(0.1 * mean_n, 1000.0) * 1.25
    elif kind == "layered":
        spec = workloads.layered_spec(scale=case["scale"])
        n, steps = sum(spec["sizes"]), case["steps"]
        rate, flops, state = 190.0, 20.0, 28.0 if case["precision"] == "fp32" else 52.0
        deg = workloads.layered_expected_edges(spec) / n
    elif kind == "aeif":
        n, steps, rate, flops, deg = case["n"], case["steps"], 7.0, 600.0, 1000.0
        state = 68.0
    elif kind == "stdp":
        n, steps, rate, flops = case["n_exc"] + case["n_inh"], case["steps"], 25.0, 40.0
        deg, state = case["k_exc"] + case["k_inh"], 28.0
    else:
        n = case["n"] * case.get("copies", 1)
        steps = case["slices"] * DELAY if kind == "calls" else case["steps"]
        rate = 55.0 if kind in ("noalloc", "delta") else 10.0
        deg, flops = case["k_exc"] + case["k_inh"], 8.0 if kind in ("noalloc", "delta") else 20.0
        state = 28.0 if case.get("precision") == "fp32" else 52.0
    spikes = n * rate * steps * H * 1e-3
    return {"bytes": 2.0 * n * state + spikes * (8.0 * deg + 12.0), "flops": n * steps * flops + spikes * deg}


# ---------------------------------------------------------------------------
# the deterministic networks in plain numpy, 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] not in ("noalloc", "delta") or case["steps"] * (case["n"] + 2000) > 6e7:
        return None   # chaotic drive-by-drive dynamics, or too long in numpy
    net = _delta_network(case, seed)
    n, steps = net["n"], case["steps"]
    P33, P30, refr = _delta_coefficients(net)
    V, r = net["V0"].copy(), np.zeros(n, dtype=np.int32)
    ring = np.zeros((DELAY, n))
    keys = []
    for t in range(steps):
        inp = ring[t % DELAY]
        free = r == 0
        V = np.where(free, P30 * net["I_e"] + P33 * V + inp, V)
        r = np.where(free, r, r - 1)
        spk = np.nonzero(V >= net["V_th"])[0]
        inp[:] = 0.0
        if len(spk):
            r[spk] = refr
            V[spk] = net["V_reset"]
            keys.append((t + 1) * n + spk)
            for s in spk:
                a, b = net["row"][s], net["row"][s + 1]
                np.add.at(inp, net["tgt"][a:b], net["w"][a:b])
    keys = np.concatenate(keys) if keys else np.zeros(0, dtype=np.int64)
    if case["kind"] == "noalloc":
        return [V, r.astype(np.int32), np.array([len(keys)]), np.array([0])]
    return [_raster(_raster_buffer(n, steps, 150.0), keys % n, keys // n, n, 0), V]
