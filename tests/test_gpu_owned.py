"""The target-owning slice kernel (one CTA per SM owns every G-th neuron and
its ring cells in shared memory) against the graph form, bit for bit, at the
sizes where its layout changes: fewer neurons than a warp, one and two neurons
per thread, uniform weights (event counts) and several weights (fixed-point or
FP64 cells), a window shorter than the longest delay (far segments), slices of
one step and of more than 32, unconnected parts (a batch), and more spikes in
a slice than its list holds.  Weights and drive are dyadic, so the sums do not
depend on their order and every difference is an error.
"""

import numpy as np
import pytest

from nestgpu import _abi

pytestmark = pytest.mark.gpu

EXP, ALPHA, DELTA = _abi.NG_IAF_PSC_EXP, _abi.NG_IAF_PSC_ALPHA, _abi.NG_IAF_PSC_DELTA


def _run(variant, precision, model, n, copies, deg, md, maxd, uniform, hot, trace, calls):
    rng = np.random.default_rng(n + 7 * md)
    N = n * copies
    d_out = rng.integers(max(0, deg - 5), deg + 6, N)
    d_out[rng.integers(0, N, max(1, N // 10))] = 0          # sources without edges
    row = np.concatenate([[0], np.cumsum(d_out)]).astype(np.int64)
    nnz = int(row[-1])
    tgt = rng.integers(0, n, nnz) + np.repeat(np.arange(N) // n * n, d_out)
    src = np.repeat(np.arange(N), d_out)
    if uniform:
        w = np.where(src % n < 0.8 * n, 60.0, -240.0)
    else:
        w = rng.choice([40.0, 80.5, -160.0, -300.25, 0.0], nnz, p=[0.4, 0.35, 0.1, 0.1, 0.05])
    if model == DELTA:
        w = w / 256.0
    eng = _abi.Engine([(model, N)], 0.1, md, maxd, precision=precision)
    if variant >= 0:
        eng.set_tuning(0, variant, -1, -1)
    eng.set_var(0, "V_m_rel", np.full(N, 16.0) if hot else rng.uniform(0.0, 14.5, N))
    eng.set_connections(row, tgt.astype(np.int32), w, rng.integers(md, maxd + 1, nnz).astype(np.int32))
    eng.set_recording((np.arange(N) % 7 != 3).astype(np.uint8))
    drive = np.where(np.arange(N) % 5 == 2, 0.0, 11000.0)
    eng.set_poisson(drive, np.where(np.arange(N) % 2, 0.25, 0.5) if model == DELTA else np.full(N, 48.0),
                    rng.integers(md, maxd + 1, N).astype(np.int32), 11, 10**9, 5)
    if trace:
        eng.set_trace(np.arange(0, N, max(1, N // 9)), ["V_m_rel"], 3)
    for k in calls:
        eng.simulate(k)
    s, t = eng.spikes()
    o = np.lexsort((s, t))
    out = [s[o], t[o]] + [eng.get_var(0, v) for v in (("V_m_rel",) if model == DELTA else ("V_m_rel", "I_syn_ex", "I_syn_in"))]
    if trace:
        out.append(eng.trace()[1])
    st, tuned = eng.stats(), eng.tuned()
    eng.close()
    return out, (st["spikes"], st["syn_events"], st["drive_events"]), st["update_launches"], tuned


CASES = [
    # precision, model, n, copies, out-degree, min_delay, max_delay, uniform weights, hot start, trace, calls
    (_abi.NG_FP64, EXP, 23, 1, 10, 15, 15, True, False, False, (600, 7, 1400)),
    (_abi.NG_FP32, EXP, 4001, 1, 60, 15, 15, True, False, False, (300, 40, 400)),
    (_abi.NG_FP64, EXP, 4001, 1, 60, 3, 20, False, False, False, (300, 40, 400)),
    (_abi.NG_FP32, EXP, 4001, 1, 60, 2, 9, False, False, True, (301, 99)),
    (_abi.NG_FP64, ALPHA, 3001, 1, 50, 10, 25, False, False, False, (300, 41, 300)),
    (_abi.NG_FP32, ALPHA, 3001, 1, 50, 10, 25, True, False, False, (300, 41, 300)),
    (_abi.NG_FP64, DELTA, 2999, 1, 40, 5, 12, False, False, True, (300, 42, 300)),
    (_abi.NG_FP32, DELTA, 2999, 1, 40, 40, 70, True, False, False, (400, 41, 400)),
    (_abi.NG_FP64, EXP, 701, 5, 40, 15, 15, True, False, False, (300, 40, 400)),
    (_abi.NG_FP32, EXP, 9001, 1, 30, 1, 6, False, True, False, (160,)),
    (_abi.NG_FP32, EXP, 80021, 1, 12, 1, 60, False, False, False, (160,)),
    (_abi.NG_FP64, EXP, 80021, 1, 12, 4, 40, False, True, False, (160,)),
]


@pytest.mark.parametrize("case", CASES)
def test_owned_equals_graph_form(case):
    ref, st0 = _run(0, *case)[:2]
    got, st1, launches, _ = _run(5, *case)
    assert len(ref[0]) > 20
    assert st0 == st1
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)
    # full slices ran many to a launch
    assert launches < sum(case[-1]) // case[5] + len(case[-1])


@pytest.mark.parametrize("md", [1, 15])
def test_default_mode_takes_it_without_trials(md):
    # a network no other test has (the process keeps what was measured), in
    # one call long enough for every trial
    case = (_abi.NG_FP64, EXP, 2111 + md, 1, 33, md, 15, False, False, False, (4000 if md > 1 else 600,))
    ref, st0 = _run(0, *case)[:2]
    got, st1, _, tuned = _run(-1, *case)
    assert st0 == st1
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)
    assert tuned["state"] == "tuned" and tuned["update_variant"] == 5 and not tuned["candidates"]


def test_single_slices_after_many():
    # calls of one slice take another form than the calls of many around them
    case = (_abi.NG_FP64, EXP, 15011, 1, 20, 5, 12, False, False, False, (200, 5, 5, 5, 3, 2, 5, 60))
    ref, st0 = _run(0, *case)[:2]
    got, st1 = _run(5, *case)[:2]
    assert len(ref[0]) > 20 and st0 == st1
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)
