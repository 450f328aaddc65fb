"""That the networks of test_gpu_owned.py run in the target-owning kernel, in
the layouts they are there for: an engine that quietly took another form would
pass the comparison of results."""

import numpy as np
import pytest

import test_gpu_owned as owned
from nestgpu import _abi

pytestmark = pytest.mark.gpu

COUNT, FIXED, F64 = 0, 1, 2
# (cell, held: at most one neuron per thread, window shorter than the longest delay, parts), case by case.
# None: the kernel does not take the network (delays beyond the window at more than one step per slice).
WANT = [(COUNT, 1, False, 1), (COUNT, 1, False, 1), (F64, 1, False, 1), (FIXED, 1, False, 1), (F64, 1, False, 1),
        (COUNT, 1, False, 1), (F64, 1, False, 1), (COUNT, 1, False, 1), (COUNT, 1, False, 5), (FIXED, 1, False, 1),
        (FIXED, 0, True, 1), None]
# layouts that no case there has: two neurons per thread with FP64 cells and with counts, counts with far segments
MORE = [
    ((_abi.NG_FP64, owned.DELTA, 80021, 1, 12, 1, 44, False, True, False, (160,)), (F64, 0, True, 1)),
    ((_abi.NG_FP64, owned.EXP, 76801, 1, 12, 1, 20, False, False, False, (160,)), (F64, 0, True, 1)),
    ((_abi.NG_FP64, owned.EXP, 80021, 1, 12, 2, 70, True, True, False, (160,)), (COUNT, 0, True, 1)),
    ((_abi.NG_FP32, owned.EXP, 80021, 1, 12, 2, 20, True, False, True, (160,)), (COUNT, 0, False, 1)),
    ((_abi.NG_FP64, owned.EXP, 40009, 1, 20, 1, 190, True, False, False, (450,)), (COUNT, 1, True, 1)),
]
# delays beyond the window in networks whose other forms are faster then
REFUSED = [
    (_abi.NG_FP64, owned.DELTA, 80021, 1, 12, 4, 40, False, True, False, (160,)),
    (_abi.NG_FP64, owned.EXP, 40009, 1, 20, 3, 190, True, False, False, (450,)),
    (_abi.NG_FP32, owned.EXP, 40009, 1, 20, 2, 70, False, False, False, (300,)),
    (_abi.NG_FP64, owned.EXP, 12503, 1, 20, 1, 160, False, False, False, (300,)),
]


def _forms(monkeypatch):
    """Every engine closed from here on leaves its slice form in the list."""
    seen, close = [], _abi.Engine.close

    def closing(self):
        if self.handle:
            seen.append((self.slice_form(), self.tuned()))
        close(self)

    monkeypatch.setattr(_abi.Engine, "close", closing)
    return seen


def _check(case, want, f, tuned, out):
    md, hot, calls = case[5], case[8], case[-1]
    total = sum(calls) // md
    assert sum(f["slices"].values()) == total
    if want is None:
        assert f["own_state"] == -1 and f["slices"]["k_run_owned"] == 0
        return
    # all but what a call starts or ends with in the middle of a slice, and calls of a few slices
    assert f["slices"]["k_run_owned"] >= total - 8 * len(calls) and f["slices"]["k_run_owned"] > 0
    cell, held, far, parts = want
    assert f["own_state"] == 1 and f["own_cell"] == cell and f["own_held"] == held and f["own_parts"] == parts
    assert (f["own_window"] < f["own_slots"]) == far == (f["own_far_edges"] > 0)
    assert f["own_ctas"] >= parts and f["own_ctas"] * f["own_neurons"] >= case[2] * case[3]
    if sum(calls) % md == 0 and calls[-1] >= 16 * md:
        assert f["form"] == tuned["update_kernel"] == "k_run_owned"
    if hot:
        # more spikes in a slice than the kernel's list holds (4,096)
        assert np.bincount((out[1] - 1) // md).max() > 4096


@pytest.mark.parametrize("k", range(len(owned.CASES)))
def test_layout_of(monkeypatch, k):
    seen = _forms(monkeypatch)
    out = owned._run(5, *owned.CASES[k])[0]
    _check(owned.CASES[k], WANT[k], *seen[0], out)


@pytest.mark.parametrize("case,want", MORE)
def test_more_layouts(monkeypatch, case, want):
    seen = _forms(monkeypatch)
    ref, st0 = owned._run(0, *case)[:2]
    got, st1 = owned._run(5, *case)[:2]
    _check(case, want, *seen[1], got)
    assert len(ref[0]) > 20 and st0 == st1
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("case", REFUSED)
def test_long_delays_keep_the_other_forms(monkeypatch, case):
    seen = _forms(monkeypatch)
    owned._run(5, *case)
    _check(case, None, *seen[0], None)


def test_what_ran_is_named(monkeypatch):
    seen = _forms(monkeypatch)
    case = list(owned.CASES[1])
    case[-1] = (300,)
    owned._run(0, *case)
    owned._run(5, *case)
    assert [(f["form"], t["update_kernel"]) for f, t in seen] == [("kernels", "k_update_iaf"),
                                                                  ("k_run_owned", "k_run_owned")]
    assert seen[0][0]["own_state"] == 0 and seen[0][0]["own_bytes"] == 0
    # at least the two bytes of an edge word
    assert seen[1][0]["own_bytes"] > 2 * seen[1][0]["own_edges"] > 0


# neurons, connected networks among them (first, size); the other neurons have no connections
@pytest.mark.parametrize("n,nets", [
    (4101, [(0, 4001)]),                            # unconnected neurons behind a network
    (4101, [(100, 4001)]),                          # ... before it
    (4130, [(0, 2000), (2100, 2000)]),              # ... and between two
    (6200, [(31 * k, 31) for k in range(200)]),     # more networks than SMs
    (5000, [(0, 4950), (4960, 9)]),                 # a network too small for an SM of its own
])
def test_parts(n, nets):
    md = 15

    def run(variant):
        rng = np.random.default_rng(n)
        deg = np.zeros(n, dtype=np.int64)
        for first, size in nets:
            deg[first:first + size] = rng.integers(10, 40, size)
        row = np.concatenate([[0], np.cumsum(deg)])
        src = np.repeat(np.arange(n), deg)
        tgt = np.zeros(len(src), dtype=np.int32)
        for first, size in nets:
            at = (src >= first) & (src < first + size)
            tgt[at] = rng.integers(first, first + size, at.sum())
        eng = _abi.Engine([(_abi.NG_IAF_PSC_EXP, n)], 0.1, md, md)
        eng.set_tuning(0, variant, -1, -1)
        eng.set_var(0, "V_m_rel", rng.uniform(0.0, 14.5, n))
        eng.set_connections(row, tgt, np.where(src % 5 < 4, 60.0, -240.0), np.full(len(src), md, dtype=np.int32))
        eng.set_recording(np.ones(n, dtype=np.uint8))
        eng.set_poisson(np.full(n, 11000.0), np.full(n, 48.0), np.full(n, md, dtype=np.int32), 0, 10**9, 3)
        eng.simulate(600)
        s, t = eng.spikes()
        o = np.lexsort((s, t))
        out = [s[o], t[o]] + [eng.get_var(0, v) for v in ("V_m_rel", "I_syn_ex", "I_syn_in")]
        f = eng.slice_form()
        eng.close()
        return out, f

    ref, got = run(0), run(5)
    assert len(ref[0][0]) > 20
    for a, b in zip(ref[0], got[0]):
        np.testing.assert_array_equal(a, b)
    f = got[1]
    assert f["slices"]["k_run_owned"] == 40
    assert f["own_parts"] <= f["own_ctas"]
    # no SM has much more than its share of the neurons
    assert f["own_neurons"] <= 2 * -(-n // f["own_ctas"])
    assert f["own_ctas"] >= 100


# precision, one weight per class, longest delay (the last: 4-byte edge words), in-edges of target 3, cell
@pytest.mark.parametrize("precision,uniform,maxd,many,cell", [
    (_abi.NG_FP64, True, 15, 12000, COUNT), (_abi.NG_FP32, False, 15, 12000, FIXED), (_abi.NG_FP64, False, 15, 12000, F64),
    (_abi.NG_FP32, True, 2500, 12000, COUNT), (_abi.NG_FP32, False, 15, 66000, None), (_abi.NG_FP64, False, 15, 66000, F64)])
def test_long_rows(precision, uniform, maxd, many, cell):
    """Rows whose segments are put together in shared memory: in one round, in
    several (60,000 edges), one segment larger than the buffer (`many` edges of
    one source to one target), sources without edges; and more in-edges than a
    count or a fixed-point cell holds."""
    n, md = 1103, 5

    def run(variant):
        rng = np.random.default_rng(9)
        deg = rng.integers(1900, 2600, n)
        deg[::50] = 0
        deg[5], deg[7] = 60000, many + 40000
        row = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
        src = np.repeat(np.arange(n), deg)
        tgt = rng.integers(0, n, len(src)).astype(np.int32)
        tgt[row[7]:row[7] + many] = 3
        w = np.where(src % 5 < 4, 0.5, -2.0)
        if not uniform:
            w = w * rng.choice([1.0, 1.25, 0.0], len(src), p=[0.5, 0.45, 0.05])
            w[row[7]:row[7] + many] = 0.25
        eng = _abi.Engine([(_abi.NG_IAF_PSC_EXP, n)], 0.1, md, maxd, precision=precision)
        eng.set_tuning(0, variant, -1, -1)
        V = rng.uniform(0.0, 14.5, n)
        V[[5, 7]] = 16.0
        eng.set_var(0, "V_m_rel", V)
        eng.set_connections(row, tgt, w, rng.integers(md, min(maxd, 60) + 1, len(src)).astype(np.int32))
        eng.set_recording(np.ones(n, dtype=np.uint8))
        eng.set_poisson(np.full(n, 11000.0), np.full(n, 48.0), np.full(n, md, dtype=np.int32), 0, 10**9, 3)
        eng.simulate(300)
        s, t = eng.spikes()
        o = np.lexsort((s, t))
        out = [s[o], t[o]] + [eng.get_var(0, v) for v in ("V_m_rel", "I_syn_ex", "I_syn_in")]
        f = eng.slice_form()
        eng.close()
        return out, f

    ref, got = run(0)[0], run(5)
    assert len(ref[0]) > 100 and {5, 7} <= set(ref[0][:2])
    for a, b in zip(ref, got[0]):
        np.testing.assert_array_equal(a, b)
    f = got[1]
    if cell is None:
        assert f["own_state"] == -1
    else:
        assert f["own_state"] == 1 and f["own_cell"] == cell and f["slices"]["k_run_owned"] == 60
        assert f["own_edges"] >= 2048 * n


def _plain(n, deg, md, seed=4, **kw):
    rng = np.random.default_rng(seed)
    eng = _abi.Engine([(_abi.NG_IAF_PSC_EXP, n)], 0.1, md, md, **kw)
    _connect(eng, n, deg, md, seed)
    eng.set_var(0, "V_m_rel", rng.uniform(0.0, 14.5, n))
    eng.set_recording(np.ones(n, dtype=np.uint8))
    eng.set_poisson(np.full(n, 11000.0), np.full(n, 48.0), np.full(n, md, dtype=np.int32), 0, 10**9, 3)
    return eng


def _connect(eng, n, deg, md, seed):
    rng = np.random.default_rng(seed)
    src = np.repeat(np.arange(n), deg)
    eng.set_connections(np.arange(n + 1, dtype=np.int64) * deg, rng.integers(0, n, n * deg).astype(np.int32),
                        np.where(src % 5 < 4, 60.0, -240.0), np.full(n * deg, md, dtype=np.int32))


def _raster(eng):
    s, t = eng.spikes()
    o = np.lexsort((s, t))
    return s[o], t[o], eng.get_var(0, "V_m_rel")


def test_layout_waits_until_it_pays():
    """Short calls on a new network build nothing; once the slices that ran
    would have repaid the build it is there; a new graph starts over, and its
    memory is given back; the results are those of one long call's form."""
    n, deg, md = 4001, 60, 15
    eng = _plain(n, deg, md)
    own = lambda: eng.slice_form()["slices"]["k_run_owned"]  # noqa: E731
    for k in (1, 15, 30, 60):
        eng.simulate(k)
        assert eng.slice_form()["own_state"] == 0 and eng.slice_form()["own_bytes"] == 0
    for _ in range(40):
        eng.simulate(20 * md)
        if own():
            break
    ran = sum(eng.slice_form()["slices"].values())
    assert own() > 0 and 60 < ran < 300
    assert eng.slice_form()["own_bytes"] > 2 * n * deg
    eng.simulate(14)                      # to the slice boundary again: 106 + 14 = 8 * 15
    first = _raster(eng)
    # short calls of a network whose layout is there: one and two slices take the other forms
    before = own()
    eng.simulate(md)
    eng.simulate(2 * md)
    assert own() == before
    eng.simulate(6 * md)
    assert own() == before + 6
    _connect(eng, n, deg, md, 5)
    f = eng.slice_form()
    assert f["own_state"] == 0 and f["own_bytes"] == 0
    eng.simulate(20 * md)
    assert eng.slice_form()["own_state"] == 0
    eng.simulate(600 * md)
    assert eng.slice_form()["own_state"] == 1
    second = _raster(eng)
    eng.set_tuning(0, 2, -1, -1)          # another form is chosen: the memory goes back
    assert eng.slice_form()["own_bytes"] == 0
    eng.close()
    ref = _plain(n, deg, md)
    ref.set_tuning(0, 0, -1, -1)
    steps = sum((1, 15, 30, 60)) + 14 + (ran - 7) * md
    ref.simulate(steps)
    for a, b in zip(first, _raster(ref)):
        np.testing.assert_array_equal(a, b)
    ref.simulate(9 * md)
    _connect(ref, n, deg, md, 5)
    ref.simulate(620 * md)
    for a, b in zip(second, _raster(ref)):
        np.testing.assert_array_equal(a, b)
    ref.close()


def test_serving_network_that_ends_soon_builds_nothing():
    """A network that does not live long enough keeps the kernels per slice; a
    longer one gets the layout, and the memory goes with the last network."""
    from nestgpu import workloads

    spec = workloads.layered_spec(seed=3, scale=0.05)
    eng = workloads.layered_engine(spec, "fp64")
    nid = workloads.layered_add(eng, spec, 40)
    eng.simulate(40)
    f = eng.slice_form()
    assert f["slices"]["kernels"] == 40 and f["own_state"] == 0 and f["own_bytes"] == 0
    eng.net_remove(nid)
    nid = workloads.layered_add(eng, spec, 5000)
    for _ in range(20):
        eng.simulate(100)
    f = eng.slice_form()
    assert f["own_state"] == 1 and f["slices"]["k_run_owned"] >= 1500 and f["own_bytes"] > 0
    eng.net_remove(nid)
    assert eng.slice_form()["own_bytes"] == 0
    eng.close()


@pytest.mark.parametrize("rates,one_weight,own", [
    (np.array([8e5]), True, True),                   # counts beyond the tabulated inputs, tables that are bisected
    (np.array([8e5, 0.0, 5e3]), False, True),        # ... with weights of their own, neurons without drive
    (np.linspace(1e3, 9e5, 40), True, True),         # more thresholds than shared memory holds
    (np.array([8e5, 1.1e6]), True, False),           # a mean too large for a table: the other forms
])
@pytest.mark.parametrize("precision", [_abi.NG_FP64, _abi.NG_FP32])
def test_drive_tables(rates, one_weight, own, precision):
    n, md = 997, 10
    idx = np.arange(n)

    def run(variant):
        eng = _plain(n, 20, md, precision=precision)
        eng.set_tuning(0, variant, -1, -1)
        w = np.full(n, 0.25) if one_weight else np.choose(idx % 3, [0.25, 0.5, -0.25])
        eng.set_poisson(rates[idx % len(rates)], w, np.full(n, md, dtype=np.int32), 3, 10**9, 21)
        eng.simulate(40 * md)
        st = eng.stats()
        out = _raster(eng) + (eng.get_var(0, "I_syn_ex"), eng.get_var(0, "I_syn_in"), np.array([st["drive_events"]]))
        f = eng.slice_form()
        eng.close()
        return out, f

    ref, got = run(0)[0], run(5)
    assert len(ref[0]) > 100 and ref[-1][0] > 10 * n
    for a, b in zip(ref, got[0]):
        np.testing.assert_array_equal(a, b)
    assert (got[1]["slices"]["k_run_owned"] == 40) == own


def test_automatic_choice_after_a_fixed_one():
    eng = _plain(2503, 30, 15)
    eng.set_tuning(0, 2, -1, -1)
    eng.simulate(300)
    assert eng.slice_form()["slices"]["k_run_owned"] == 0
    eng.set_tuning(1)
    eng.simulate(6000)
    f, t = eng.slice_form(), eng.tuned()
    got = _raster(eng)
    eng.close()
    assert f["slices"]["k_run_owned"] == 400 and t["state"] == "tuned" and t["update_variant"] == 5
    ref = _plain(2503, 30, 15)
    ref.set_tuning(0, 0, -1, -1)
    ref.simulate(6300)
    for a, b in zip(got, _raster(ref)):
        np.testing.assert_array_equal(a, b)
    ref.close()
