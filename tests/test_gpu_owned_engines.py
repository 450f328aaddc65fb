"""Engines of one process whose kernels (the target-owning slice kernel, the
target-tiled delivery) have layouts of different sizes: what one engine sets
up must not reach another.  Weights and drive are dyadic (or the form is fixed
point), so each engine's results equal, bit for bit, those of the same network
run alone."""

import threading

import numpy as np
import pytest

from nestgpu import _abi

from test_gpu_serving import PB_SIZES, _pb

pytestmark = pytest.mark.gpu

MD = 15
CALLS = (300, 150, 450)


def _engine(n, seed):
    rng = np.random.default_rng(seed)
    deg = rng.integers(20, 60, n)
    row = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    nnz = int(row[-1])
    src = np.repeat(np.arange(n), deg)
    eng = _abi.Engine([(_abi.NG_IAF_PSC_EXP, n)], 0.1, MD, MD)
    eng.set_tuning(0, 5, -1, -1)
    eng.set_var(0, "V_m_rel", rng.uniform(0.0, 14.5, n))
    eng.set_connections(row, rng.integers(0, n, nnz).astype(np.int32), np.where(src < 0.8 * n, 60.0, -240.0),
                        np.full(nnz, MD, dtype=np.int32))
    eng.set_recording(np.ones(n, dtype=np.uint8))
    eng.set_poisson(np.full(n, 11000.0), np.full(n, 48.0), np.full(n, MD, dtype=np.int32), 0, 10**9, seed)
    return eng


def _result(eng):
    s, t = eng.spikes()
    o = np.lexsort((s, t))
    out = [s[o], t[o]] + [eng.get_var(0, v) for v in ("V_m_rel", "I_syn_ex", "I_syn_in")]
    eng.close()
    return out


def _alone(n, seed):
    eng = _engine(n, seed)
    for k in CALLS:
        eng.simulate(k)
    return _result(eng)


def _assert_same(a, b):
    assert len(a[0]) > 20
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


# the larger layout first: the smaller one's set-up comes between its launches
@pytest.mark.parametrize("sizes", [(9001, 611), (611, 9001)])
def test_engines_in_turn(sizes):
    want = [_alone(n, n) for n in sizes]
    engines = [_engine(n, n) for n in sizes]
    for k in CALLS:
        for e in engines:
            e.simulate(k)
    for e, w in zip(engines, want):
        _assert_same(_result(e), w)


def test_engines_on_two_threads():
    sizes = (9001, 611)
    want = [_alone(n, n) for n in sizes]
    engines = [_engine(n, n) for n in sizes]
    failed = []

    def work(e):
        try:
            for k in CALLS:
                e.simulate(k)
        except Exception as ex:  # reported by the test's thread
            failed.append(ex)

    threads = [threading.Thread(target=work, args=(e,)) for e in engines]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for e, w in zip(engines, want):
        _assert_same(_result(e), w)


def test_tiled_engines():
    """The second engine's shorter delays give its tiles a smaller window."""
    n = sum(PB_SIZES)

    def engine(max_delay):
        return _abi.Engine([(_abi.NG_IAF_PSC_EXP, 20_000)], 0.1, 1, max_delay, precision=_abi.NG_FP32, serving=True,
                           max_networks=2, edge_capacity=30_000_000, max_abs_weight=1000.0,
                           tile_capacity=_abi.tile_table_entries(n, max_delay, False))

    def run(with_other):
        eng = engine(40)
        V0 = np.random.default_rng(8).uniform(0.0, 14.0, n)
        nid = eng.net_add(n, 600, 17, {"tau_syn_ex": 0.5, "tau_syn_in": 0.5, "V_m_rel": V0}, build=_pb(seed=21),
                          poisson=(np.full(n, 9000.0), 87.8, 15))
        other = engine(3) if with_other else None
        eng.simulate(600)
        s, t = eng.net_spikes(nid)
        o = np.lexsort((s, t))
        out = s[o], t[o], eng.net_get_var(nid, "V_m_rel", n)
        eng.close()
        if other:
            other.close()
        return out

    _assert_same(run(False), run(True))
