"""aeif_cond_alpha's update, whose lanes walk a slice's lags on their own: long
slices (more spikes of a CTA's neurons than its list holds), slices of one step
and a size that fills no CTA give, in whole slices, the raster and state of the
same steps run in partial slices of a few lags, bit for bit."""

import numpy as np
import pytest

from nestgpu import _abi

pytestmark = pytest.mark.gpu


def _run(precision, n, md, t_ref, calls):
    rng = np.random.default_rng(n + md)
    deg = rng.integers(5, 30, n)
    row = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    nnz = int(row[-1])
    eng = _abi.Engine([(_abi.NG_AEIF_COND_ALPHA, n)], 0.1, md, 2 * md, precision=precision)
    eng.set_var(0, "tau_syn_ex", np.full(n, 1.0))
    eng.set_var(0, "t_ref", np.full(n, t_ref))
    eng.set_var(0, "V_m", rng.uniform(-70.6, -52.0, n))
    eng.set_var(0, "I_e", np.where(np.arange(n) % 3 == 0, 4000.0, 300.0))
    eng.set_connections(row, rng.integers(0, n, nnz).astype(np.int32), rng.choice([1.0, 0.5, -2.0, -4.0], nnz),
                        rng.integers(md, 2 * md + 1, nnz).astype(np.int32))
    eng.set_recording(np.ones(n, dtype=np.uint8))
    eng.set_poisson(np.full(n, 15000.0), np.full(n, 1.0), np.full(n, md, dtype=np.int32), 0, 10**9, 5)
    for k in calls:
        eng.simulate(k)
    s, t = eng.spikes()
    o = np.lexsort((s, t))
    out = [s[o], t[o]] + [eng.get_var(0, v) for v in ("V_m", "w", "g_ex", "integration_step")]
    eng.close()
    return out


@pytest.mark.parametrize("precision,n,md,t_ref", [
    (_abi.NG_FP64, 131, 100, 0.0), (_abi.NG_FP32, 131, 100, 0.0), (_abi.NG_FP64, 65, 15, 2.0), (_abi.NG_FP64, 200, 1, 0.0),
])
def test_aeif_whole_slices_equal_partial_ones(precision, n, md, t_ref):
    steps = 4 * md if md > 1 else 60
    whole = _run(precision, n, md, t_ref, [steps])
    part = _run(precision, n, md, t_ref, _parts(steps))
    assert len(whole[0]) > n // 8
    for a, b in zip(whole, part):
        np.testing.assert_array_equal(a, b)


def _parts(steps):
    out, at = [], 0
    while at < steps:
        out.append(min(1 + len(out) % 4, steps - at))
        at += out[-1]
    return out
