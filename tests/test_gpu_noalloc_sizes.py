"""ng_simulate_noalloc at the sizes where its launch changes (one neuron,
fewer neurons than a CTA of the cluster has warps, the largest network of the
one-launch form, the next larger one, which runs slice by slice), rows longer
and shorter than a warp's share, in one call and in continued calls that stop
inside slices: raster and V_m equal ng_simulate's bit for bit."""

import math

import numpy as np
import pytest

from test_zz_no_alloc import _NoAlloc, _assert_same, _run_engine

pytestmark = pytest.mark.gpu


def _net(n, md, maxd):
    rng = np.random.default_rng(n)
    deg = rng.integers(0, min(300, 2 * n) + 1, n)
    deg[::3] = rng.integers(0, 4, len(deg[::3]))
    row = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    nnz = int(row[-1])
    h, tau_m, C_m = (1.0 / 1000.0) * 100, 20.0, 250.0
    P33 = math.exp(-h / tau_m)
    return {
        "n": n, "P33": np.full(n, P33), "P30": np.full(n, 1 / C_m * (1 - P33) * tau_m),
        "V_th_rel": np.full(n, 20.0), "V_reset_rel": np.full(n, 10.0),
        "V_min_rel": np.full(n, -np.finfo(np.float64).max), "I_e": rng.uniform(300.0, 500.0, n),
        "refr": np.full(n, 20, dtype=np.int32), "V0": rng.uniform(0.0, 20.5, n), "row_ptr": row,
        "target": rng.integers(0, n, nnz).astype(np.int32), "weight": rng.choice([0.0625, 0.03125, -0.125], nnz),
        "delay": rng.integers(md, maxd + 1, nnz).astype(np.int32), "params": (C_m, tau_m, 2.0, 0.0, 20.0, 10.0),
        "min_delay": md, "max_delay": maxd,
    }


@pytest.mark.parametrize("n,md,maxd", [(1, 3, 3), (31, 15, 15), (1000, 7, 12), (8192, 20, 25), (8193, 20, 25)])
def test_noalloc_sizes(n, md, maxd):
    net = _net(n, md, maxd)
    steps = 8 * md + 3
    ref = _run_engine(net, steps)
    one = _NoAlloc(net)
    src, stamp, k, skipped = one.call(steps)
    assert k == len(src) and skipped == 0
    _assert_same((src, stamp, one.V.cpu().numpy()), ref)
    parts = _NoAlloc(net)
    at, got = 0, []
    for c in (2, md, 1, 3 * md - 1, steps):
        c = min(c, steps - at)
        s, t, _, _ = parts.call(c, at, 1 if at else 0)
        got.append((s, t))
        at += c
    _assert_same((np.concatenate([g[0] for g in got]), np.concatenate([g[1] for g in got]), parts.V.cpu().numpy()), ref)
