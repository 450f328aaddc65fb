"""ng_simulate_noalloc's one-launch form at the sizes where its shares of 16
CTAs change (fewer neurons than CTAs, CTAs left empty, one neuron past a whole
share, a last CTA that is not full), in busy networks: raster and V_m equal
ng_simulate's bit for bit."""

import numpy as np
import pytest

from test_gpu_noalloc_sizes import _net
from test_zz_no_alloc import _NoAlloc, _assert_same, _run_engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,md,maxd", [(15, 4, 9), (17, 15, 15), (513, 9, 9), (4097, 5, 20), (8177, 10, 10)])
def test_noalloc_cluster_shares(n, md, maxd):
    net = _net(n, md, maxd)
    net["I_e"] = np.linspace(400.0, 1500.0, n)    # up to 250 Hz
    steps = 30 * md + 2
    ref = _run_engine(net, steps)
    assert len(ref[0]) > n // 2
    run = _NoAlloc(net)
    at, got = 0, []
    for c in (4 * md + 1, md - 1, 13 * md, steps):
        c = min(c, steps - at)
        s, t, k, skipped = run.call(c, at, 1 if at else 0)
        assert k == len(s) and skipped == 0
        got.append((s, t))
        at += c
    _assert_same((np.concatenate([g[0] for g in got]), np.concatenate([g[1] for g in got]), run.V.cpu().numpy()), ref)
