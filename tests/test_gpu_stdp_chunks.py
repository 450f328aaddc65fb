"""stdp_pl_synapse_hom rows at the edges of the delivery's 256-connection
chunks (0, 1, 255, 256, 257 and 600 connections per source; several spikes of
a source in a slice) and targets whose histories flush over several chunks of
incoming connections: raster equal to the oracle's, weights within rtol 1e-10
(exp and pow of device and host may differ in the last bit)."""

import numpy as np
import pytest

from nestgpu import _abi

from test_gpu_stdp import _engine_run, _oracle_run, _spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("md,maxd", [(12, 12), (6, 20)])
def test_stdp_chunk_edges(md, maxd):
    sp = _spec(_abi.NG_IAF_PSC_EXP, md, maxd, n=900, seed=17)
    rng = np.random.default_rng(4)
    pdeg = np.resize([0, 1, 255, 256, 257, 600], 300)
    psrc = np.repeat(np.arange(300), pdeg)
    # two targets in five connections are among 40 neurons: long incoming lists
    ptgt = np.where(rng.random(len(psrc)) < 0.4, rng.integers(0, 40, len(psrc)), rng.integers(0, 900, len(psrc)))
    sp.update(psrc=psrc, ptgt=ptgt, pd=rng.integers(md, maxd + 1, len(psrc)), n_pl=300,
              pw=rng.uniform(0.5, 3.0, len(psrc)), drive=(20000.0, 16.0))
    es, et, eV, ew = _engine_run(_abi.NG_IAF_PSC_EXP, sp, _abi.NG_FP64, [5, 31, 11964])
    os_, ot, oV, ow = _oracle_run(_abi.NG_IAF_PSC_EXP, sp, 12000)
    assert np.bincount(es, minlength=900).max() > 48      # histories of 64 entries were flushed
    np.testing.assert_array_equal(es, os_)
    np.testing.assert_array_equal(et, ot)
    np.testing.assert_allclose(eV, oV, rtol=1e-10, atol=1e-10)
    np.testing.assert_allclose(ew, ow, rtol=1e-10)
