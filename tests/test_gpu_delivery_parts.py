"""Delivery of long segments in parts, thin warps of small groups and small iaf blocks against
the oracle, bit for bit: segment lengths around the parts' limits (128 edges, sixteen parts) and
neuron counts around the steps of the neurons-per-warp rule (1036 neurons at one per warp)."""
import numpy as np
import pytest

import nestgpu as ngpu
import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def fresh_engine():
    ngpu.Reset()
    ngpu.SetVerbosityLevel(0)
    yield
    ngpu.Reset()


def _net(api, model, n, k, w):
    api.SetKernelStatus("rnd_seed", 11)
    neuron = api.Create(model, n, 2)
    if model.startswith("aeif_cond"):
        api.SetStatus(neuron, {"E_rev": [0.0, -85.0]})
    pg = api.Create("poisson_generator")
    api.SetStatus(pg, "rate", 8000.0)
    api.Connect(pg, neuron, {"rule": "all_to_all"}, {"weight": w[0], "delay": 1.0, "receptor": 0})
    h = max(1, n // 2)
    api.ConnectFixedIndegreeGPU(neuron[0:h], neuron, k, w[1] / k, 1.5, 1.5, receptor=0, seed=3)
    api.ActivateSpikeCount(neuron)
    api.Simulate(31.7)
    v = "V_m_rel" if model == "iaf_psc_exp" else "V_m"
    return (np.asarray(api.GetStatus(neuron, "spike_count")).ravel(),
            np.asarray(api.GetStatus(neuron, v), dtype=np.float32).ravel())


# segments of about 2 k edges (half of the neurons are sources)
@pytest.mark.parametrize("n,k", [(64, 63), (64, 65), (100, 129), (40, 700), (33, 2100), (257, 300)])
def test_segment_parts_match_oracle(n, k):
    c, v = _net(ngpu, "iaf_psc_exp", n, k, (45.0, 300.0))
    o = orc.Oracle()
    co, vo = _net(o, "iaf_psc_exp", n, k, (45.0, 300.0))
    assert co.sum() > 0 and np.array_equal(c, co)
    assert np.array_equal(v, vo)
    assert ngpu.GetStats()["n_events"] == o.NEvents()


@pytest.mark.parametrize("n", [1, 31, 1036, 1037, 2073])
def test_thin_warps_match_oracle(n):
    c, v = _net(ngpu, "aeif_cond_beta_multisynapse", n, 10, (0.4, 2.0))
    co, vo = _net(orc.Oracle(), "aeif_cond_beta_multisynapse", n, 10, (0.4, 2.0))
    assert co.sum() > 0 and np.array_equal(c, co)
    assert np.array_equal(v, vo)
