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


# group sizes and batch lengths on both sides of the iaf kernel's variants: 64-thread blocks below
# 37,888 neurons, input two steps ahead there from four steps on, and in large groups where the
# batch's accumulators exceed 100 MB (15 steps: 416,667 neurons)
@pytest.mark.parametrize("n,delay", [(1, 0.2), (63, 0.3), (65, 0.4), (37887, 0.3), (37887, 0.4), (37888, 0.4),
                                     (410000, 1.5), (420000, 1.5)])
def test_iaf_kernel_variants_match_oracle(n, delay):
    def run(api):
        api.SetKernelStatus("rnd_seed", 11)
        neuron = api.Create("iaf_psc_exp", n)
        pg = api.Create("poisson_generator")
        api.SetStatus(pg, "rate", 9000.0)
        api.Connect(pg, neuron, {"rule": "all_to_all"}, {"weight": 60.0, "delay": 1.0, "receptor": 0})
        api.ConnectFixedIndegreeGPU(neuron, neuron, 2, 40.0, delay, delay, receptor=1, seed=3)
        api.ActivateSpikeCount(neuron)
        api.Simulate(9.7)
        return (np.asarray(api.GetStatus(neuron, "spike_count")).ravel(),
                np.asarray(api.GetStatus(neuron, "V_m_rel"), dtype=np.float32).ravel())
    c, v = run(ngpu)
    co, vo = run(orc.Oracle())
    assert np.array_equal(c, co) and np.array_equal(v, vo)
    assert n < 1000 or co.sum() > 0


# both forms of the delivery kernel (parts and four edges in flight from 32 edges a segment on, while
# the batch's accumulators stay below 12 MB; whole segments otherwise) and every lane group
@pytest.mark.parametrize("n,k,hi", [(64, 31, 1.5), (64, 33, 1.5), (200, 40, 4.0), (52000, 33, 1.5)])
@pytest.mark.parametrize("group,prefetch", [(32, False), (16, True), (8, False)])
def test_delivery_forms_match_oracle(n, k, hi, group, prefetch):
    def run(api):
        api.SetKernelStatus("rnd_seed", 5)
        neuron = api.Create("iaf_psc_exp", n)
        pg = api.Create("poisson_generator")
        api.SetStatus(pg, "rate", 8000.0)
        api.Connect(pg, neuron, {"rule": "all_to_all"}, {"weight": 45.0, "delay": 1.0, "receptor": 0})
        api.ConnectFixedIndegreeGPU(neuron, neuron, k, 100.0 / k, 1.5, hi, receptor=0, seed=3)
        api.ActivateSpikeCount(neuron)
        api.Simulate(14.3)
        return (np.asarray(api.GetStatus(neuron, "spike_count")).ravel(),
                np.asarray(api.GetStatus(neuron, "V_m_rel"), dtype=np.float32).ravel())
    ngpu.SetDeliverGroup(group)
    ngpu.SetDeliverPrefetch(prefetch)
    c, v = run(ngpu)
    o = orc.Oracle()
    co, vo = run(o)
    assert co.sum() > 0 and np.array_equal(c, co) and np.array_equal(v, vo)
    assert ngpu.GetStats()["n_events"] == o.NEvents()


@pytest.mark.parametrize("n", [1036, 1037])
def test_step_model_in_thin_warps_matches_oracle(n):
    """The step model proposing in groups of one and of two neurons per warp."""
    from test_oracle_learn import random_params
    p = random_params(21)
    p[1461], p[1462] = np.float32(np.log(0.02)), 0.5

    def run(api):
        api.SetKernelStatus("rnd_seed", 11)
        neuron = api.Create("aeif_cond_beta_multisynapse", n, 4)
        api.SetStatus(neuron, {"E_rev": [0.0, 0.0, -85.0, -85.0]})
        pg = api.Create("poisson_generator")
        api.SetStatus(pg, "rate", 4000.0)
        api.Connect(pg, neuron, {"rule": "all_to_all"}, {"weight": 1.5, "delay": 1.0, "receptor": 0})
        api.ConnectFixedIndegreeGPU(neuron, neuron, 10, 0.1, 1.5, 1.5, receptor=1, seed=3)
        api.ActivateSpikeCount(neuron)
        if api is ngpu:
            ngpu.StepModelSet(p)
            ngpu.StepModelEnable(True)
        else:
            api.StepModelSet(p, enable=True)
        api.Simulate(12.0)
        return (np.asarray(api.GetStatus(neuron, "spike_count")).ravel(),
                np.asarray(api.GetStatus(neuron, "V_m"), dtype=np.float32).ravel())
    c, v = run(ngpu)
    co, vo = run(orc.Oracle())
    assert co.sum() > 0 and np.array_equal(c, co) and np.array_equal(v, vo)
