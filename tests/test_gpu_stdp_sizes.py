"""The plasticity kernels at the edges of their work splits against the oracle: in-degrees around
the 32-edge chunks and the eight warps' round (256 edges), target counts around the 32 targets of
a block, many spikes arriving in one step (more than a delay group's warps), single targets.

Tolerance: the engine's FP64 exp and pow come from CUDA, the oracle's from the C library; both
are within a few last places of FP64, so an updated weight differs by at most one FP32 rounding
(6e-8 relative) per update; each edge is updated at most ten times here: 6e-7."""
import numpy as np
import pytest

import nestgpu as ngpu
import oracle as orc

pytestmark = pytest.mark.gpu


def _weights(api, ids):
    st = getattr(api, "GetConnStatusList", None)
    return np.asarray(st(ids, "weight") if st is not None else api.GetStatus(ids, "weight"), dtype=np.float32)


def _run(api, n_pre, n_post):
    syn = api.CreateSynGroup("stdp", {"tau_plus": 20.0, "tau_minus": 20.0, "lambda": 0.1, "alpha": 1.0,
                                      "mu_plus": 0.5, "mu_minus": 0.6, "Wmax": 2.0})
    sg = api.Create("spike_generator", 2)
    pre = api.Create("iaf_psc_exp", n_pre)
    post = api.Create("iaf_psc_exp", n_post)
    api.SetStatus([sg[0]], {"spike_times": [2.0, 9.0, 21.0]})
    api.SetStatus([sg[1]], {"spike_times": [5.0, 14.0, 23.5]})
    api.Connect([sg[0]], pre, {"rule": "all_to_all"}, {"weight": 5000.0, "delay": 1.0, "receptor": 0})
    api.Connect([sg[1]], post, {"rule": "all_to_all"}, {"weight": 5000.0, "delay": 1.0, "receptor": 0})
    api.Connect(pre, post, {"rule": "all_to_all"}, {"weight": 1.0, "delay": 1.2, "receptor": 1, "synapse_group": syn})
    api.Simulate(32.0)
    return _weights(api, api.GetConnections(pre, post))


@pytest.mark.parametrize("n_pre,n_post", [(1, 1), (31, 33), (32, 32), (33, 65), (257, 3), (700, 2)])
def test_plasticity_kernel_sizes(n_pre, n_post):
    ngpu.Reset()
    ngpu.SetVerbosityLevel(0)
    w = _run(ngpu, n_pre, n_post)
    ngpu.Reset()
    wo = _run(orc.Oracle(), n_pre, n_post)
    assert w.size == n_pre * n_post and np.all(w != 1.0)
    assert np.allclose(w, wo, rtol=6e-7, atol=0.0)
