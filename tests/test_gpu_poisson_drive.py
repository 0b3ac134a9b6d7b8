"""Poisson generators drawn by a kernel of their own (networks in which some neuron has several
generators) against the oracle, bit for bit: batch lengths around the four-step Philox blocks,
edge counts around the kernel's 256-thread blocks, a mean count above 10 (split into chunks), a
generator with a time window, mixed numbers of generators per neuron, both receptors."""
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


def _net(api, model, n, gens, delay):
    api.SetKernelStatus("rnd_seed", 77)
    aeif = model.startswith("aeif")
    neuron = api.Create(model, n, 2)
    if model == "aeif_cond_beta_multisynapse":
        api.SetStatus(neuron, {"E_rev": [0.0, -85.0]})
    w = {"aeif_cond_beta_multisynapse": 0.8, "iaf_psc_exp": 40.0}[model]
    pg = api.Create("poisson_generator", gens)
    for i in range(gens):
        # the last generator's mean count per step is 12 (two chunks of 6)
        api.SetStatus([pg[i]], "rate", 120000.0 if i == gens - 1 else 900.0 / gens + 11.0 * i)
    if gens > 2:
        api.SetStatus([pg[1]], {"start": 3.0, "stop": 11.0})
    for i in range(gens):
        last = i == gens - 1
        # the last generator feeds part of the neurons only, with a small weight, on receptor 1
        api.Connect([pg[i]], neuron[0:max(1, n // 3)] if last else neuron, {"rule": "all_to_all"},
                    {"weight": -0.01 * w if last and not aeif else (0.002 * w if last else w), "delay": 1.0,
                     "receptor": 1 if last else 0})
    api.Connect(neuron, neuron, {"rule": "fixed_indegree", "indegree": min(4, n)}, {"weight": 0.2 * w, "delay": delay, "receptor": 0})
    api.ActivateSpikeCount(neuron)
    api.Simulate(17.3)
    api.Simulate(9.0)
    v = "V_m" if aeif else "V_m_rel"
    return (np.asarray(api.GetStatus(neuron, "spike_count")).ravel(),
            np.asarray(api.GetStatus(neuron, v), dtype=np.float32).ravel())


@pytest.mark.parametrize("delay", [0.1, 0.2, 0.4, 1.5, 4.0])
@pytest.mark.parametrize("model,n,gens", [("iaf_psc_exp", 1, 2), ("iaf_psc_exp", 257, 3),
                                          ("aeif_cond_beta_multisynapse", 129, 5)])
def test_several_generators_per_neuron_bitexact(model, n, gens, delay):
    c, v = _net(ngpu, model, n, gens, delay)
    co, vo = _net(orc.Oracle(), model, n, gens, delay)
    assert np.array_equal(c, co)
    assert np.array_equal(v, vo)


def test_persistent_loop_toggled_between_calls():
    """Turning the persistent step loop on and off between calls moves the draws between the
    kernels without repeating or dropping any."""
    def run(toggle):
        ngpu.Reset()
        ngpu.SetVerbosityLevel(0)
        neuron = ngpu.Create("iaf_psc_exp", 65)
        pg = ngpu.Create("poisson_generator", 3)
        ngpu.SetStatus(pg, "rate", 3000.0)
        ngpu.Connect(pg, neuron, {"rule": "all_to_all"}, {"weight": 40.0, "delay": 1.0, "receptor": 0})
        for on in toggle:
            ngpu.SetPersistent(on)
            ngpu.Simulate(5.0)
        return np.asarray(ngpu.GetStatus(neuron, "V_m_rel"))
    assert np.array_equal(run([False] * 4), run([False, True, False, True]))


# generators per neuron up to which the draws stay in the update kernel, by steps per batch
@pytest.mark.parametrize("batch,line", [(1, 4), (2, 2), (3, 1), (4, 1)])
@pytest.mark.parametrize("beyond", [0, 1])
def test_both_sides_of_the_line_bitexact(batch, line, beyond):
    """Neurons with none, one and up to the line's number of generators, or one more, in one group."""
    gens = line + beyond

    def run(api):
        api.SetKernelStatus("rnd_seed", 9)
        neuron = api.Create("iaf_psc_exp", 130)
        pg = api.Create("poisson_generator", gens)
        for i in range(gens):
            api.SetStatus([pg[i]], "rate", 12000.0 / gens + 300.0 * i)
            # neuron j has generators 0 .. j mod (gens + 1) - 1
            api.Connect([pg[i]], [neuron[j] for j in range(130) if j % (gens + 1) > i], {"rule": "all_to_all"},
                        {"weight": 70.0, "delay": 0.1 * (i + 1), "receptor": i % 2})
        api.Connect(neuron, neuron, {"rule": "fixed_indegree", "indegree": 3}, {"weight": 10.0, "delay": 0.1 * batch, "receptor": 0})
        api.ActivateSpikeCount(neuron)
        launches = 0
        for t in (10.0, 1.2):
            l0 = ngpu.GetLaunchCount() if api is ngpu else 0
            api.Simulate(t)
            launches = ngpu.GetLaunchCount() - l0 if api is ngpu else 0
        return (np.asarray(api.GetStatus(neuron, "spike_count")).ravel(),
                np.asarray(api.GetStatus(neuron, "V_m_rel"), dtype=np.float32).ravel(), launches)
    ngpu.SetPersistent(False)
    c, v, launches = run(ngpu)
    co, vo, _ = run(orc.Oracle())
    assert ngpu.GetBatchLength() == batch
    assert launches == 12 // batch * (3 if beyond else 2) + 1     # delivery, draws, update; the clock
    assert co.sum() > 0 and np.array_equal(c, co) and np.array_equal(v, vo)


@pytest.mark.parametrize("n,delay", [(37887, 0.3), (37888, 0.4), (113664, 1.5), (113665, 1.5)])
def test_one_neuron_with_more_generators(n, delay):
    """All neurons with one generator, a few in the middle with six: in large groups the single
    draws stay in the update kernel."""
    def run(api):
        api.SetKernelStatus("rnd_seed", 21)
        neuron = api.Create("iaf_psc_exp", n)
        pg = api.Create("poisson_generator", 6)
        api.SetStatus(pg, "rate", 9000.0)
        for i in range(6):
            api.Connect([pg[i]], neuron if i == 0 else neuron[n // 2:n // 2 + 3], {"rule": "all_to_all"},
                        {"weight": 60.0 if i == 0 else 9.0, "delay": 1.0, "receptor": 0})
        api.ConnectFixedIndegreeGPU(neuron, neuron, 2, 40.0, delay, delay, receptor=1, seed=3)
        api.ActivateSpikeCount(neuron)
        api.Simulate(9.7)
        return (np.asarray(api.GetStatus(neuron, "spike_count")).ravel(),
                np.asarray(api.GetStatus(neuron, "V_m_rel"), dtype=np.float32).ravel())
    c, v = run(ngpu)
    co, vo = run(orc.Oracle())
    assert co.sum() > 0 and np.array_equal(c, co) and np.array_equal(v, vo)


def test_few_generators_do_not_keep_the_loop_away():
    """One-step batches: up to four generators per neuron the loop draws them, beyond that the
    per-batch kernels run."""
    for gens, loop in ((4, 1), (5, 0)):
        ngpu.Reset()
        ngpu.SetVerbosityLevel(0)
        neuron = ngpu.Create("iaf_psc_exp", 65)
        pg = ngpu.Create("poisson_generator", gens)
        ngpu.SetStatus(pg, "rate", 3000.0)
        ngpu.Connect(pg, neuron, {"rule": "all_to_all"}, {"weight": 40.0, "delay": 1.0, "receptor": 0})
        ngpu.Connect(neuron, neuron, {"rule": "fixed_indegree", "indegree": 3}, {"weight": 10.0, "delay": 0.1, "receptor": 0})
        ngpu.Simulate(1.0)
        assert ngpu.GetLaunchMapping()["persistent"] == loop
