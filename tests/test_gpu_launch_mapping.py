"""The launch mapping that the engine chooses where no call sets one: what GetLaunchMapping reports
of it, and how Autotune starts from it and leaves it."""
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


def _aeif(n):
    neuron = ngpu.Create("aeif_cond_beta_multisynapse", n, 2)
    ngpu.SetStatus(neuron, {"E_rev": [0.0, -85.0], "I_e": 600.0})
    ngpu.ConnectFixedIndegreeGPU(neuron, neuron, 2, 0.1, 1.0, 1.5, receptor=0, seed=1)
    return neuron


def _iaf(n, lo=0.1, hi=0.5):
    neuron = ngpu.Create("iaf_psc_exp", n)
    ngpu.SetStatus(neuron, "I_e", 600.0)
    ngpu.ConnectFixedIndegreeGPU(neuron, neuron, 3, 1.0, lo, hi, receptor=0, seed=1)
    return neuron


# 64-thread blocks; beyond the neurons resident at once the hand-off and the capped kernel
@pytest.mark.parametrize("n,want", [(2000, (64, 0, 0, 0)), (150000, (64, 2, 1, 1))])
def test_automatic_aeif_mapping_is_reported(n, want):
    _aeif(n)
    ngpu.Simulate(1.0)
    m = ngpu.GetLaunchMapping()
    assert (m["update_threads"], m["update_occupancy"], m["update_trial_iter"], m["rk5_budget"]) == want


@pytest.mark.parametrize("n,lo,hi,forced,want", [(500, 0.1, 0.5, None, 1), (500, 1.0, 1.5, None, 0), (500, 1.0, 1.5, True, 1),
                                                 (500, 0.1, 0.5, False, 0), (500, 0.1, 19.3, True, 0)])
def test_persistent_loop_in_use_is_reported(n, lo, hi, forced, want):
    _iaf(n, lo, hi)
    if forced is not None:
        ngpu.SetPersistent(forced)
    ngpu.Simulate(2.0)
    assert ngpu.GetLaunchMapping()["persistent"] == want
    l0 = ngpu.GetLaunchCount()
    ngpu.Simulate(2.0)
    assert (ngpu.GetLaunchCount() - l0 == 2) == bool(want)


def test_autotune_leaves_short_calls_to_the_per_batch_kernels():
    """A single step after Autotune goes the way it goes without it: the loop that wins on long
    calls costs more there."""
    from workloads import microcircuit
    microcircuit(ngpu, scale=0.03)
    ngpu.Simulate(5.0)

    def launches(fn):
        l0 = ngpu.GetLaunchCount()
        fn()
        return ngpu.GetLaunchCount() - l0
    before = launches(ngpu.SimulationStep)
    ngpu.EndSimulation()
    assert ngpu.Autotune(50)["persistent"] == 1 and launches(lambda: ngpu.Simulate(2.0)) == 2
    assert launches(ngpu.SimulationStep) == before > 2
    ngpu.EndSimulation()


def test_autotune_keeps_what_is_automatic():
    """Settings without influence on a network (here the aeif ones, without an aeif group) stay as
    they were."""
    _iaf(500, 1.0, 1.5)
    ngpu.Simulate(2.0)
    keys = ["update_threads", "update_occupancy", "update_trial_iter", "rk5_budget"]
    before = ngpu.GetLaunchMapping()
    after = ngpu.Autotune(20)
    assert [before[k] for k in keys] == [after[k] for k in keys]


def test_failed_autotune_leaves_the_settings():
    """A trial that fails (its barriers wait for one block too many) ends the call with the
    settings of before; the loop itself stays off, as after any such failure."""
    _iaf(500)
    ngpu.Simulate(2.0)
    before = ngpu.GetLaunchMapping()
    ngpu._lib.NGPU_TestBarrierTimeout(1)
    with pytest.raises(ValueError, match="timed out"):
        ngpu.Autotune(20)
    ngpu._lib.NGPU_TestBarrierTimeout(0)
    after = ngpu.GetLaunchMapping()
    assert before.pop("persistent") == 1 and after.pop("persistent") == 0
    assert before == after


@pytest.mark.parametrize("k,hi,loop", [(2400, 0.1, True), (2600, 0.1, False), (2400, 0.2, True), (2600, 0.2, False),
                                       (3300, 0.3, True), (4200, 0.3, False)])
def test_long_first_segments_stay_with_the_per_batch_kernels(k, hi, loop):
    """Edges of one and two steps' delay are delivered by the spiking neuron's own block: above 2500 of
    them a source the loop is not chosen.  The results are the same either way."""
    def run(setting):
        ngpu.Reset()
        ngpu.SetVerbosityLevel(0)
        n = ngpu.Create("iaf_psc_exp", 100)
        ngpu.SetStatus(n, "I_e", 600.0)
        ngpu.ConnectFixedIndegreeGPU(n, n, k, 0.01, 0.1, hi, receptor=0, seed=1)
        ngpu.ActivateSpikeCount(n)
        if setting is not None:
            ngpu.SetPersistent(setting)
        ngpu.Simulate(1.0)
        m = ngpu.GetLaunchMapping()["persistent"]
        ngpu.Simulate(30.0)
        return m, np.asarray(ngpu.GetStatus(n, "spike_count")).ravel(), np.asarray(ngpu.GetStatus(n, "V_m_rel")).ravel()
    got, off, on = run(None), run(False), run(True)
    assert (got[0], off[0], on[0]) == (int(loop), 0, 1)
    assert got[1].sum() > 0
    for other in (off, on):
        assert np.array_equal(got[1], other[1]) and np.array_equal(got[2], other[2])


@pytest.mark.parametrize("ports,n,delay,want", [(5, 60, 1.0, (128, 0, 0, 4)), (20, 33, 0.3, (128, 0, 0, 4)), (6, 45, 0.1, (128, 0, 0, 0)),
                                                (1, 60, 0.1, (64, 0, 0, 0)), (1, 130000, 0.1, (128, 0, 0, 4))])
def test_one_port_and_any_number_of_ports(ports, n, delay, want):
    """The mappings of their own, against the oracle where that is quick."""
    def run(api):
        api.SetKernelStatus("rnd_seed", 4)
        neuron = api.Create("aeif_cond_beta_multisynapse", n, ports)
        api.SetStatus(neuron, {"E_rev": [-85.0 if p % 3 == 2 else 0.0 for p in range(ports)],
                               "tau_decay": [2.0 + p for p in range(ports)], "tau_rise": [1.0 + 0.5 * p for p in range(ports)]})
        pg = api.Create("poisson_generator")
        api.SetStatus(pg, "rate", 8000.0)
        api.Connect(pg, neuron, {"rule": "all_to_all"}, {"weight": 1.0, "delay": 1.0, "receptor": 0})
        for p in range(ports):
            api.ConnectFixedIndegreeGPU(neuron, neuron, 3, 0.2, delay, delay, receptor=p, seed=p + 1)
        api.ActivateSpikeCount(neuron)
        api.Simulate(20.0 if n < 1000 else 1.0)
        return (np.asarray(api.GetStatus(neuron, "spike_count")).ravel(),
                np.asarray(api.GetStatus(neuron, "V_m"), dtype=np.float32).ravel())
    c, v = run(ngpu)
    m = ngpu.GetLaunchMapping()
    assert (m["update_threads"], m["update_occupancy"], m["update_trial_iter"], m["rk5_budget"]) == want
    if n < 1000:
        co, vo = run(orc.Oracle())
        assert co.sum() > 0 and np.array_equal(c, co) and np.array_equal(v, vo)


@pytest.mark.parametrize("n,want", [(50000, (64, 0, 0, 0)), (76000, (64, 2, 1, 1))])
def test_both_sides_of_the_resident_neurons_match_oracle(n, want):
    """Groups below and above the neurons that are resident at once (56,832 for two ports): no
    hand-off, and the capped kernel with the straggler kernel."""
    def run(api):
        api.SetKernelStatus("rnd_seed", 6)
        neuron = api.Create("aeif_cond_beta_multisynapse", n, 2)
        api.SetStatus(neuron, {"E_rev": [0.0, -85.0]})
        pg = api.Create("poisson_generator")
        api.SetStatus(pg, "rate", 8000.0)
        api.Connect(pg, neuron, {"rule": "all_to_all"}, {"weight": 2.0, "delay": 0.1, "receptor": 0})
        api.ConnectFixedIndegreeGPU(neuron, neuron, 2, 0.3, 1.0, 1.5, receptor=1, seed=5)
        api.ActivateSpikeCount(neuron)
        api.Simulate(6.0)
        return (np.asarray(api.GetStatus(neuron, "spike_count")).ravel(),
                np.asarray(api.GetStatus(neuron, "V_m"), dtype=np.float32).ravel())
    c, v = run(ngpu)
    m = ngpu.GetLaunchMapping()
    assert (m["update_threads"], m["update_occupancy"], m["update_trial_iter"], m["rk5_budget"]) == want
    co, vo = run(orc.Oracle())
    assert co.sum() > 1000 and np.array_equal(c, co) and np.array_equal(v, vo)
