"""The persistent step loop of iaf_psc_exp networks against the oracle and the per-batch kernels,
bit for bit: neuron counts around the blocks and at the loop's capacity, delay ranges from one
step to its largest number of delay groups (first total delays of one, two and more steps, which
take different paths), calls of one, two and three steps, and turns between the two forms."""
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


def _net(api, n, lo, hi, k=20):
    """Two populations of about n / 3 and 2 n / 3 neurons, delays lo .. hi ms."""
    api.SetKernelStatus("rnd_seed", 5)
    na = max(1, n // 3)
    a = api.Create("iaf_psc_exp", na)
    b = api.Create("iaf_psc_exp", max(1, n - na))
    api.SetStatus(b, {"tau_ex": 0.7, "I_e": 300.0})
    pg = api.Create("poisson_generator", 2)
    api.SetStatus(pg, "rate", 9000.0)
    api.SetStatus([pg[1]], {"start": 2.0, "stop": 14.0})
    api.Connect([pg[0]], a, {"rule": "all_to_all"}, {"weight": 60.0, "delay": 1.0, "receptor": 0})
    api.Connect([pg[1]], b, {"rule": "all_to_all"}, {"weight": 60.0, "delay": 1.0, "receptor": 0})
    for s, src in enumerate((a, b)):
        for t, tgt in enumerate((a, b)):
            api.ConnectFixedIndegreeGPU(src, tgt, k, 20.0 if s == 0 else -15.0, lo, hi, receptor=s, seed=10 + 2 * s + t)
    api.ActivateSpikeCount(a)
    api.ActivateSpikeCount(b)
    return a, b


def _state(api, pops):
    return (np.concatenate([np.asarray(api.GetStatus(p, "spike_count")).ravel() for p in pops]),
            np.concatenate([np.asarray(api.GetStatus(p, "V_m_rel"), dtype=np.float32).ravel() for p in pops]))


def _count_launches(fn):
    l0 = ngpu.GetLaunchCount()
    fn()
    return ngpu.GetLaunchCount() - l0


@pytest.mark.parametrize("n,lo,hi", [(2, 0.1, 0.1), (147, 0.1, 0.2), (149, 0.1, 3.0), (1000, 0.2, 0.2), (1000, 0.2, 1.7),
                                     (700, 0.3, 2.0), (300, 1.5, 1.5), (900, 0.1, 19.2)])
def test_delay_ranges_match_oracle(n, lo, hi):
    ngpu.SetPersistent(True)
    pops = _net(ngpu, n, lo, hi)
    o = orc.Oracle()
    opops = _net(o, n, lo, hi)
    for t in (20.0, 0.1, 0.2, 0.3, 13.7):
        assert _count_launches(lambda: ngpu.Simulate(t)) == 2
        o.Simulate(t)
    c, v = _state(ngpu, pops)
    co, vo = _state(o, opops)
    assert co.sum() > 0 and np.array_equal(c, co)
    assert np.array_equal(v, vo)
    assert ngpu.GetStats()["n_events"] == o.NEvents() and ngpu.GetStats()["status"] == 0


@pytest.mark.parametrize("n,hi,loop", [(576 * 148, 1.0, True), (576 * 148 + 1, 1.0, False), (400, 19.2, True),
                                       (400, 19.3, False)])
def test_capacity_and_what_lies_beyond_it(n, hi, loop):
    """The largest network of the loop (its two generators take no thread), one neuron more, and
    one delay group too many (these two run in the per-batch kernels) equal the per-batch kernels."""
    res = []
    for pers in (True, False):
        ngpu.Reset()
        ngpu.SetVerbosityLevel(0)
        ngpu.SetPersistent(pers)
        pops = _net(ngpu, n, 0.1, hi, k=5)
        launches = _count_launches(lambda: ngpu.Simulate(12.0))
        assert (launches == 2) == (pers and loop)
        res.append(_state(ngpu, pops) + (ngpu.GetStats()["n_events"],))
    assert res[0][0].sum() > 0 and all(np.array_equal(x, y) for x, y in zip(*res))


def test_turns_between_the_forms():
    """Forced persistent calls, per-batch calls and single steps, spikes in flight at every change,
    give what the per-batch kernels alone give."""
    def run(modes):
        ngpu.Reset()
        ngpu.SetVerbosityLevel(0)
        pops = _net(ngpu, 500, 0.1, 2.9)
        for m in modes:
            ngpu.SetPersistent(m)
            ngpu.Simulate(4.0)
            for _ in range(3):
                ngpu.SimulationStep()
            ngpu.EndSimulation()
            ngpu.Simulate(0.7)
        return _state(ngpu, pops) + (ngpu.GetStats()["n_events"],)
    want = run([False] * 4)
    assert want[0].sum() > 100
    for modes in ([True] * 4, [True, False, True, False]):
        assert all(np.array_equal(x, y) for x, y in zip(run(modes), want))


def test_automatic_choice_by_call_length():
    """Without a call to SetPersistent: the loop from four steps a call on, shorter calls and single
    steps per batch, on the same ring and accumulators; what the per-batch kernels alone give."""
    def run(auto):
        ngpu.Reset()
        ngpu.SetVerbosityLevel(0)
        pops = _net(ngpu, 500, 0.1, 2.9)
        if not auto:
            ngpu.SetPersistent(False)
        loops = []
        for t in (4.0, 0.3, 0.4, 1.1, 0.2, 0.1, 5.0, 0.3, 2.0):
            loops.append(_count_launches(lambda: ngpu.Simulate(t)) == 2)
            ngpu.SimulationStep()
            ngpu.EndSimulation()
        return _state(ngpu, pops) + (ngpu.GetStats()["n_events"],), loops
    (got, loops), (want, none) = run(True), run(False)
    assert loops == [True, False, True, True, False, False, True, False, True] and not any(none)
    assert want[0].sum() > 50 and all(np.array_equal(x, y) for x, y in zip(got, want))


def test_two_networks_in_two_threads():
    """Two host threads run a network each at the same time (one engine per thread): their
    persistent launches share the GPU and the results are those of each network alone in the
    per-batch kernels."""
    import threading

    def run(out, key):
        ngpu.SetOnException(1)     # error handling is per thread
        ngpu.SetVerbosityLevel(0)
        pops = _net(ngpu, 800 + key, 0.1, 2.0)
        if out is alone:
            ngpu.SetPersistent(False)
        for _ in range(20):
            ngpu.Simulate(5.0)
        out[key] = _state(ngpu, pops)
        ngpu.Reset()

    alone, both = {}, {}
    for key in (0, 1):
        t = threading.Thread(target=run, args=(alone, key))
        t.start()
        t.join()
    threads = [threading.Thread(target=run, args=(both, key)) for key in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for key in (0, 1):
        assert alone[key][0].sum() > 0
        assert all(np.array_equal(x, y) for x, y in zip(alone[key], both[key]))


@pytest.mark.parametrize("forced", [None, True])
def test_blocks_that_cannot_all_start(forced):
    """A launch whose blocks do not all start (here its gate waits for one block too many) changes
    nothing and its steps run per batch: counts, potentials, records and the time are those of the
    per-batch kernels alone, spikes in flight included, and the next call is a loop again."""
    def run(modes):
        ngpu.Reset()
        ngpu.SetVerbosityLevel(0)
        pops = _net(ngpu, 400, 0.1, 2.0)
        rec = ngpu.CreateRecord("", ["V_m_rel", "spike"], [pops[0][0], pops[1][3]], [0, 0])
        launches = []
        for m in modes:
            if modes[0] is None:
                ngpu.SetPersistent(False)
            elif forced:
                ngpu.SetPersistent(True)
            ngpu._lib.NGPU_TestLoopStart(m or 0)
            launches.append(_count_launches(lambda: ngpu.Simulate(4.0)))
            if forced:
                ngpu.SimulationStep()
                ngpu.EndSimulation()
        ngpu._lib.NGPU_TestLoopStart(0)
        return _state(ngpu, pops) + (ngpu.GetStats()["n_events"], np.asarray(ngpu.GetRecordData(rec))), launches
    want, _ = run([None] * 4)
    got, launches = run([0, 2, 0, 2])
    assert want[0].sum() > 50 and all(np.array_equal(x, y) for x, y in zip(got, want))
    assert launches[0] == launches[2] == 2 and min(launches[1], launches[3]) > 2
    assert ngpu.GetStats()["status"] == 0


def test_refused_launch():
    """A refused cooperative launch: the engine's own choice goes on per batch and says so, a loop
    that was asked for fails; SetPersistent brings the loop back."""
    ngpu.SetPersistent(False)
    pops = _net(ngpu, 400, 0.1, 2.0)
    ngpu.Simulate(8.0)
    want = _state(ngpu, pops)
    ngpu.Reset()
    ngpu.SetVerbosityLevel(0)
    pops = _net(ngpu, 400, 0.1, 2.0)
    ngpu.Simulate(4.0)
    assert ngpu.GetLaunchMapping()["persistent"] == 1
    ngpu._lib.NGPU_TestLoopStart(1)
    ngpu.Simulate(4.0)
    assert all(np.array_equal(x, y) for x, y in zip(_state(ngpu, pops), want))
    assert ngpu.GetLaunchMapping()["persistent"] == 0
    ngpu.SetPersistent(True)
    with pytest.raises(ValueError, match="cooperative launch"):
        ngpu.Simulate(4.0)
    ngpu._lib.NGPU_TestLoopStart(0)
    ngpu.EndSimulation()
    assert _count_launches(lambda: ngpu.Simulate(4.0)) == 2


def test_generators_take_no_place_in_the_loop():
    """More generator nodes than the loop has threads, beside a network that fits it."""
    def run(pers):
        ngpu.Reset()
        ngpu.SetVerbosityLevel(0)
        pops = _net(ngpu, 300, 0.1, 2.0)
        ngpu.Create("poisson_generator", 576 * 148)
        if not pers:
            ngpu.SetPersistent(False)
        launches = _count_launches(lambda: ngpu.Simulate(8.0))
        return _state(ngpu, pops), launches
    (got, launches), (want, _) = run(True), run(False)
    assert launches == 2
    assert want[0].sum() > 0 and all(np.array_equal(x, y) for x, y in zip(got, want))


def test_table_of_the_loop_follows_the_settings():
    """What the loop's argument table holds changes between calls: parameters (uniform ones become
    arrays), recording, generator rates; against the per-batch kernels."""
    def run(pers):
        ngpu.Reset()
        ngpu.SetVerbosityLevel(0)
        pops = _net(ngpu, 400, 0.1, 2.0)
        if not pers:
            ngpu.SetPersistent(False)
        rec = ngpu.CreateRecord("", ["V_m_rel"], [pops[0][1]], [0])
        ngpu.Simulate(3.0)
        ngpu.SetStatus(pops[1], "I_e", 350.0)
        ngpu.Simulate(3.0)
        ngpu.SetNeuronScalParam(pops[0][5], 3, "I_e", 420.0)
        ngpu.Simulate(3.0)
        ngpu.SetGraphSteps(50)
        ngpu.Simulate(3.0)
        assert (ngpu.GetLaunchMapping()["persistent"] == 1) == pers
        return _state(ngpu, pops) + (np.asarray(ngpu.GetRecordData(rec)),)
    got, want = run(True), run(False)
    assert want[0].sum() > 20 and all(np.array_equal(x, y) for x, y in zip(got, want))


@pytest.mark.parametrize("k,lo,hi", [(62, 0.1, 0.1), (66, 0.1, 0.1), (500, 0.1, 1.0), (700, 0.1, 1.0), (130, 0.3, 0.3), (9, 0.1, 1.7)])
def test_segment_lengths_match_oracle(k, lo, hi):
    """Mean segments around 64 edges, where the delivery warps go from eight lanes a segment to a
    warp, and longer ones than a warp has in flight (128 edges)."""
    def run(api):
        api.SetKernelStatus("rnd_seed", 8)
        n = api.Create("iaf_psc_exp", 300)
        pg = api.Create("poisson_generator")
        api.SetStatus(pg, "rate", 12000.0)
        api.Connect(pg, n, {"rule": "all_to_all"}, {"weight": 45.0, "delay": 1.0, "receptor": 0})
        api.ConnectFixedIndegreeGPU(n, n, k, 60.0 / k, lo, hi, receptor=0, seed=2)
        api.ActivateSpikeCount(n)
        api.Simulate(25.0)
        return _state(api, [n])
    ngpu.SetPersistent(True)
    got = run(ngpu)
    o = orc.Oracle()
    want = run(o)
    assert ngpu.GetLaunchMapping()["persistent"] == 1
    assert want[0].sum() > 50 and all(np.array_equal(x, y) for x, y in zip(got, want))
    assert ngpu.GetStats()["n_events"] == o.NEvents()


def test_generators_of_all_kinds_match_oracle():
    """One generator on receptor 1, one with a mean count above ten, one that is off at first, several
    per neuron; recorded spike times."""
    def run(api):
        api.SetKernelStatus("rnd_seed", 12)
        n = api.Create("iaf_psc_exp", 120)
        pg = api.Create("poisson_generator", 5)
        for i, (rate, receptor, w) in enumerate([(9000.0, 0, 50.0), (9000.0, 1, 50.0), (130000.0, 1, 4.0), (9000.0, 0, 55.0),
                                                 (4000.0, 0, 60.0)]):
            api.SetStatus([pg[i]], "rate", rate)
            api.Connect([pg[i]], n[24 * i:24 * i + 24], {"rule": "all_to_all"}, {"weight": w, "delay": 1.0, "receptor": receptor})
        api.SetStatus([pg[3]], {"start": 4.0})
        api.Connect([pg[0]], n[96:120], {"rule": "all_to_all"}, {"weight": 30.0, "delay": 0.5, "receptor": 1})
        api.ConnectFixedIndegreeGPU(n, n, 20, 8.0, 0.1, 1.0, receptor=0, seed=2)
        api.ActivateSpikeCount(n)
        api.ActivateRecSpikeTimes(n, 200)
        api.Simulate(17.0)
        api.Simulate(9.0)
        return _state(api, [n]) + (np.concatenate([np.asarray(t, dtype=np.float32) for t in api.GetRecSpikeTimes(n)]),)
    ngpu.SetPersistent(True)
    got, want = run(ngpu), run(orc.Oracle())
    assert ngpu.GetLaunchMapping()["persistent"] == 1
    assert want[0].sum() > 100 and all(np.array_equal(x, y) for x, y in zip(got, want))
