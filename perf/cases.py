"""Performance cases of the spiking engine: what a user's simulation script has it do, through
the public nestgpu module, from single closed-loop steps of a small network to 1e9 synapses.

Every case is a network that a script has built and run in (prepare) and one call, or a short
series of calls, that advances it and reads its results (run).  All engine settings are the
defaults.  The engine keeps one network per host thread, so each prepared network lives on a
thread of its own and `run` hands it the pass; one pass is then exactly the calls that a
single-network script makes.

Families (the "kind" of a case):
  steps     a closed loop: SimulationStep and a read of some membrane potentials, step by step
  adex      aeif_cond_beta_multisynapse, excitatory and inhibitory sources drawn per target,
            delays on a range, Poisson drive (one generator, or many independent ones)
  learned   the same with four receptors of per-neuron time constants and the step model on
  hetero    another aeif model with per-neuron parameters, spike times recorded and read
  brunel    iaf_psc_exp, one delay, Poisson drive, a multimeter on ten neurons
  layers    eight iaf_psc_exp populations with the layered microcircuit's connection
            probabilities; delays start at one time step
  stdp      iaf_psc_exp with plastic excitatory synapses
  ensemble  many independent networks of uneven size, both models, advanced together
"""
import os
import queue
import sys
import threading

import numpy as np

_PKG = os.path.join(os.getcwd(), "nest-gpu_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import nestgpu as ngpu  # noqa: E402
from ensemble import build_ensemble, ensemble_spec  # noqa: E402
from workloads import MC_K_EXT, MC_N, MC_NEURON, microcircuit_synapses, psc_over_psp  # noqa: E402

DT = 0.1
AEIF = "aeif_cond_beta_multisynapse"
V_READ = 200            # neurons whose membrane potential a pass reads


def listed():
    return [
        # a robot or a live display: one step, read 8 potentials, next step (the smallest call)
        {"name": "steps_1k", "kind": "steps", "n": 1000, "k": 100, "dlo": 1.5, "dhi": 1.5, "gens": 1, "rate": 8000.0,
         "steps": 20, "warm": 60.0},
        # the small balanced network with its 400 separate Poisson inputs per neuron
        {"name": "balanced_1k", "kind": "adex", "n": 1000, "k": 100, "dlo": 1.5, "dhi": 1.5, "gens": 400, "rate": 20.0,
         "ms": 20.0, "warm": 60.0},
        # four receptors of per-neuron time constants, step sizes proposed by the step model
        {"name": "learned_1k", "kind": "learned", "n": 1000, "k": 100, "dlo": 1.5, "dhi": 1.5, "gens": 1, "rate": 4000.0,
         "ms": 30.0, "warm": 10.0},
        # current-based AdEx with per-neuron parameters, spike times read after each call
        {"name": "hetero_6k", "kind": "hetero", "n": 6007, "k": 250, "dlo": 0.5, "dhi": 2.0, "model": "aeif_psc_exp_multisynapse",
         "rate": 8000.0, "ms": 30.0, "warm": 30.0},
        # an ordinary AdEx network on a workstation's scale, sizes off the round numbers
        {"name": "adex_23k", "kind": "adex", "n": 23003, "k": 625, "dlo": 1.0, "dhi": 2.0, "gens": 1, "rate": 8000.0,
         "ms": 50.0, "warm": 100.0},
        # the headline network: 1M neurons, 1e9 synapses (the largest)
        {"name": "adex_1M", "kind": "adex", "n": 1000000, "k": 1000, "dlo": 1.0, "dhi": 2.0, "gens": 1, "rate": 8000.0,
         "ms": 50.0, "warm": 150.0},
        # the classic balanced network of integrate-and-fire neurons with one delay
        {"name": "brunel_12k", "kind": "brunel", "n": 12500, "k": 1250, "dlo": 1.5, "dhi": 1.5, "rate": 18000.0,
         "ms": 100.0, "warm": 20.0},
        # the layered microcircuit at a tenth of its populations: many short one-step batches
        {"name": "layers_8k", "kind": "layers", "scale": 0.1, "ms": 100.0, "warm": 100.0},
        # the layered microcircuit's populations at full size (77,169 neurons)
        {"name": "layers_77k", "kind": "layers", "scale": 1.0, "ms": 100.0, "warm": 200.0},
        # plastic excitatory synapses: one step per batch, weights change as it runs
        {"name": "stdp_4k", "kind": "stdp", "n": 4000, "k": 100, "ms": 50.0, "warm": 50.0},
        # 256 independent networks of 1k to 50k neurons in one engine
        {"name": "ensemble_256", "kind": "ensemble", "nets": 256, "spec": 2024, "ms": 20.0, "warm": 60.0},
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    kind = rng.choice(["steps", "adex", "adex", "adex", "learned", "hetero", "brunel", "layers", "layers", "stdp",
                       "ensemble"])
    if kind == "layers":
        return {"kind": kind, "scale": round(_log(rng, 0.04, 1.0), 4), "ms": round(rng.uniform(20.0, 100.0), 1),
                "warm": 50.0}
    if kind == "ensemble":
        return {"kind": kind, "nets": int(_log(rng, 8, 256)), "spec": rng.randrange(1, 10000),
                "ms": round(rng.uniform(5.0, 20.0), 1), "warm": 30.0}
    if kind == "stdp":
        return {"kind": kind, "n": int(_log(rng, 300, 5000)), "k": int(_log(rng, 20, 100)),
                "ms": round(rng.uniform(20.0, 50.0), 1), "warm": 50.0}
    if kind == "brunel":
        n = int(_log(rng, 1000, 30000))
        return {"kind": kind, "n": n, "k": int(_log(rng, 100, 1250)), "dlo": 1.5, "dhi": 1.5,
                "rate": round(rng.uniform(15000.0, 20000.0), 1), "ms": round(rng.uniform(30.0, 100.0), 1), "warm": 20.0}
    dlo = rng.choice([0.1, 0.5, 1.0, 1.5])
    dhi = round(dlo + rng.choice([0.0, 0.3, 1.0]), 1)
    if kind == "hetero":
        return {"kind": kind, "n": int(_log(rng, 500, 8000)), "k": int(_log(rng, 50, 400)), "dlo": dlo, "dhi": dhi,
                "model": rng.choice(["aeif_psc_exp_multisynapse", "aeif_psc_alpha_multisynapse",
                                     "aeif_cond_alpha_multisynapse"]),
                "rate": 8000.0, "ms": round(rng.uniform(15.0, 30.0), 1), "warm": 30.0}
    if kind == "learned":
        return {"kind": kind, "n": int(_log(rng, 300, 3000)), "k": 100, "dlo": 1.5, "dhi": 1.5, "gens": 1, "rate": 4000.0,
                "ms": round(rng.uniform(10.0, 30.0), 1), "warm": 10.0}
    if kind == "steps":
        return {"kind": kind, "n": int(_log(rng, 200, 5000)), "k": 100, "dlo": dlo, "dhi": dhi, "gens": 1,
                "rate": 8000.0, "steps": rng.randrange(5, 30), "warm": 60.0}
    n = int(_log(rng, 500, 300000))
    gens = rng.choice([1, 1, int(_log(rng, 2, 400))])
    if n > 5000:
        gens = 1
    return {"kind": "adex", "n": n, "k": int(_log(rng, 100, 1000)), "dlo": dlo, "dhi": dhi, "gens": gens,
            "rate": round(8000.0 / gens, 2), "ms": round(rng.uniform(10.0, 50.0), 1), "warm": 50.0}


# ---------------------------------------------------------------------------
# networks
# ---------------------------------------------------------------------------
def _split(n, k):
    """Excitatory neurons, and excitatory and inhibitory in-degree (80 / 20)."""
    return int(0.8 * n), int(round(0.8 * k)), k - int(round(0.8 * k))


def _sources(case, seed, neuron, ne, w_exc, w_inh, ports=(0, 1)):
    _, ke, ki = _split(case["n"], case["k"])
    ngpu.ConnectFixedIndegreeGPU(neuron[0:ne], neuron, ke, w_exc, case["dlo"], case["dhi"], receptor=ports[0], seed=seed + 1)
    ngpu.ConnectFixedIndegreeGPU(neuron[ne:case["n"]], neuron, ki, w_inh, case["dlo"], case["dhi"], receptor=ports[1],
                                 seed=seed + 2)


def _scaled(case):
    """Weights for other in-degrees than 1000: the summed input stays that of 1000 sources."""
    return 0.05 * (1000.0 / case["k"]), 0.35 * (1000.0 / case["k"])


def _taus(seed, n, ports=4):
    rng = np.random.RandomState(seed)
    return np.round(rng.uniform(0.2, 1.0, (n, ports)), 3), np.round(rng.uniform(2.0, 20.0, (n, ports)), 3)


def _step_model(seed):
    """A small step model of the documented layout: normalisation around the states that the
    network meets, small seeded weights, proposals around 0.05 ms."""
    rng = np.random.RandomState(seed)
    nf, nh = 10, 32

    def bf16(a):
        u = np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)
        return ((u + 0x7FFF + ((u >> 16) & 1)) & np.uint32(0xFFFF0000)).view(np.float32).ravel()

    mu = [-60.0, 80.0, 5.0, 5.0, 5.0, 5.0, 0.0, 0.0, -3.0, -3.0]
    isig = [0.1, 0.01, 0.2, 0.2, 0.2, 0.2, 0.5, 0.5, 1.0, 1.0]
    p = [mu, isig, bf16(rng.uniform(-0.3, 0.3, (nh, nf))), np.zeros(nh), bf16(rng.uniform(-0.2, 0.2, (nh, nh))), np.zeros(nh),
         bf16(rng.uniform(-0.1, 0.1, nh)), [0.0], [np.log(0.05)], [0.5], [0.9], [0.0]]
    return np.concatenate([np.asarray(x, dtype=np.float32).ravel() for x in p])


def _build(case, seed):
    """Creates the case's network in the calling thread's engine; returns the node sequences."""
    ngpu.Reset()
    ngpu.SetVerbosityLevel(0)
    kind = case["kind"]
    ngpu.SetKernelStatus("rnd_seed", 1000 + seed)
    if kind == "ensemble":
        spec = ensemble_spec(case["nets"], seed=case["spec"])
        for i, net in enumerate(spec):
            net["seed"] = (net["seed"] + 7 * seed) % (1 << 30) + 1
        groups, _ = build_ensemble(ngpu, spec)
        return list(groups.values())
    if kind == "layers":
        return _layers(case, seed)
    n = case["n"]
    if kind == "brunel":
        neuron = ngpu.Create("iaf_psc_exp", n)
        ngpu.SetStatus(neuron, {"tau_m": 20.0, "tau_ex": 0.5, "tau_in": 0.5, "Theta_rel": 20.0, "V_reset_rel": 10.0})
        pg = ngpu.Create("poisson_generator")
        ngpu.SetStatus(pg, "rate", case["rate"])
        ngpu.Connect(pg, neuron, {"rule": "all_to_all"}, {"weight": 45.0, "delay": 1.0, "receptor": 0})
        ne, _, _ = _split(n, case["k"])
        w = 45.0 * 1250.0 / case["k"]
        _sources(case, seed, neuron, ne, w, -5.0 * w)
        ngpu.CreateRecord("", ["V_m_rel"] * 10, [neuron[j] for j in range(10)], [0] * 10)
        ngpu.ActivateSpikeCount(neuron)
        return [neuron]
    if kind == "stdp":
        neuron = ngpu.Create("iaf_psc_exp", n)
        syn = ngpu.CreateSynGroup("stdp", {"tau_plus": 20.0, "tau_minus": 25.0, "lambda": 0.005, "alpha": 1.1,
                                           "mu_plus": 0.5, "mu_minus": 0.8, "Wmax": 80.0})
        pg = ngpu.Create("poisson_generator")
        ngpu.SetStatus(pg, "rate", 8000.0)
        ngpu.Connect(pg, neuron, {"rule": "all_to_all"}, {"weight": 25.0, "delay": 1.0, "receptor": 0})
        ne, ke, ki = _split(n, case["k"])
        ngpu.Connect(neuron[0:ne], neuron, {"rule": "fixed_total_number", "total_num": n * ke},
                     {"weight": 40.0, "receptor": 0, "synapse_group": syn,
                      "delay": {"distribution": "normal_clipped", "mu": 1.5, "low": 0.5, "high": 3.0, "sigma": 0.6}})
        ngpu.Connect(neuron[ne:n], neuron, {"rule": "fixed_total_number", "total_num": n * ki},
                     {"weight": -120.0, "receptor": 1, "delay": 0.8})
        ngpu.ActivateSpikeCount(neuron)
        return [neuron]
    ne, _, _ = _split(n, case["k"])
    if kind == "hetero":
        model = case["model"]
        neuron = ngpu.Create(model, n, 2)
        rng = np.random.RandomState(seed)
        v_th = np.round(rng.normal(-50.4, 1.0, n), 3)
        tau_w = np.round(rng.uniform(100.0, 180.0, n), 2)
        for i in range(n):
            ngpu.SetNeuronScalParam(neuron[i], 1, "V_th", float(v_th[i]))
            ngpu.SetNeuronScalParam(neuron[i], 1, "tau_w", float(tau_w[i]))
        if model == "aeif_cond_alpha_multisynapse":
            ngpu.SetStatus(neuron, {"E_rev": [0.0, -85.0], "tau_syn": [2.0, 5.0]})
            w_pg, w_exc, w_inh = 0.4, 0.5, 2.0
        else:
            ngpu.SetStatus(neuron, {"tau_syn": [2.0, 5.0]})
            w_pg, w_exc, w_inh = 40.0, 25.0, -75.0
        pg = ngpu.Create("poisson_generator")
        ngpu.SetStatus(pg, "rate", case["rate"])
        ngpu.Connect(pg, neuron, {"rule": "all_to_all"}, {"weight": w_pg, "delay": 1.0, "receptor": 0})
        f = 250.0 / case["k"]
        _sources(case, seed, neuron, ne, w_exc * f, w_inh * f)
        ngpu.ActivateSpikeCount(neuron)
        ngpu.ActivateRecSpikeTimes(neuron, 64)
        return [neuron]
    ports = 4 if kind == "learned" else 2
    neuron = ngpu.Create(AEIF, n, ports)
    if kind == "learned":
        ngpu.SetStatus(neuron, {"E_rev": [0.0, 0.0, -85.0, -85.0]})
        rise, decay = _taus(seed, n)
        for i in range(n):
            ngpu.SetNeuronArrayParam(neuron[i], 1, "tau_rise", [float(x) for x in rise[i]])
            ngpu.SetNeuronArrayParam(neuron[i], 1, "tau_decay", [float(x) for x in decay[i]])
    else:
        ngpu.SetStatus(neuron, {"E_rev": [0.0, -85.0]})
    pg = ngpu.Create("poisson_generator", case["gens"])
    ngpu.SetStatus(pg, "rate", case["rate"])
    w_pg = 1.0 if kind == "learned" else 0.1
    ngpu.Connect(pg, neuron, {"rule": "all_to_all"}, {"weight": w_pg, "delay": 1.0, "receptor": 0})
    if kind == "learned":
        _sources(case, seed, neuron, ne, 0.05, 0.35, ports=(1, 2))
    else:
        _sources(case, seed, neuron, ne, *_scaled(case))
    ngpu.ActivateSpikeCount(neuron)
    return [neuron]


def _layer_degrees():
    """In-degrees [target][source] of the full-size microcircuit, kept at every scale."""
    return np.round(microcircuit_synapses(1.0) / MC_N[:, None].astype(float)).astype(int)


def _layers(case, seed):
    """The layered microcircuit's populations at `scale`, its in-degrees, mean weights and
    drive; delays uniform around the model's means."""
    m = MC_NEURON
    n_pop = np.round(MC_N * case["scale"]).astype(int)
    k_in = _layer_degrees()
    pscp = psc_over_psp(m["C_m"], m["tau_m"], m["tau_syn"])
    rng = np.random.RandomState(seed)
    pops = []
    for i in range(8):
        p = ngpu.Create("iaf_psc_exp", int(n_pop[i]))
        ngpu.SetStatus(p, {"tau_ex": m["tau_syn"], "tau_in": m["tau_syn"], "E_L": m["E_L"], "Theta_rel": m["V_th"] - m["E_L"],
                           "V_reset_rel": m["V_reset"] - m["E_L"], "t_ref": m["t_ref"], "I_e": 0.0})
        # spread the starting potentials in 40 slices of each population
        cut = np.linspace(0, int(n_pop[i]), 41).astype(int)
        for a, b in zip(cut[:-1], cut[1:]):
            if b > a:
                ngpu.SetStatus(p[int(a):int(b)], "V_m_rel", float(rng.normal(2.0, 5.0)))
        pops.append(p)
    bg = ngpu.Create("poisson_generator", 8)
    for i in range(8):
        ngpu.SetStatus([bg[i]], "rate", float(8.0 * MC_K_EXT[i]))
    for i, tgt in enumerate(pops):
        for j, src in enumerate(pops):
            if k_in[i][j] <= 0:
                continue
            psp = 0.15 * (2.0 if (i, j) == (0, 2) else 1.0) * (-4.0 if j % 2 else 1.0)
            dlo, dhi = (0.1, 1.4) if j % 2 else (0.1, 2.9)
            ngpu.ConnectFixedIndegreeGPU(src, tgt, int(k_in[i][j]), psp * pscp, dlo, dhi, receptor=j % 2,
                                         seed=100 * seed + 8 * i + j + 1)
        ngpu.Connect([bg[i]], tgt, {"rule": "all_to_all"}, {"weight": 0.15 * pscp, "delay": 1.5})
    for p in pops:
        ngpu.ActivateSpikeCount(p)
    return pops


class Network(object):
    """A network on its own host thread (the engine keeps one network per thread)."""

    def __init__(self, case, seed):
        self.case = case
        self.todo, self.done = queue.SimpleQueue(), queue.SimpleQueue()
        self.thread = threading.Thread(target=_serve, args=(self.todo, self.done), daemon=True)
        self.thread.start()
        self.nodes = self.call(_ready, case, seed)

    def call(self, fn, *args):
        self.todo.put((fn, args))
        ok, value = self.done.get()
        if not ok:
            raise value
        return value

    def __del__(self):
        try:
            self.todo.put(None)
            self.thread.join()
        except Exception:
            pass


def _serve(todo, done):
    while True:
        job = todo.get()
        if job is None:
            ngpu.Reset()
            return
        try:
            done.put((True, job[0](*job[1])))
        except Exception as e:
            done.put((False, e))
        job = None


def _ready(case, seed):
    nodes = _build(case, seed)
    if case["kind"] == "learned":
        ngpu.StepModelSet(_step_model(seed))
        ngpu.StepModelEnable(True)
    extra = None
    if case["kind"] == "stdp":
        extra = ngpu.GetConnections(nodes[0][0:1], nodes[0])[:8]
    if case["warm"] > 0.0:
        ngpu.Simulate(case["warm"])     # the run-in that scripts discard
    if case["kind"] == "hetero":
        ngpu.GetRecSpikeTimes(nodes[0][0:1])
    return nodes, extra


def prepare(case, seed):
    return Network(case, seed)


def _v_name(kind):
    return "V_m_rel" if kind in ("brunel", "layers", "stdp") else "V_m"


def _results(case, nodes):
    """What a script reads after a call: every neuron's spike count, some potentials."""
    out = {}
    for g, seq in enumerate(nodes):
        out["spikes%d" % g] = ngpu.GetSpikeCountArray(seq)
    first = nodes[0]
    name = _v_name(case["kind"])
    if case["kind"] == "ensemble" and not ngpu.IsNeuronScalVar(first[0], name):
        name = "V_m_rel"
    out["V"] = np.asarray(ngpu.GetNeuronVar(first[0], min(V_READ, len(first)), name), dtype=np.float32)
    return out


def _pass(case, nodes, extra):
    kind = case["kind"]
    if kind == "steps":
        trace = []
        for _ in range(case["steps"]):
            ngpu.SimulationStep()
            trace.append(ngpu.GetNeuronVar(nodes[0][0], 8, "V_m"))
        return {"trace": np.asarray(trace, dtype=np.float32)}
    ngpu.Simulate(case["ms"])
    out = _results(case, nodes)
    if kind == "hetero":
        times = ngpu.GetRecSpikeTimes(nodes[0][0:min(500, case["n"])])
        out["times"] = np.array([sum(t) for t in times], dtype=np.float32)
        out["ntimes"] = np.array([len(t) for t in times], dtype=np.int64)
    elif kind == "stdp":
        out["weights"] = np.asarray(ngpu.GetStatus(extra, "weight"), dtype=np.float32)
    return out


def run(state):
    return state.call(_pass, state.case, *state.nodes)


# ---------------------------------------------------------------------------
# work and tolerance
# ---------------------------------------------------------------------------
def _load(case):
    """(aeif neurons, iaf neurons, synapses, mean firing rate [Hz] expected, steps)."""
    kind = case["kind"]
    if kind == "ensemble":
        spec = ensemble_spec(case["nets"], seed=case["spec"])
        na = sum(s["n"] for s in spec if s["model"] == AEIF)
        return na, sum(s["n"] for s in spec) - na, sum(s["n"] * s["indegree"] for s in spec), 20.0, case["ms"] / DT
    if kind == "layers":
        n = np.round(MC_N * case["scale"])
        return 0, float(n.sum()), float((_layer_degrees().sum(axis=1) * n).sum()), 4.0, case["ms"] / DT
    n, e = case["n"], case["n"] * float(case["k"])
    if kind == "brunel":
        return 0, n, e, 20.0, case["ms"] / DT
    if kind == "stdp":
        return 0, n, e, 20.0, case["ms"] / DT
    steps = case["steps"] if kind == "steps" else case["ms"] / DT
    return n, 0, e, {"learned": 100.0, "hetero": 20.0}.get(kind, 16.0), steps


def work(case):
    """Bytes: every neuron's state in and out once, 8 bytes (target, weight) per delivered
    synaptic event, the results.  Flops: 110 FP32 operations per derivative evaluation of an
    adaptive RK5 step, six evaluations per neuron and time step at least; about 20 per
    integrate-and-fire neuron and step; 60 integer and FP32 operations per Poisson draw."""
    na, ni, e, hz, steps = _load(case)
    ports = 4 if case["kind"] == "learned" else 2
    events = e * hz * steps * DT / 1000.0
    state = na * 4.0 * (2 + 2 * ports + 4) + ni * 16.0
    draws = (na + ni) * case.get("gens", 1) * steps
    derivs = na * steps * 6.0
    return {"bytes": 2.0 * state + 8.0 * events + 4.0 * (na + ni),
            "flops": derivs * (110.0 if ports == 2 else 180.0) + ni * steps * 20.0 + events * 2.0 + draws * 60.0}


def tolerance(case):
    """Measured in FP32 against exact() and FP64: potentials agree to 3e-7 (iaf) and 1e-6 to 1e-4
    (AdEx, an adaptive step at a tolerance of 1e-6) as long as no spike moves by a step.  In the
    AdEx networks above some thousand neurons a few do within a pass: 4e-3 to 2e-2 of the
    potentials' 2-norm, one neuron's reset amplitude, counts of a few neurons in a thousand."""
    return {"rel": 0.02, "max": 0.95, "differ": 0.01}


# ---------------------------------------------------------------------------
# the same networks in FP64 with numpy
# ---------------------------------------------------------------------------
_U32 = np.uint64(0xFFFFFFFF)


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 (Salmon et al., SC'11) on arrays of 32-bit words held in uint64."""
    k0, k1 = int(k0) & 0xFFFFFFFF, int(k1) & 0xFFFFFFFF
    s = np.uint64(32)
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c0, np.uint64(0xCD9E8D57) * c2
        c0, c1, c2, c3 = (p1 >> s) ^ c1 ^ np.uint64(k0), p1 & _U32, (p0 >> s) ^ c3 ^ np.uint64(k1), p0 & _U32
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c0, c1, c2, c3


def _in_edges(src0, ns, nt, k, dlo, dhi, seed):
    """Sources, targets and delays (steps) of a generated fixed in-degree block."""
    t = np.repeat(np.arange(nt, dtype=np.uint64), k)
    kk = np.tile(np.arange(k, dtype=np.uint64), nt)
    z = np.zeros_like(t)
    r0, r1, _, _ = _philox(t, kk, z, z + np.uint64(0x9E3779B9), seed & 0xFFFFFFFF, seed >> 32)
    s = np.uint64(32)
    lo, hi = int(round(dlo / DT)), int(round(dhi / DT))
    return (src0 + ((r0 * np.uint64(ns)) >> s)).astype(np.int64), t.astype(np.int64), \
        (lo + ((r1 * np.uint64(hi - lo + 1)) >> s)).astype(np.int64)


class _Poisson(object):
    """The engine's counter-based Poisson input: draws of `gens` generators, each connected to
    all n neurons, summed per neuron and step."""

    def __init__(self, case, seed, n, rate, gens):
        self.n, self.gens = n, gens
        self.key = 1000 + seed + 12345
        self.lam = np.float32(np.float32(0.1) / np.float64(1000.0)) * np.float32(rate)
        self.block, self.words = -1, None

    def at(self, tidx):
        if tidx * float(np.float32(0.1)) < 1.0:         # the drive's delay
            return np.zeros(self.n)
        if tidx >> 2 != self.block:
            self.block = tidx >> 2
            i = np.tile(np.arange(self.n, dtype=np.uint64), self.gens)
            g = np.repeat(np.arange(self.gens, dtype=np.uint64), self.n)
            z = np.zeros_like(i)
            self.words = _philox(i, g, z + np.uint64(self.block), z, (self.key & 0xFFFFFFFF) ^ 0x6A09E667,
                                 (self.key >> 32) ^ 0xBB67AE85)
        # the counts are input data: inversion of 24-bit uniforms, in FP32 like the engine's
        f32 = np.float32
        u = ((self.words[tidx & 3] >> np.uint64(8)).astype(f32) + f32(0.5)) * f32(2.0 ** -24)
        k = np.zeros(u.size)
        p = f = f32(np.exp(-float(self.lam)))
        j = 0
        left = np.nonzero(u > f)[0]
        while left.size and j < 1000 and p > f32(2.0 ** -30):
            k[left] += 1
            j += 1
            p = (p * self.lam) * f32(1.0 / j)
            f = f + p
            left = left[u[left] > f]
        return k.reshape(self.gens, self.n).sum(axis=0)


class _Delay(object):
    """Delayed delivery: edges sorted by source, a ring of input arrays per port."""

    def __init__(self, n, ports, blocks):
        src = np.concatenate([b[0] for b in blocks])
        order = np.argsort(src, kind="stable")
        self.off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))])
        self.tgt = np.concatenate([b[1] + b[3] * n for b in blocks])[order]
        self.d = np.concatenate([b[2] for b in blocks])[order]
        self.w = np.concatenate([np.full(b[0].size, float(np.float32(b[4]))) for b in blocks])[order]
        self.R = int(self.d.max()) + 1
        self.ring = np.zeros((self.R, ports * n))
        self.shape = (ports, n)

    def emit(self, spiking, step):
        for s in spiking:
            a, b = self.off[s], self.off[s + 1]
            np.add.at(self.ring, ((step + self.d[a:b]) % self.R, self.tgt[a:b]), self.w[a:b])

    def arrive(self, step):
        x = self.ring[step % self.R].reshape(self.shape).copy()
        self.ring[step % self.R] = 0.0
        return x


_A = np.array
_CK = [_A([0.2]), _A([3 / 40.0, 9 / 40.0]), _A([0.3, -0.9, 1.2]), _A([-11 / 54.0, 2.5, -70 / 27.0, 35 / 27.0]),
       _A([1631 / 55296.0, 175 / 512.0, 575 / 13824.0, 44275 / 110592.0, 253 / 4096.0])]
_C5 = _A([37 / 378.0, 0.0, 250 / 621.0, 125 / 594.0, 0.0, 512 / 1771.0])
_CE = _C5 - _A([2825 / 27648.0, 0.0, 18575 / 48384.0, 13525 / 55296.0, 277 / 14336.0, 0.25])


def _aeif_f(y, e_rev, it1, it2):
    """aeif_cond_beta_multisynapse with the default parameters; y [2 + 2 ports, m]."""
    v, w = np.minimum(y[0], 0.0), y[1]
    g, g1 = y[2::2], y[3::2]
    cur = (g * (e_rev[:, None] - v)).sum(axis=0)
    with np.errstate(over="ignore"):
        spike = 2.0 * np.exp((v + 50.4) / 2.0)
    d = np.empty_like(y)
    d[0] = (-30.0 * (v + 70.6 - spike) + cur - w) / 281.0
    d[1] = (4.0 * (v + 70.6) - w) / 144.0
    d[3::2] = -g1 * it1
    d[2::2] = g1 - g * it2
    return d


def _aeif_step(y, x, h, t1, e_rev, it1, it2):
    """All neurons to t1 with adaptive Cash-Karp steps; returns the spiking neurons."""
    hmin = 1e-3 * float(np.float32(0.1))
    act = np.arange(y.shape[1])
    spikes = []
    for _ in range(200000):
        if not act.size:
            break
        ya, ha, hmax = y[:, act], h[act], t1 - x[act]
        a1, a2 = it1[:, act], it2[:, act]
        k = [_aeif_f(ya, e_rev, a1, a2)]
        scal = np.abs(ya) + np.abs(k[0] * ha) + 0.1
        todo = np.arange(act.size)
        new = ya.copy()
        while todo.size:
            hh = np.maximum(np.minimum(ha[todo], hmax[todo]), hmin)
            yy, ks = ya[:, todo], [k[0][:, todo]]
            for row in _CK:
                ks.append(_aeif_f(yy + hh * sum(c * q for c, q in zip(row, ks)), e_rev, a1[:, todo], a2[:, todo]))
            yn = yy + hh * sum(c * q for c, q in zip(_C5, ks) if c)
            err = np.max(np.abs(hh * sum(c * q for c, q in zip(_CE, ks) if c)) / scal[:, todo], axis=0) * 1e6
            ok = (err <= 1.0) | (hh <= hmin * 1.00001)
            good = todo[ok]
            new[:, good] = yn[:, ok]
            x[act[good]] += hh[ok]
            with np.errstate(divide="ignore"):
                grown = np.where(err > 1.889568e-4, 0.9 * hh * err ** -0.2, 5.0 * hh)
                less = np.maximum(0.9 * hh * err ** -0.25, 0.1 * hh)
            ha[good] = grown[ok]
            ha[todo[~ok]] = less[~ok]
            todo = todo[~ok]
        fired = new[0] >= 0.0
        new[0, fired] = -60.0
        new[1, fired] += 80.5
        spikes.append(act[fired])
        y[:, act], h[act] = new, ha
        act = act[x[act] < t1 - hmin]
    return np.concatenate(spikes) if spikes else np.zeros(0, dtype=np.int64)


def _exact_aeif(case, seed):
    n, ports = case["n"], 4 if case["kind"] == "learned" else 2
    ne, ke, ki = _split(n, case["k"])
    if ports == 4:
        rise, decay = (a.astype(np.float32).astype(np.float64).T for a in _taus(seed, n))
        w, pe, pi, w_pg = (0.05, 0.35), 1, 2, 1.0
        e_rev = _A([0.0, 0.0, -85.0, -85.0])
    else:
        rise, decay = np.full((2, n), 2.0), np.full((2, n), 20.0)
        w, pe, pi, w_pg = _scaled(case), 0, 1, 0.1
        e_rev = _A([0.0, -85.0])
    tp = decay * rise * np.log(decay / rise) / (decay - rise)
    g0 = (1.0 / rise - 1.0 / decay) / (np.exp(-tp / decay) - np.exp(-tp / rise))
    net = _Delay(n, ports, [_in_edges(0, ne, n, ke, case["dlo"], case["dhi"], seed + 1) + (pe, w[0]),
                            _in_edges(ne, n - ne, n, ki, case["dlo"], case["dhi"], seed + 2) + (pi, w[1])])
    drive = _Poisson(case, seed, n, case["rate"], case["gens"])
    y = np.zeros((2 + 2 * ports, n))
    y[0] = -70.6
    x, h = np.zeros(n), np.full(n, 1e-2 * float(np.float32(0.1)))
    count = np.zeros(n, dtype=np.int64)
    dt = float(np.float32(0.1))
    warm = int(round(case["warm"] / DT))
    steps = case["steps"] if case["kind"] == "steps" else int(round(case["ms"] / DT))
    trace = []
    for s in range(1, warm + steps + 1):
        fired = _aeif_step(y, x, h, dt * s, e_rev, 1.0 / rise, 1.0 / decay)
        np.add.at(count, fired, 1)
        net.emit(fired, s)
        inp = net.arrive(s)
        inp[0] += float(np.float32(w_pg)) * drive.at(s)
        y[3::2] += inp * g0
        if s > warm:
            trace.append(y[0, :8].copy())
    if case["kind"] == "steps":
        return {"trace": np.array(trace)}
    return {"spikes0": count.astype(np.int32), "V": y[0, :V_READ].copy()}


def _exact_iaf(case, seed):
    """The brunel family: iaf_psc_exp by its exact propagators."""
    n, dt, tm, ts, c = case["n"], float(np.float32(0.1)), 20.0, 0.5, 250.0
    ne, ke, ki = _split(n, case["k"])
    w = 45.0 * 1250.0 / case["k"]
    net = _Delay(n, 2, [_in_edges(0, ne, n, ke, case["dlo"], case["dhi"], seed + 1) + (0, w),
                        _in_edges(ne, n - ne, n, ki, case["dlo"], case["dhi"], seed + 2) + (1, -5.0 * w)])
    drive = _Poisson(case, seed, n, case["rate"], 1)
    p11, p22 = np.exp(-dt / ts), np.exp(-dt / tm)
    p21 = tm * ts / (c * (tm - ts)) * (p22 - p11)
    p11, p22, p21 = (float(np.float32(p)) for p in (p11, p22, p21))   # they are FP32 model parameters
    ref = int(round(2.0 / DT))
    cur, v, r = np.zeros((2, n)), np.zeros(n), np.zeros(n, dtype=np.int64)
    count = np.zeros(n, dtype=np.int64)
    for s in range(1, int(round(case["warm"] / DT)) + int(round(case["ms"] / DT)) + 1):
        free = r == 0
        v = np.where(free, v * p22 + (cur[0] + cur[1]) * p21, v)
        r = np.where(free, 0, r - 1)
        cur *= p11
        fired = np.nonzero(v >= 20.0)[0]
        v[fired], r[fired] = 10.0, ref
        count[fired] += 1
        net.emit(fired, s)
        cur += net.arrive(s)
        cur[0] += 45.0 * drive.at(s)
    return {"spikes0": count.astype(np.int32), "V": v[:V_READ].copy()}


def exact(case, seed):
    """FP64 results, for the networks that numpy can run in the time allowed."""
    kind = case["kind"]
    if kind == "brunel" and case["n"] * case["k"] <= 2000000:
        return _exact_iaf(case, seed)
    if kind in ("steps", "adex", "learned"):
        steps = case["warm"] / DT + case.get("steps", case.get("ms", 0.0) / DT)
        if case["n"] * case["k"] <= 2000000 and case["n"] * steps * max(1.0, case["gens"] / 50.0) <= 7e6:
            return _exact_aeif(case, seed)
    return None
