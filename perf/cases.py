"""The calls a user of this framework makes, as cases to time.

A case is a dict of plain values; `kind` names the entry point it goes
through and the other values its sizes:

- ``scaling``   AstroBackend.run_bernoulli: the astrocyte kernel-scaling
                workload (resident cells, input generated on the device),
                `steps` steps, then the state read back;
- ``dropin``    the astrocyte backend a host simulation binds: per step an
                input push, an update and a calcium pull;
- ``device``    asg_astro_update_noalloc on device arrays the caller owns;
- ``network``   one network: Network.step, then its spikes, recorded rows
                and state;
- ``sweep``     many small networks of uneven size advanced as one Batch;
- ``server``    simulation requests submitted to a Server and waited for.

Networks are taken past their opening burst in prepare(), as a user's
pre-simulation does, so that repeated passes see the same regime.
"""
from __future__ import annotations

import ctypes as C
import json
import math

import numpy as np
import torch

from astrosimgpu_b200 import _lib, workloads
from astrosimgpu_b200.astro import AstroBackend, ScalingWorkload
from astrosimgpu_b200.network import Batch, Model, Network, Server, config_path

# Arithmetic of one cell-step: the Li-Rinzel RK4 (four right-hand sides) and
# the AdEx RK4 (four right-hand sides with an exponential each).
ASTRO_FLOPS = 441
NEURON_FLOPS = 400


def listed():
    return [
        # A small astrocyte population (odd size): launches and latency.
        {"name": "scaling_4k", "kind": "scaling", "n": 4099, "steps": 1000},
        # The published kernel-scaling size: arithmetic throughput.
        {"name": "scaling_10m", "kind": "scaling", "n": 10_000_000, "steps": 100},
        # The astrocytes of the shipped 500-neuron model driven by a host
        # simulation, with per-cell parameters and noise: call latency.
        {"name": "dropin_100", "kind": "dropin", "n": 100, "steps": 20, "noise": True},
        # The same backend at the kernel-scaling size: copies and update.
        {"name": "dropin_10m", "kind": "dropin", "n": 10_000_000, "steps": 2, "noise": False},
        # Caller-owned device arrays near the entry point's largest size.
        {"name": "device_1m", "kind": "device", "n": 1_000_003, "noise": False},
        # The shipped 500-neuron model (100 astrocytes recorded): step latency.
        {"name": "use_case", "kind": "network", "config": "use_case", "warm": 2000,
         "steps": 2000},
        # The shipped 5,000-neuron model.
        {"name": "scale_1000", "kind": "network", "config": "scale_1000", "warm": 1000,
         "steps": 1000},
        # 10,000 neurons, ~10 M synapses, every astrocyte emitting SIC.
        {"name": "paper_sparse", "kind": "network", "config": "paper_sparse_dt005",
         "warm": 16000, "steps": 1000},
        # Serving-shaped networks alone: an ordinary and the largest request.
        {"name": "serving_200k", "kind": "network", "serving": 200_003, "warm": 400,
         "steps": 200},
        {"name": "serving_1m", "kind": "network", "serving": 1_000_000, "warm": 400,
         "steps": 100},
        # The 64-instance parameter sweep.
        {"name": "sweep_64", "kind": "sweep", "instances": 64, "warm": 500, "steps": 1000},
        # A burst of requests of mixed size through the server.
        {"name": "server_10", "kind": "server", "requests": 10, "n_max": 40_000,
         "steps": 500},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scaling", "dropin", "device", "network", "network", "network", "sweep",
                       "server"])
    if kind == "scaling":
        n = _log_int(rng, 1000, 5_000_000)
        return {"kind": kind, "n": n, "steps": max(20, min(1000, _log_int(rng, 2e8, 5e8) // n))}
    if kind == "dropin":
        return {"kind": kind, "n": _log_int(rng, 50, 3_000_000), "steps": rng.randint(2, 8),
                "noise": rng.random() < 0.5}
    if kind == "device":
        return {"kind": kind, "n": _log_int(rng, 100, 1 << 20), "noise": rng.random() < 0.5}
    if kind == "network":
        if rng.random() < 0.4:
            return {"kind": kind, "config": rng.choice(["quick", "bursting", "c0_literal",
                                                        "random_pool", "no_spiking"]),
                    "warm": rng.randint(1000, 2000), "steps": rng.randint(500, 2000)}
        n = _log_int(rng, 500, 400_000)
        return {"kind": kind, "serving": n, "warm": 400,
                "steps": max(100, min(2000, _log_int(rng, 1e7, 3e7) // n))}
    if kind == "sweep":
        return {"kind": kind, "instances": rng.randint(4, 64), "warm": rng.randint(300, 600),
                "steps": rng.randint(300, 1000)}
    return {"kind": kind, "requests": rng.randint(2, 10), "n_max": _log_int(rng, 1000, 40_000),
            "steps": rng.randint(100, 500)}


# ------------------------------------------------------------------- inputs


def _pinned(n, dtype=torch.float64):
    return torch.empty(max(int(n), 1), dtype=dtype, pin_memory=torch.cuda.is_available())


def _scaling_workload(case, seed):
    return ScalingWorkload(int(case["n"]), seed=int(seed) % 100_000 + 1)


def _astro_inputs(case, seed):
    """State, per-cell parameters (spread +-5 %) and per-step inputs (a few
    percent of the cells receive an event) of `dropin` and `device` cases."""
    n, k = int(case["n"]), int(case.get("steps", 1))
    g = np.random.default_rng(int(seed))
    w = ScalingWorkload(n, seed=int(seed) % 100_000 + 1)
    state = [x0 * (1.0 + 0.1 * (2.0 * g.random(n) - 1.0)) for x0 in w.rest]
    params = [v * (1.0 + 0.1 * (g.random(n) - 0.5))
              for v in (w.Ca_tot, w.IP3_0, w.tau_IP3, w.delta_IP3)]
    pushed = []
    for _ in range(k):
        a = np.zeros(n)
        cells = g.integers(0, n, max(1, n // 50))
        a[cells] = w.weight * g.random(len(cells))
        pushed.append(a)
    noise = dict(noise_std=0.0003 if case["noise"] else 0.0, noise_seed=int(seed) + 17)
    return w, state, params, pushed, noise


def _network_model(case, seed):
    s = int(seed) % 100_000 + 1
    if "serving" in case:
        return Model(text=workloads.serving_config(int(case["serving"]), s, 100.0), pre_time=0.0,
                     fixed_indegree=100, gen_device=0)
    return Model(config_path(case["config"]), seed=s, pre_time=0.0)


_N_KEYS = ("V", "w", "g_ex", "dg_ex", "g_in", "dg_in", "I_sic")
_A_KEYS = ("Ca", "IP3", "h")


class _StateBuffers:
    """Pinned host arrays for the dynamic state of one or more networks (one
    array per field, the networks one after another)."""

    def __init__(self, sizes):
        n, na = sum(s[0] for s in sizes), sum(s[1] for s in sizes)
        self.t = {k: _pinned(n) for k in _N_KEYS}
        self.t["refractory"] = _pinned(n, torch.int32)
        self.t.update({k: _pinned(na) for k in _A_KEYS})
        self.out = {k: t[: na if k in _A_KEYS else n] for k, t in self.t.items()}
        self.states = []
        i = a = 0
        for m, ma in sizes:
            st = _lib.State()
            for k, t in self.t.items():
                size, off = (4, i) if k == "refractory" else (8, a if k in _A_KEYS else i)
                ctype = C.c_int32 if size == 4 else C.c_double
                setattr(st, k, C.cast(t.data_ptr() + size * off, C.POINTER(ctype)))
            self.states.append(st)
            i, a = i + m, a + ma


class _RasterBuffers:
    """Host arrays a run's spikes are fetched into: the first `count` entries
    of `steps` and `sources`, -1 beyond them."""

    def __init__(self, cap):
        self.steps, self.sources = np.full(cap, -1, np.int64), np.full(cap, -1, np.int32)
        self.used = 0

    def fetch(self, calls):
        """Fetches one raster after another; `calls` are (entry point, its
        leading arguments).  Returns the number of spikes of each."""
        at, counts = 0, []
        for name, *args in calls:
            n = C.c_int64()
            _lib.call(name, *args,
                      C.cast(self.steps.ctypes.data + 8 * at, _lib.c_int64_p),
                      C.cast(self.sources.ctypes.data + 4 * at, _lib.c_uint32_p),
                      len(self.steps) - at, C.byref(n))
            at += n.value
            counts.append(n.value)
        self.steps[at:self.used] = -1
        self.sources[at:self.used] = -1
        self.used = at
        return np.array(counts, np.int64)


def _raster_cap(neurons, steps):
    return 20_000 + int(neurons) * int(steps) // 40


# ------------------------------------------------------------------ prepare


def prepare(case, seed):
    return {"scaling": _prepare_scaling, "dropin": _prepare_dropin, "device": _prepare_device,
            "network": _prepare_network, "sweep": _prepare_sweep,
            "server": _prepare_server}[case["kind"]](case, seed)


def _prepare_scaling(case, seed):
    w = _scaling_workload(case, seed)
    host = [_pinned(w.n) for _ in range(3)]
    return {"kind": "scaling", "w": w, "steps": int(case["steps"]), "first": 0,
            "backend": AstroBackend(*w.initial_state()), "host": host}


def _prepare_dropin(case, seed):
    w, state, params, pushed, noise = _astro_inputs(case, seed)
    ins = [_pinned(w.n) for _ in pushed]
    for t, a in zip(ins, pushed):
        t.copy_(torch.from_numpy(a))
    return {"kind": "dropin", "w": w, "noise": noise, "index": 0,
            "backend": AstroBackend(*state, *params), "ins": ins,
            "outs": [_pinned(w.n) for _ in pushed]}


def _prepare_device(case, seed):
    w, state, params, pushed, noise = _astro_inputs(case, seed)
    dev = [torch.from_numpy(a).cuda() for a in (*state, *params)]
    return {"kind": "device", "w": w, "noise": noise, "index": 0, "state": dev[:3],
            "params": dev[3:], "pushed": torch.from_numpy(pushed[0]).cuda(),
            "input": torch.zeros(w.n, dtype=torch.float64, device="cuda")}


def _prepare_network(case, seed):
    m = _network_model(case, seed)
    rec = m.record_opts() if "config" in case else _lib.RecordOpts(0, 100, 1, 0, 0)
    net = Network(m, record=rec)
    net.step(int(case["warm"]))
    net.fetch_spikes()
    net.fetch_record()
    return {"kind": "network", "net": net, "steps": int(case["steps"]),
            "host": _StateBuffers([(net.n, net.na)]),
            "raster": _RasterBuffers(_raster_cap(net.n, case["steps"]))}


def _sweep_models(case, seed):
    seeds = [int(seed) % 100_000 + k for k in range(1, 9)]
    return [Model(text=t, pre_time=0.0)
            for t in workloads.sweep_configs(int(case["instances"]), seeds=seeds)]


def _prepare_sweep(case, seed):
    b = Batch(_sweep_models(case, seed), record=_lib.RecordOpts(0, 100, 1, 0, 0))
    b.step(int(case["warm"]))
    for i in range(len(b.models)):
        b.fetch_spikes(i)
    sizes = [(d.n_exc + d.n_inh, d.n_astro) for d in b.descs]
    return {"kind": "sweep", "batch": b, "steps": int(case["steps"]),
            "host": _StateBuffers(sizes),
            "raster": _RasterBuffers(_raster_cap(sum(n for n, _ in sizes), case["steps"]))}


def _prepare_server(case, seed):
    g = np.random.default_rng(int(seed))
    sizes = np.exp(g.uniform(math.log(500.0), math.log(case["n_max"]), int(case["requests"])))
    sizes[0] = case["n_max"]
    models = [Model(text=workloads.serving_config(int(n), int(seed) % 100_000 + 1 + k, 100.0),
                    pre_time=0.0, fixed_indegree=100, gen_device=0)
              for k, n in enumerate(sizes)]
    return {"kind": "server", "server": Server(), "models": models, "steps": int(case["steps"]),
            "raster": _RasterBuffers(_raster_cap(case["requests"] * case["n_max"], case["steps"]))}


# ---------------------------------------------------------------------- run


def _f64(t):
    return C.cast(t.data_ptr(), _lib.c_double_p)


def run(state):
    kind = state["kind"]
    if kind == "scaling":
        w, k = state["w"], state["steps"]
        state["backend"].run_bernoulli(w, state["first"], k)
        state["first"] += k
        _lib.call("asg_astro_pull_state", state["backend"]._h, *[_f64(t) for t in state["host"]])
        return state["host"]
    if kind == "dropin":
        w, b, z = state["w"], state["backend"], state["noise"]
        for t, out in zip(state["ins"], state["outs"]):
            _lib.call("asg_astro_push_input", b._h, _f64(t))
            b.update(w.consts, w.h_step, w.substeps, noise_std=z["noise_std"], independent=True,
                     noise_seed=z["noise_seed"], noise_index=state["index"])
            _lib.call("asg_astro_pull_calcium", b._h, _f64(out))
            state["index"] += 1
        return state["outs"]
    if kind == "device":
        w, z = state["w"], state["noise"]
        state["input"].copy_(state["pushed"])
        _lib.call("asg_astro_update_noalloc", w.n,
                  *[C.c_void_p(t.data_ptr())
                    for t in (*state["state"], state["input"], *state["params"])],
                  _lib.dptr(w.consts), w.h_step, w.substeps, z["noise_std"], 1, 0.0,
                  z["noise_seed"], state["index"],
                  C.c_void_p(torch.cuda.current_stream().cuda_stream))
        state["index"] += 1
        return [*state["state"], state["input"]]
    if kind == "network":
        net = state["net"]
        net.step(state["steps"])
        _lib.call("asg_pull_state", net._h, C.byref(state["host"].states[0]))
        raster = state["raster"]
        counts = raster.fetch([("asg_fetch_spikes", net._h)])
        rec = net.fetch_record()
        return {"state": state["host"].out, "spikes": counts, "spike_steps": raster.steps,
                "spike_sources": raster.sources,
                "rows": [rec[k] for k in ("Ca", "IP3", "V", "I_sic")]}
    if kind == "sweep":
        b, raster = state["batch"], state["raster"]
        b.step(state["steps"])
        for i, st in enumerate(state["host"].states):
            _lib.call("asg_batch_pull_state", b._h, i, C.byref(st))
        counts = raster.fetch([("asg_batch_fetch_spikes", b._h, i)
                               for i in range(len(b.models))])
        return {"state": state["host"].out, "spikes": counts, "spike_steps": raster.steps,
                "spike_sources": raster.sources}
    srv, raster = state["server"], state["raster"]
    ids = [srv.submit(m, state["steps"]) for m in state["models"]]
    results = [srv.wait(i) for i in ids]
    counts = raster.fetch([("asg_serve_fetch_spikes", srv._h, i) for i in ids])
    return {"spikes": counts, "spike_steps": raster.steps, "spike_sources": raster.sources,
            "edges": np.array([int(r.spike_edges) for r in results], np.int64)}


# --------------------------------------------------------------------- work


def _network_work(n, na, edges, steps):
    return {"bytes": 2 * (60.0 * n + 24.0 * na) + 24.0 * n + 32.0 * na + 4.0 * edges,
            "flops": float(steps) * (NEURON_FLOPS * n + ASTRO_FLOPS * na)}


def work(case):
    kind = case["kind"]
    if kind == "scaling":  # state in and out once, every cell advanced `steps` times
        return {"bytes": 48.0 * case["n"], "flops": float(ASTRO_FLOPS) * case["n"] * case["steps"]}
    if kind == "dropin":  # parameters and state once, input and calcium each step
        n, k = case["n"], case["steps"]
        return {"bytes": n * (32.0 + 48.0 + 16.0 * k), "flops": float(ASTRO_FLOPS) * n * k}
    if kind == "device":  # state and input in and out, parameters in
        return {"bytes": 96.0 * case["n"], "flops": float(ASTRO_FLOPS) * case["n"]}
    if kind == "network":
        if "serving" in case:
            n = case["serving"]
            return _network_work(n, n, 132.0 * n, case["steps"])
        with open(config_path(case["config"])) as f:
            c = json.load(f)
        n = c["N"]["N_E"] + c["N"]["N_I"]
        p3 = c["connectivity"]["p_third_if_primary"]
        edges = c["connectivity"]["p_primary"] * n * (n + 2.0 * p3 * c["N"]["N_E"])
        return _network_work(n, c["N"]["N_A"], edges, case["steps"])
    if kind == "sweep":
        sizes = [(250, 500, 1000, 2000, 4000)[i % 5] for i in range(case["instances"])]
        n = float(sum(sizes))
        return _network_work(n, n / 5, 132.0 * n, case["steps"])
    n = case["n_max"] * (1.0 + 0.25 * (case["requests"] - 1))
    return _network_work(n, n, 132.0 * n, case["steps"])


# -------------------------------------------------------------------- exact
#
# The model in plain 64-bit numpy / torch.


def exact(case, seed):
    kind = case["kind"]
    if kind == "scaling":
        return _exact_scaling(case, seed)
    if kind == "dropin":
        return _exact_dropin(case, seed)
    if kind == "device":
        w, st, params, pushed, z = _astro_inputs(case, seed)
        st = _astro_advance(w, [torch.from_numpy(a) for a in st],
                            [torch.from_numpy(a) for a in params], torch.from_numpy(pushed[0]),
                            _astro_noise(z, w.n, 0))
        return [*st, torch.zeros(w.n, dtype=torch.float64)]
    if kind == "network" and "config" in case and case["warm"] + case["steps"] <= 5000:
        return _exact_network(case, seed)
    return None  # minutes of plain numpy


_M64 = (1 << 64) - 1
_PHI, _MIX_A, _MIX_B = 0x9E3779B97F4A7C15, 0xBF58476D1CE4E5B9, 0x94D049BB133111EB


def _unit(seed, stream, counter):
    """The counter RNG's uniform draw in [0, 1) for arrays of streams."""
    with np.errstate(over="ignore"):
        z = (np.uint64(seed & _M64) + np.asarray(stream, np.uint64) * np.uint64(_PHI)
             + np.uint64(counter) * np.uint64(_MIX_A))
        z = (z ^ (z >> np.uint64(30))) * np.uint64(_MIX_A)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(_MIX_B)
        z = z ^ (z >> np.uint64(31))
    return (z >> np.uint64(11)).astype(np.float64) * (1.0 / 9007199254740992.0)


def _streams(n, index, stride):
    with np.errstate(over="ignore"):
        return np.uint64(index * stride & _M64) + np.arange(n, dtype=np.uint64)


def _normal(seed, streams):
    u1 = np.maximum(_unit(seed, streams, 0), 1e-300)
    return np.sqrt(-2.0 * np.log(u1)) * np.cos(2.0 * math.pi * _unit(seed, streams, 1))


def _poisson(seed, streams, lam):
    """Knuth's product method (the draws the model makes for lambda <= 30)."""
    limit, count, k = math.exp(-lam), np.zeros(len(streams)), 1
    product = _unit(seed, streams, 0)
    live = np.nonzero(product > limit)[0]
    while len(live):
        count[live] += 1.0
        product[live] *= _unit(seed, streams[live], k)
        k += 1
        live = live[product[live] > limit]
    return count


def _astro_noise(z, n, index):
    if z["noise_std"] == 0.0:
        return 0.0
    return z["noise_std"] * torch.from_numpy(_normal(z["noise_seed"], _streams(n, index, 1000003)))


def _li_rinzel(c, p, ca, ip3, h, noise):
    kd1, kd2, kact, kinh, km, kr, r_rel, r_leak, r_up, ratio = (float(v) for v in c)
    ca_tot, ip3_0, tau, _ = p
    grad = (ca_tot - ca) / ratio - ca
    m = ip3 / (ip3 + kd1)
    q = ca / (ca + kact)
    release = ratio * r_rel * (m * m * m) * (q * q * q) * (h * h * h) * grad
    uptake = r_up * ca * ca / (km * km + ca * ca)
    opening = kr * kinh * (ip3 + kd1) / (ip3 + kd2)
    return (release - uptake + ratio * r_leak * grad + noise, (ip3_0 - ip3) / tau,
            opening * (1.0 - h) - kr * ca * h)


def _clip(x, lo, hi):
    return torch.clamp(x, lo, hi) if isinstance(x, torch.Tensor) else np.clip(x, lo, hi)


def _astro_rk4(c, p, st, inp, noise, h):
    ca, ip3, hh = st
    ip3 = ip3 + p[3] * inp
    x = (ca, ip3, hh)
    k1 = _li_rinzel(c, p, *x, noise)
    k2 = _li_rinzel(c, p, *[a + 0.5 * h * k for a, k in zip(x, k1)], noise)
    k3 = _li_rinzel(c, p, *[a + 0.5 * h * k for a, k in zip(x, k2)], noise)
    k4 = _li_rinzel(c, p, *[a + h * k for a, k in zip(x, k3)], noise)
    ca, ip3, hh = (a + (h / 6.0) * (r1 + 2.0 * r2 + 2.0 * r3 + r4)
                   for a, r1, r2, r3, r4 in zip(x, k1, k2, k3, k4))
    top = p[0]
    ca = torch.minimum(ca, torch.as_tensor(top, dtype=ca.dtype, device=ca.device)) \
        if isinstance(ca, torch.Tensor) else np.minimum(ca, top)
    return [_clip(ca, 0.0, None), _clip(ip3, 0.0, None), _clip(hh, 0.0, 1.0)]


def _astro_advance(w, st, params, inp, noise):
    for _ in range(w.substeps):
        st = _astro_rk4(w.consts, params, st, inp, noise, w.h_step)
        inp = 0.0
    return st


def _exact_scaling(case, seed):
    w = _scaling_workload(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if dev == "cpu" and w.n * int(case["steps"]) > 20_000_000:
        return None

    def shr(z, k):  # logical shift of int64 words
        return (z >> k) & ((1 << (64 - k)) - 1)

    def i64(v):
        return v - (1 << 64) if v >= 1 << 63 else v

    st = [torch.from_numpy(a).to(dev) for a in w.initial_state()]
    params = (w.Ca_tot, w.IP3_0, w.tau_IP3, w.delta_IP3)
    base = w.seed + torch.arange(w.n, dtype=torch.int64, device=dev) * i64(_PHI)
    threshold = math.ceil(w.p * 2.0 ** 53)
    for step in range(int(case["steps"])):
        z = base + i64((1000 + step) * _MIX_A & _M64)
        z = (z ^ shr(z, 30)) * i64(_MIX_A)
        z = (z ^ shr(z, 27)) * i64(_MIX_B)
        z = z ^ shr(z, 31)
        event = (shr(z, 11) < threshold).to(torch.float64)
        st = _astro_advance(w, st, params, w.weight * event, 0.0)
    return st


def _exact_dropin(case, seed):
    w, st, params, pushed, z = _astro_inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    st = [torch.from_numpy(a).to(dev) for a in st]
    params = [torch.from_numpy(a).to(dev) for a in params]
    out = []
    for k, a in enumerate(pushed):
        noise = _astro_noise(z, w.n, k)
        noise = noise.to(dev) if isinstance(noise, torch.Tensor) else noise
        st = _astro_advance(w, st, params, torch.from_numpy(a).to(dev), noise)
        out.append(st[0])
    return out


def _exact_network(case, seed):
    """The step loop of the model on the built tables; None in the places of
    the spikes (whole numbers)."""
    m = _network_model(case, seed)
    d = m.desc()
    NE, N, NA = d.n_exc, d.n_exc + d.n_inh, d.n_astro
    cells = m.cells()
    tables = [m.table(k) for k in range(4)]  # exc, inh, neuron->astro, astro->neuron
    h = d.dt / d.substeps
    sd, two = d.seed, (slice(0, NE), slice(NE, N))
    # population parameters spread over the neurons
    prm = {}
    for name, _ in _lib.NeuronParams._fields_:
        prm[name] = np.where(np.arange(N) < NE, getattr(d.exc, name), getattr(d.inh, name))
    consts = [getattr(d.astro, k) for k in
              ("Kd_IP3_1", "Kd_IP3_2", "Kd_act", "Kd_inh", "Km_SERCA", "k_IP3R", "rate_IP3R",
               "rate_L", "rate_SERCA", "ratio_ER_cyt")]
    ap = [cells[k] for k in ("Ca_tot", "IP3_0", "tau_IP3", "delta_IP3")]
    V = np.where(np.arange(N) < NE, d.V_m_init_exc, d.V_m_init_inh)
    w, ge, dge, gi, dgi, isic = (np.zeros(N) for _ in range(6))
    refr = np.zeros(N, np.int32)
    astro = [np.full(NA, d.Ca_init), np.full(NA, d.IP3_init), np.full(NA, d.h_init)]
    x, u, t_last = np.ones(N), np.full(N, d.stp.U), np.full(N, -1e12)
    slots = max(d.d_e_steps, d.d_i_steps, d.d_a2n_steps, 1) + 1
    r_ex, r_in, r_sic = (np.zeros((slots, N)) for _ in range(3))
    r_as = np.zeros((slots, NA))
    pending = np.zeros(slots, bool)
    a2n_src = np.repeat(np.arange(NA), np.diff(tables[3][0]))
    xe, xi = np.exp(-h / prm["tau_syn_ex"]), np.exp(-h / prm["tau_syn_in"])
    rec = m.record_opts()
    am, nm = min(rec.astro_max, NA), min(rec.neuron_max, N)
    rows = [[], [], [], []]

    def rates(V, w, ge, gi, I):
        v = np.minimum(V, prm["V_peak"])
        rel = v - prm["E_L"]
        spike = prm["g_L"] * prm["Delta_T"] * np.exp((v - prm["V_th"]) / prm["Delta_T"])
        dV = (-prm["g_L"] * rel + spike - ge * (v - prm["E_ex"]) - gi * (v - prm["E_in"]) - w
              + prm["I_e"] + I) / prm["C_m"]
        return dV, (prm["a"] * rel - w) / prm["tau_w"]

    def term(inp, n, index, salt, stride):
        """Noise of one population's cells `n` (an index range)."""
        every = max(1, int(math.floor(inp.noise_dt / d.dt + 0.5)))
        if not inp.gauss_noise_std > 0.0:
            return 0.0
        if not inp.independent_noise:
            raise NotImplementedError("shared noise")
        streams = _streams(n.stop, index // every, stride)[n.start:]
        return inp.gauss_noise_std * _normal(sd ^ salt, streams)

    for step in range(int(case["warm"]) + int(case["steps"])):
        s = step % slots
        exc_in, inh_in, ip3_in = (np.zeros(k) for k in (N, N, NA))
        for v in (r_ex[s], -r_in[s]):
            exc_in += np.where(v > 0.0, v, 0.0)
            inh_in -= np.where(v < 0.0, v, 0.0)
        if pending[s]:
            isic = r_sic[s].copy()
            pending[s] = False
        ip3_in += r_as[s]
        r_ex[s] = r_in[s] = r_sic[s] = r_as[s] = 0.0
        if d.input_astro.poiss_rate > 0.0:
            ip3_in += d.input_astro.poiss_weight * _poisson(
                sd ^ 0xC2B2AE3D27D4EB4F, _streams(NA, step, 1000003),
                d.input_astro.poiss_rate * d.dt * 1e-3)
        noise = term(d.input_astro, slice(0, NA), step, 0x9E3779B97F4A7C15, 1000003)
        for k in range(d.substeps):
            astro = _astro_rk4(consts, ap, astro, ip3_in if k == 0 else 0.0, noise, h)
        I = isic.copy()
        for sl, inp in zip(two, (d.input_exc, d.input_inh)):
            if inp.poiss_rate > 0.0:
                exc_in[sl] += inp.poiss_weight * _poisson(
                    sd ^ 0x2545F4914F6CDD1D, _streams(N, step, 1000003)[sl],
                    inp.poiss_rate * d.dt * 1e-3)
            I[sl] += term(inp, sl, step, 0x9E3779B185EBCA87, 1000033)
        dge = dge + exc_in * (math.e / prm["tau_syn_ex"])
        dgi = dgi + inh_in * (math.e / prm["tau_syn_in"])
        spiked = np.zeros(N, bool)
        for _ in range(d.substeps):
            ge1, dge1 = xe * (ge + h * dge), xe * dge
            gi1, dgi1 = xi * (gi + h * dgi), xi * dgi
            held = refr > 0
            gem, gim = 0.5 * (ge + ge1), 0.5 * (gi + gi1)
            V0 = np.where(held, cells["V_reset"], V)
            k1 = rates(V0, w, ge, gi, I)
            k2 = rates(V + 0.5 * h * k1[0], w + 0.5 * h * k1[1], gem, gim, I)
            k3 = rates(V + 0.5 * h * k2[0], w + 0.5 * h * k2[1], gem, gim, I)
            k4 = rates(V + h * k3[0], w + h * k3[1], ge1, gi1, I)
            Vn, wn = (a + (h / 6.0) * (p + 2.0 * q + 2.0 * r + t)
                      for a, p, q, r, t in zip((V, w), k1, k2, k3, k4))
            V = np.where(held, V0, Vn)
            w = np.where(held, w + h * k1[1], wn)
            ge, dge, gi, dgi = ge1, dge1, gi1, dgi1
            fire = ~held & (V >= prm["V_peak"])
            refr = np.where(held, refr - 1, refr)
            refr = np.where(fire, (prm["t_ref"] / h + 0.5).astype(np.int32), refr)
            w = np.where(fire, w + cells["b"], w)
            V = np.where(fire, cells["V_reset"], V)
            spiked |= fire
        now = step * d.dt
        for j in np.nonzero(spiked)[0]:
            f = 1.0
            if d.stp.enabled:
                gap = now - t_last[j]
                xd = math.exp(-gap / d.stp.tau_rec)
                ud = 0.0 if d.stp.tau_fac < 1e-10 else math.exp(-gap / d.stp.tau_fac)
                x[j] = 1.0 + (x[j] - x[j] * u[j] - 1.0) * xd
                u[j] = d.stp.U + u[j] * (1.0 - d.stp.U) * ud
                t_last[j] = now
                f = x[j] * u[j]
            for ring, (rs, tg), row, wt, dl in (
                    ((r_ex, tables[0], j, d.w_e, d.d_e_steps),
                     (r_as, tables[2], j, d.w_n2a, d.d_e_steps)) if j < NE else
                    ((r_in, tables[1], j - NE, -d.w_i, d.d_i_steps),)):
                np.add.at(ring[(step + dl) % slots], tg[rs[row]:rs[row + 1]], wt * f)
        if step % d.sic_interval == 0:
            y = (astro[0] - d.astro.SIC_th) * 1000.0
            fac = np.where(y > 1.0, d.astro.SIC_scale * np.log(np.maximum(y, 1.0)), 0.0)
            pending[(step + d.d_a2n_steps) % slots] = True
            if fac.any():
                np.add.at(r_sic[(step + d.d_a2n_steps) % slots], tables[3][1],
                          d.w_a2n * fac[a2n_src])
        if step >= int(case["warm"]) and step % rec.record_every == 0:
            for r, a, k in zip(rows, (astro[0], astro[1], V, isic), (am, am, nm, nm)):
                if k:
                    r.append(a[:k].copy())
    out = dict(zip(_N_KEYS, (V, w, ge, dge, gi, dgi, isic)), refractory=None)
    out.update(zip(_A_KEYS, astro))
    rows = [np.array(r).reshape(len(r), k) for r, k in zip(rows, (am, am, nm, nm))]
    return {"state": out, "spikes": None, "spike_steps": None, "spike_sources": None,
            "rows": rows}
