"""Launches of several steps against launches of one.  With spike and SIC
delays of d steps a launch advances every cell by up to d/2 steps; plain
launches (use_graphs=-1) take one step each, and both give the same bits:
rasters, state, counters and, for a checkpoint taken by either, the other's
continuation.  Run lengths end below, at and past a launch's steps; delays
cover one, two and several steps per launch, unequal delays, SIC summed in
the neuron thread, a step ahead of its arrival, and by side batches; the
astrocytes emit from the start, so the SIC sums are not empty."""
import json

import numpy as np
import pytest

from astrosimgpu_b200 import _lib
from astrosimgpu_b200.network import Batch, Model, Network, Server, config_path

pytestmark = pytest.mark.gpu

REC = _lib.RecordOpts(0, 7, 1, 20, 15)
RUNS = (1, 2, 5, 6, 7, 8, 64, 3, 131)


def model(d_e, d_i, d_a2n, seed=3, **sizes):
    c = json.load(open(config_path("quick")))
    c["synapse"].update({"d_e": d_e, "d_i": d_i, "d_a2n": d_a2n, "w_a2n": 0.5})
    c["astrocyte"].update({"Ca_init": 0.35, "IP3": 0.6})
    c["connectivity"].update({"pool_type": "random", "pool_size": 3, "p_third_if_primary": 0.6})
    c["simulation"]["seed"] = seed
    c["N"].update(sizes)
    return Model(text=json.dumps(c), pre_time=0.0)


def outcome(net, rec=True):
    out = dict(net.state(), **net.counters())
    out["spikes_at"], out["spikes_of"] = net.fetch_spikes()
    if rec:
        out.update(("rec_" + k, v) for k, v in net.fetch_record().items())
    return out


def assert_same(a, b, *what):
    assert a.keys() == b.keys()
    for k in a:
        assert np.array_equal(a[k], b[k]), (k, *what)


@pytest.mark.parametrize("d_e,d_i,d_a2n", [(1.0, 1.0, 1.0), (0.2, 0.3, 1.0), (0.4, 0.7, 0.5),
                                           (1.7, 1.6, 1.0), (1.0, 1.5, 0.2), (2.0, 1.2, 1.3),
                                           (0.9, 1.0, 2.0), (1.0, 1.0, 0.1)])
@pytest.mark.parametrize("opts", [{}, {"occupancy": 2}, {"sic_mode": 1}])
def test_same_bits_as_single_steps(d_e, d_i, d_a2n, opts):
    m = model(d_e, d_i, d_a2n)
    a = Network(m, record=REC, chunk_steps=37, **opts)
    b = Network(m, record=REC, chunk_steps=37, use_graphs=-1, **opts)
    for n in RUNS:
        a.step(n)
        b.step(n)
        assert_same(outcome(a), outcome(b), n)
    assert a.counters()["sic_edges"] > 0 and a.counters()["spikes"] > 0


@pytest.mark.parametrize("d_a2n", [1.0, 2.0])
def test_checkpoints_continue_in_either_form(d_a2n):
    m = model(1.0, 1.0, d_a2n)
    forms = [{}, {"use_graphs": -1}, {"use_graphs": 2}]
    nets = [Network(m, record=REC, **f) for f in forms]
    for n in nets:
        n.step(203)
    blobs = [n.checkpoint() for n in nets]
    for n in nets:
        n.step(150)
    want = nets[0].state()
    for blob in blobs:
        for f in forms:
            n = Network(m, record=REC, **f)
            n.step(11)  # its own factors and lists, replaced by the checkpoint's
            n.restore(blob)
            n.step(150)
            got = n.state()
            for k in want:
                assert np.array_equal(got[k], want[k]), (k, f)


def test_batch_and_server_with_unequal_ends():
    """Instances of different sizes and delays share the shortest launch; a
    request that ends inside a chunk gives what it gives alone."""
    models = [model(1.0, 1.0, 1.0, 1), model(1.7, 1.6, 1.0, 2, N_E=300, N_I=70, N_A=90),
              model(0.6, 0.8, 0.9, 4)]
    ends = (97, 131, 203)
    alone = []
    for m, n in zip(models, ends):
        net = Network(m, record=REC, use_graphs=-1)
        net.step(n)
        alone.append(net.fetch_spikes())
    b = Batch(models, record=REC)
    b.step(97)
    for i in range(3):
        st, src = b.fetch_spikes(i)
        keep = alone[i][0] < 97
        assert np.array_equal(st, alone[i][0][keep]) and np.array_equal(src, alone[i][1][keep])
    s = Server()
    ids = [s.submit(m, n) for m, n in zip(models, ends)]
    for i, a in zip(ids, alone):
        s.wait(i)
        st, src = s.fetch_spikes(i)
        assert np.array_equal(st, a[0]) and np.array_equal(src, a[1])
    s.close()
