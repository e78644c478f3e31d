"""Rare paths of launches of several steps, against launches of one: several
noise draws in one launch (an interval shorter than it), Poisson counts around
the 255 that the packed draws hold, astrocytes in FP32, a tuned network, a
restore to step 0, and an instance whose delays allow one step per launch that
joins and leaves while the others' SIC factors are in use."""
import json
import time

import numpy as np
import pytest

from astrosimgpu_b200 import _lib
from astrosimgpu_b200.network import Model, Network, Server, config_path

pytestmark = pytest.mark.gpu
RUNS = (7, 64, 5, 131, 30)


def model(seed=3, d=1.0, **sections):
    c = json.load(open(config_path("quick")))
    c["synapse"].update({"d_e": d, "d_i": d, "d_a2n": d, "w_a2n": 0.5})
    c["astrocyte"].update({"Ca_init": 0.35, "IP3": 0.6})
    c["connectivity"].update({"pool_type": "random", "pool_size": 3, "p_third_if_primary": 0.6})
    c["simulation"]["seed"] = seed
    for k, v in sections.items():
        c[k].update(v)
    return Model(text=json.dumps(c), pre_time=0.0)


def compare(m, **opts):
    rec = _lib.RecordOpts(0, 7, 1, 20, 15)
    a = Network(m, record=rec, **opts)
    b = Network(m, record=rec, use_graphs=-1, **opts)
    for n in RUNS:
        a.step(n)
        b.step(n)
        for k, v in b.state().items():
            assert np.array_equal(a.state()[k], v), (n, k)
        for x, y in zip(a.fetch_spikes(), b.fetch_spikes()):
            assert np.array_equal(x, y), n
        ra, rb = a.fetch_record(), b.fetch_record()
        for k in rb:
            assert np.array_equal(ra[k], rb[k]), (n, k)
        assert a.counters() == b.counters()
    assert a.last_timing()[1] < b.last_timing()[1] == RUNS[-1]
    assert np.isfinite(a.state()["V"]).all() and a.counters()["sic_edges"] > 0


@pytest.mark.parametrize("occupancy", [1, 2])
@pytest.mark.parametrize("steps", [1, 2, 3])
@pytest.mark.parametrize("independent", [True, False])
def test_noise_intervals_shorter_than_a_launch(occupancy, steps, independent):
    z = {"noise_dt": 0.1 * steps, "independent_noise": independent}
    compare(model(input_exc=z, input_inh=z, input_astro=z), occupancy=occupancy)


@pytest.mark.parametrize("occupancy", [1, 2])
def test_poisson_counts_around_255(occupancy):
    # 255 and 250 events per step on average, of weights that leave the drive as it is
    compare(model(input_exc={"poiss_rate": 2.55e6, "poiss_weight": 0.001},
                  input_inh={"poiss_rate": 2.50e6, "poiss_weight": 0.001},
                  input_astro={"poiss_rate": 2.55e6, "poiss_weight": 1e-6}), occupancy=occupancy)


@pytest.mark.parametrize("occupancy", [1, 2])
@pytest.mark.parametrize("sic_mode", [1, 2])
def test_fp32_astrocytes(occupancy, sic_mode):
    compare(model(), occupancy=occupancy, sic_mode=sic_mode, astro_precision=32)


def test_tuned_network_and_restore_to_step_0():
    m = model()
    want = Network(m, use_graphs=-1)
    blob0 = want.checkpoint()
    want.step(200)
    a = Network(m)
    a.step(60)
    a.autotune(24)  # leaves the state
    a.step(140)
    for k, v in want.state().items():
        assert np.array_equal(a.state()[k], v), k
    for net in (a, Network(m)):
        for _ in range(2):
            net.restore(blob0)
            net.step(200)
            for k, v in want.state().items():
                assert np.array_equal(net.state()[k], v), k


def test_single_step_request_joins_and_leaves():
    long, short = model(5, N={"N_E": 900, "N_I": 200, "N_A": 300}), model(6, d=0.1)
    alone = []
    for m, n in ((long, 60_000), (short, 300)):
        net = Network(m, use_graphs=1)
        net.step(n)
        alone.append(net.fetch_spikes())
        assert net.counters()["sic_edges"] > 0
    s = Server()
    i = s.submit(long, 60_000)
    seen = []
    for _ in range(3):
        chunks = s.stats()["chunks"]
        while s.stats()["chunks"] < chunks + 4:
            time.sleep(0.0005)
        j = s.submit(short, 300)
        assert s.wait(j, timeout_ms=60_000).status == 0
        seen.append(s.fetch_spikes(j))
    assert not s.poll(i)[0]  # it ran throughout
    assert s.wait(i, timeout_ms=60_000).status == 0
    seen.append(s.fetch_spikes(i))
    s.close()
    for got, ref in zip(seen, [alone[1]] * 3 + [alone[0]]):
        for x, y in zip(got, ref):
            assert np.array_equal(x, y)
