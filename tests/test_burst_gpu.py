"""The opening burst of a large network (10^5 spikes in a chunk), in calls of many
steps, whose launches take several each, and of a few, whose launches take one:
the bits of single steps throughout, and the spikes in order."""
import numpy as np
import pytest

from astrosimgpu_b200 import _lib, workloads
from astrosimgpu_b200.network import Model, Network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sic_mode", [0, 2])  # SIC by the neuron's thread, by its own role
def test_opening_burst_same_bits(sic_mode):
    m = Model(text=workloads.serving_config(200_000, 3, 100.0), pre_time=0.0, fixed_indegree=100,
              gen_device=0)
    rec = _lib.RecordOpts(0, 9, 1, 40, 40)
    a = Network(m, record=rec, sic_mode=sic_mode)
    b = Network(m, record=rec, sic_mode=sic_mode, use_graphs=-1)
    for n in (96, 60, 3, 1, 64, 6, 31):
        a.step(n)
        b.step(n)
        for k, v in a.state().items():
            assert np.array_equal(v, b.state()[k]), (n, k)
        (at, of), (at_b, of_b) = a.fetch_spikes(), b.fetch_spikes()
        assert np.array_equal(at, at_b) and np.array_equal(of, of_b), n
        assert np.array_equal(np.lexsort((of, at)), np.arange(len(at))), n
        ra, rb = a.fetch_record(), b.fetch_record()
        for k in ra:
            assert np.array_equal(ra[k], rb[k]), (n, k)
        assert a.counters() == b.counters()
