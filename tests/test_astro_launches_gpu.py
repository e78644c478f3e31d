"""A call of the astrocyte workload runs as launches of bounded length: at most
2^17 substeps of a cell each, however small the population.  Splitting a call,
by the engine or by the caller, changes no bit."""
import numpy as np
import pytest

from astrosimgpu_b200.astro import AstroBackend, ScalingWorkload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
def test_a_long_call_of_a_small_population_is_several_launches(precision):
    w = ScalingWorkload(7, substeps=400)  # 327 steps per launch
    got = []
    for calls in ((700,), (300, 400), (327, 327, 46)):
        g = AstroBackend(*w.initial_state())
        run = g.run_bernoulli if precision == 64 else g.run_bernoulli_f32
        first, kernels = 0, []
        for n in calls:
            kernels.append(run(w, first, n)[1])
            first += n
        got.append(g.pull_state())
        assert kernels == [-(-n // 327) for n in calls]
    for a in got[1:]:
        for x, y in zip(a, got[0]):
            assert np.array_equal(x, y)
