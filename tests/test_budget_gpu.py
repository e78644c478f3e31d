"""The memory budget holds for all that instances keep on the device: their
arenas and the buffers of launches of several steps.  The buffers are taken
only where the budget has room beside the arenas -- otherwise launches take one
step each, with the same bits -- and a request that fits the budget of a server
is admitted beside running ones as if there were no such buffers."""
import re
import time

import numpy as np
import pytest

from astrosimgpu_b200 import _lib, workloads
from astrosimgpu_b200.network import Batch, Model, Network, Server, config_path

pytestmark = pytest.mark.gpu


def serving(n, seed=3):
    return Model(text=workloads.serving_config(n, seed, 100.0), pre_time=0.0, fixed_indegree=100,
                 gen_device=0)


def test_one_step_per_launch_without_room():
    m = Model(config_path("quick"), pre_time=0.0)
    free = Network(m)
    arena = len(free.checkpoint()) - 8
    free.step(200)
    tight, roomy = Network(m, mem_budget=arena), Network(m, mem_budget=arena + (16 << 20))
    for net in (tight, roomy):
        net.step(200)
        for k, v in free.state().items():
            assert np.array_equal(net.state()[k], v), k
    assert tight.last_timing()[1] == 200
    assert roomy.last_timing()[1] == free.last_timing()[1] < 100
    with pytest.raises(_lib.AsgError):
        Network(m, mem_budget=arena - 1)


def test_a_batch_stays_within_its_budget():
    """Three arenas fill the budget: none of the instances holds more."""
    import torch
    models = [serving(100_000, s) for s in (1, 2, 3)]
    one = Network(models[0])
    arena = len(one.checkpoint()) - 8
    one.close()
    used = {}
    for name, budget in (("plenty", 0), ("tight", 3 * arena + (1 << 20))):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        b = Batch(models, mem_budget=budget)
        b.step(20)
        used[name] = before - torch.cuda.mem_get_info()[0]
        kernels = b.last_timing()[1]
        b.close()
    # 100,000 cells x 5 steps x 2 lists x 32 bytes, and 18 rows of factors each
    buffers = 3 * (32_000_000 + 18 * 800_000)
    assert kernels == 20
    assert used["plenty"] > 3 * arena + buffers // 2
    assert used["tight"] < 3 * arena + buffers // 4


def test_a_request_is_admitted_beside_the_buffers_of_a_running_one():
    a, b = serving(20_000, 5), serving(20_000, 6)
    with pytest.raises(_lib.AsgError) as e:
        Server(mem_budget=1).submit(a, 10)
    need = int(re.search(r"needs ~(\d+) device bytes", str(e.value)).group(1))
    alone = []
    for m, n in ((a, 40_000), (b, 500)):
        net = Network(m)
        net.step(n)
        alone.append(net.fetch_spikes())
    s = Server(mem_budget=2 * need + (1 << 20))
    i = s.submit(a, 40_000)
    while s.stats()["chunks"] < 4:
        time.sleep(0.001)
    first = s.stats()
    assert first["kernels"] < 64 * first["chunks"] / 2  # it runs several steps per launch
    j = s.submit(b, 500)
    for k, want in ((j, alone[1]), (i, alone[0])):
        assert s.wait(k, timeout_ms=60_000).status == 0
        for x, y in zip(s.fetch_spikes(k), want):
            assert np.array_equal(x, y)
    assert s.stats()["peak_resident"] == 2
    s.close()


def arena_of(m):
    net = Network(m)
    size = len(net.checkpoint()) - 8
    net.close()
    return size


def test_a_server_keeps_memory_beside_large_requests():
    """What a request leaves stays with the server's pool for the next one (at
    most 2 GB), also where the requests that run on hold more than that."""
    import torch
    m, small = serving(150_000, 4), serving(20_000, 5)
    assert arena_of(m) > (2 << 30)
    before = torch.cuda.mem_get_info()[0]

    def held():
        return before - torch.cuda.mem_get_info()[0]

    s = Server()
    i = s.submit(m, 200_000)
    while s.stats()["chunks"] < 4:
        time.sleep(0.001)
    s.wait(s.submit(small, 64))
    with_small, least = held(), 1 << 60
    for _ in range(4):
        j = s.submit(small, 64)
        while not s.poll(j)[0]:
            least = min(least, held())
    s.cancel(i)
    s.wait(i)
    s.close()
    assert least > with_small - (64 << 20), (least, with_small)


def test_a_server_keeps_no_more_than_its_budget():
    import torch
    m = serving(20_000, 5)
    arena = arena_of(m)
    before = torch.cuda.mem_get_info()[0]
    with pytest.raises(_lib.AsgError) as e:
        Server(mem_budget=1).submit(m, 10)
    need = int(re.search(r"needs ~(\d+) device bytes", str(e.value)).group(1))
    small = Server(mem_budget=need)
    assert small.wait(small.submit(m, 100)).status == 0
    torch.cuda.synchronize()
    held = before - torch.cuda.mem_get_info()[0]
    small.close()
    assert held < need + (48 << 20), (held, need, arena)
