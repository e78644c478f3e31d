"""An admission that runs out of device memory anywhere -- the targets, a
ring's numbering, the SIC lists, the arena -- is repeated with one set's tables
on the device at a time, and gives the same network.  One allocation is made to
fail on the host; each process tries another one."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import sys
sys.path.insert(0, %r)
import hashlib
from astrosimgpu_b200.network import Model, Network, config_path
m = Model(config_path("scale_1000"), pre_time=0.0)
net = Network(m, sic_mode=int(sys.argv[1]))
net.step(150)
h = hashlib.sha256()
for k, v in sorted(net.state().items()):
    h.update(v.tobytes())
print(net.counters()["spikes"], h.hexdigest())
""" % ROOT


@pytest.mark.parametrize("sic_mode", [1, 2])  # uncut lists (device), cut chains (host)
def test_every_allocation_may_fail_once(sic_mode):
    outs = {}
    todo = ["0", "2", "5", "9", "10", "12", "17", "21", "28", "40", "47", "52", "54", "55", "56"]
    for k in range(0, len(todo), 5):
        procs = {at: subprocess.Popen([sys.executable, "-c", CODE, str(sic_mode)],
                                      env=dict(os.environ, ASG_FAIL_SCRATCH_AT=at), text=True,
                                      stdout=subprocess.PIPE, stderr=subprocess.PIPE)
                 for at in todo[k:k + 5]}
        for at, p in procs.items():
            out, err = p.communicate(timeout=120)
            assert p.returncode == 0, (at, err[-800:])
            outs[at] = out
    assert int(outs["0"].split()[0]) > 0
    for at, out in outs.items():
        assert out == outs["0"], at
