"""SIC lists built on the device (sets of 2^16 edges and more) against the C
restatement: targets with more than 255 edges from one astrocyte (an entry's
multiplicity is split), pools of one and of many astrocytes, sizes that do not
fill the last slice of 32 targets, and a set just below and above the size
that takes the device path; and the target check of a large set."""
import ctypes as C
import json

import numpy as np
import pytest

from astrosimgpu_b200 import _lib
from astrosimgpu_b200.network import Model, Network, config_path
from oracle import config as oc

pytestmark = pytest.mark.gpu


def text(n_e, n_i, n_a, pool, p, p3):
    c = json.load(open(config_path("use_case")))
    c["N"].update({"N_E": n_e, "N_I": n_i, "N_A": n_a})
    c["connectivity"].update({"p_primary": p, "p_third_if_primary": p3, "pool_size": pool,
                              "pool_type": "random"})
    c["astrocyte"].update({"Ca_init": 0.35, "IP3": 0.6})
    c["synapse"]["w_a2n"] = 0.01
    return json.dumps(c)


@pytest.mark.parametrize("n_e,n_i,n_a,pool,p,p3", [(700, 33, 3, 1, 1.0, 1.0),
                                                   (307, 64, 257, 9, 0.8, 0.9),
                                                   (400, 97, 50, 2, 0.6, 0.54),
                                                   (400, 97, 50, 2, 0.6, 0.56)])
def test_sic_sums_against_restatement(n_e, n_i, n_a, pool, p, p3):
    t = text(n_e, n_i, n_a, pool, p, p3)
    net = Network(Model(text=t, pre_time=0.0), record=_lib.RecordOpts(0, 10, 1, 0, 0), sic_mode=1)
    net.step(40)
    port = oc.PortNetwork(oc.load(text=t))
    st, src = port.run(40)
    got, want = net.state(), port.state()
    assert np.array_equal(net.fetch_spikes()[0], st)
    assert np.abs(want["I_sic"]).max() > 0
    # the sums are the same additions in the same order; the factor's log may
    # differ in its last bit (2^-52 relative, well below the network tolerance)
    assert np.all(np.abs(got["I_sic"] - want["I_sic"]) <= 1e-12 * np.abs(want["I_sic"]))


def test_bad_target_of_a_large_set_is_refused():
    m = Model(config_path("scale_1000"), pre_time=0.0)
    d = m.desc()
    rs, tg = m.table(0)
    tg = tg.copy()
    tg[123456], tg[200000] = 5000, 7777
    bad = _lib.NetworkDesc.from_buffer_copy(d)
    bad.exc_primary.target = _lib.u32ptr(tg)
    h = C.c_void_p()
    st = _lib.load().asg_create(C.byref(bad), None, None, C.byref(h))
    assert st == 1 and not h
    assert b"exc_primary: target[123456] = 5000 out of range (5000)" in _lib.load().asg_last_error()
