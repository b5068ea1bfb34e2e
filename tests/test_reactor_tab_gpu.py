"""Batched ROK4E reactors on the repacked mechanism against the oracle, attempt by attempt: five species
(another lane layout than nine), the longest mechanism and the longest side of a reaction that fit a
table, temperatures that start and move beyond the fits, third bodies that are absent, and a mechanism
with two middle temperatures, which runs the generic kernel."""
import ctypes as C
import copy
import os

import numpy as np
import pytest

import cb200
import helpers
from cb200 import abi, cases, mech as mechmod
from test_chemistry_tab_gpu import mechanism

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden", "h2_li2004.json")
FUEL = {"H2": 2.0, "O2": 1.0, "N2": 3.76}
RADICALS = {"H": 1.0, "O2": 1.0, "O": 0.4, "OH": 0.2}


def setting(kind):
    """(mechanism, mole numbers, T0, p0, h0, attempts)"""
    if kind == "ceiling":  # every fit ends at 1500 K: the ignition leaves it
        d = copy.deepcopy(mechmod.load_json(GOLD).d)
        d["t_high"] = [1500.0] * 9
        return mechmod.MechStruct(d), dict(FUEL, H=0.1), [1450.0, 1499.9, 1500.1, 2000.0], 2e6, 1e-7, 12
    if kind == "cold":  # below the fits: 200 K, 300 K for N2
        return mechmod.load_json(GOLD), RADICALS, [150.0, 195.0, 250.0, 299.0, 305.0], 1e5, 1e-8, 12
    m = mechanism(kind)
    if kind in ("five", "five_h2"):
        x = RADICALS if kind == "five" else dict(RADICALS, H2=1.0)
        return m, x, [900.0, 999.9, 1500.0, 2500.0, 4000.0], 3e5, 1e-8, 12
    if kind == "eight":
        # a first step near the error bound: from 1e-10 s the error norm of the first attempts is all
        # rounding, and an ulp of T0 moves the oracle's own time by 3e-9
        return m, dict(FUEL, H=0.01), [1100.0, 1300.0], 1e5, 1e-6, 12
    if kind == "no_body":
        return m, FUEL, [1100.0, 1500.0, 3000.0], 1e6, 1e-7, 12
    return m, dict(FUEL, H=0.01), [950.0, 1100.0, 1500.0], 1e6, 1e-7, 12


KINDS = ["h2", "full", "eight", "five", "five_h2", "ceiling", "cold", "no_body", "middles"]
RTOL, ATOL, T_END = 1e-6, 1e-6, 1.0


def composition(m, x):
    y = np.array([x.get(n, 0.0) * w for n, w in zip(m.species, m.mw)])
    return y / y.sum()


@pytest.mark.parametrize("kind", KINDS)
def test_reactors_against_oracle(oracle_lib, kind):
    import torch
    m, x, t0, p0, h0, attempts = setting(kind)
    n, y = len(t0), composition(m, x)
    p = cases.make_param(n_var=5 + m.ns, n_spec=m.ns, dim=1, inviscid_scheme=abi.INV_HLLC, reconstruction=abi.REC_WENO5,
                         mech=m.ptr())
    ctx = cb200.Context(p)

    def dev(a):
        return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")

    st = torch.zeros(n * C.sizeof(abi.Reactor), dtype=torch.uint8, device="cuda")
    args = dev(t0), dev([p0] * n), dev(np.tile(y, (n, 1))), dev([T_END] * n)
    ctx.reactor_setup(st.data_ptr(), n, *(a.data_ptr() for a in args), h0)
    ctx.reactor_advance(st.data_ptr(), n, attempts, RTOL, ATOL)
    torch.cuda.synchronize()
    raw = st.cpu().numpy().tobytes()
    ctx.close()
    for i in range(n):
        s = abi.Reactor.from_buffer_copy(raw, i * C.sizeof(abi.Reactor))
        o = oracle_lib.reactor_run(m, t0[i], p0, y, T_END, h0, RTOL, ATOL, max_attempts=attempts)
        assert (s.step, s.n_reject, s.status) == (o.step, o.n_reject, o.status)
        # the bar of the reactor tests: the controller's powers of the error norm move the steps by 1e-10
        assert abs(s.time - o.time) <= 1e-9 * o.time
        assert abs(s.T - o.T) <= 1e-9 * o.T
        assert abs(s.p - o.p) <= 1e-9 * o.p
        a, b = (np.array(list(q.rhoY)[:m.ns]) for q in (s, o))
        assert np.abs(a - b).max() <= 1e-9 * b.max()
