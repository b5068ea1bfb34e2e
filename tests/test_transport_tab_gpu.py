"""The FP64 property kernels on a repacked mechanism against the oracle: padded planes around the
edges of their tiles of 128 nodes, 2-D blocks (one plane evaluated, the ghost planes copied),
temperatures in both ranges of the NASA7 fits and beyond them, absent species, five species, and a
mechanism whose transport data do not fit a table (a zero well depth), which runs the generic kernel."""
import copy
import os

import numpy as np
import pytest

import helpers
import oracle_py
from cb200 import abi, cases, mech as mechmod
from cb200.field import HostBlock, array_specs

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden", "h2_li2004.json")
NAMES = ("mul", "thermal_conductivity", "rho_D", "acoustic_speed", "gamma", "mach")


@pytest.mark.parametrize("dims,kind", [((1, 1, 1), "h2"), ((10, 2, 2), "h2"), ((11, 2, 2), "h2"), ((58, 1, 3), "h2"),
                                       ((19, 14, 5), "h2"), ((21, 9, 1), "planar"), ((9, 5, 4), "mixed_middles"),
                                       ((9, 5, 4), "generic"), ((19, 14, 5), "five"), ((21, 9, 1), "planar_five")])
def test_properties_against_oracle(dims, kind):
    import torch
    import cb200
    from cb200.field import DeviceBlock
    mech = mechmod.load_json(GOLD)
    if kind in ("mixed_middles", "generic"):
        d = copy.deepcopy(mech.d)
        if kind == "mixed_middles":  # the thermodynamic table needs one middle temperature
            d["t_mid"][3] = 1100.0
        else:
            d["sqrt_WiDivWjPl1Mul8"][5] = -1.0  # never so in earnest: only the generic kernel takes it
        mech = mechmod.MechStruct(d)
    elif kind.endswith("five"):
        mech = helpers.sub_mechanism(mech, ("H", "O2", "O", "OH", "HO2"))
    planar = kind.startswith("planar")
    rng = np.random.default_rng(sum(dims))
    g = 3
    b = HostBlock(*dims, g, array_specs(*dims, g, 5 + mech.ns, mech.ns))
    shape = b.a["bv"][0].shape
    y = rng.uniform(0, 1, (mech.ns,) + shape) ** 4
    y[2][rng.uniform(0, 1, shape) < 0.2] = 0.0
    y /= y.sum(axis=0)
    b.a["sv"][...] = y
    b.a["bv"][0] = rng.uniform(0.05, 2.0, shape)
    for c in range(1, 4):
        b.a["bv"][c] = rng.uniform(-900, 900, shape)
    b.a["bv"][4] = 1e5
    b.a["bv"][5] = rng.choice([180.0, 299.0, 300.0, 999.0, 1000.0, 1001.0, 1700.0, 3500.0, 3600.0, 5200.0], shape)
    if planar:  # eliminate_k_gradient leaves copies of plane 0 on the ghost planes
        for name in ("bv", "sv"):
            b.a[name][:] = b.a[name][:, g:g + 1]
    p = cases.make_param(n_var=5 + mech.ns, n_spec=mech.ns, dim=2 if planar else 3, inviscid_scheme=abi.INV_HLLC,
                         reconstruction=abi.REC_MUSCL, rho_ref=1.0, v_ref=700.0, mech=mech.ptr())
    dev = DeviceBlock(b)
    ctx = cb200.Context(p)
    ctx.bind(0, dev.view(), [])
    ctx.properties(0)
    torch.cuda.synchronize()
    got = dev.to_host(NAMES)
    ctx.close()
    oracle_py.properties(p, b)
    for n in NAMES:
        # sums of at most 81 products of powers with exponents up to 2.2 of arguments known to an ulp
        assert np.isfinite(b.a[n]).all()
        bar = 5e-14
        if n == "rho_D":
            # its numerator is the mixture's sum of m species less the species' own share Y: the rounding
            # of the sum, at most half an ulp for each species, counts 1 / (1 - Y) times
            bar = bar + mech.ns * 2.0 ** -53 / (1 - y)
        assert (np.abs(got[n] - b.a[n]) <= bar * np.abs(b.a[n])).all(), n
