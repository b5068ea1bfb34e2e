"""Residuals at block sizes around the edges of the sweep tiles, against the oracle: runs of a k plane
along x around 510 and 254 nodes; 14, 30 or 62 own nodes by 16 or 8 columns along y and z; 30 (x) and 14 (y, z) own
nodes of the 2nd-order viscous tiles.  One residual at 1e-12 of each variable's largest value, the bar
of the parity tests.  Whole steps of a mixture of five species with NASA7 fits."""
import os

import numpy as np
import pytest

import helpers
import oracle_py
from cb200 import abi, cases, mech as mechmod

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden", "h2_li2004.json")


def gpu_rhs(p, hb, faces):
    import torch
    import cb200
    from cb200.field import DeviceBlock
    dev = DeviceBlock(hb)
    ctx = cb200.Context(p)
    ctx.bind(0, dev.view(), faces)
    ctx.rhs(0)
    torch.cuda.synchronize()
    out = dev.to_host(["dq"])["dq"]
    ctx.close()
    return out


@pytest.mark.parametrize("dims", [(16, 30, 6), (17, 31, 6), (8, 62, 6), (9, 63, 6), (6, 6, 33), (57, 8, 6), (43, 10, 6), (15, 14, 15)])
@pytest.mark.parametrize("scheme,rec", [(abi.INV_AUSMP, abi.REC_WENO7), (abi.INV_HLLC, abi.REC_WENO5), (abi.INV_WENO7_CH, abi.REC_MUSCL)],
                         ids=["ausm_weno7", "hllc_weno5", "weno7_ch"])
def test_air_sweeps(dims, scheme, rec):
    p, hb, faces = helpers.curvilinear_air_case(*dims, scheme=scheme, reconstruction=rec, seed=sum(dims))
    got = gpu_rhs(p, hb, faces)
    oracle_py.rhs(p, hb, faces)
    assert helpers.rel_err(got, hb.a["dq"]) < 1e-12


@pytest.mark.parametrize("n", [13, 14, 15, 16, 17, 29, 31])
def test_mixture_sweeps_and_viscous(n):
    mech = mechmod.load_json(GOLD)
    c = cases.h2_air_box(mech, n_nodes=n, seed=n)
    p, hb, faces = c.param, c.blocks[0], c.faces[0]
    rng = np.random.default_rng(n)
    y = hb.a["sv"] + rng.uniform(0, 0.02, hb.a["sv"].shape)
    hb.a["sv"][...] = y / y.sum(axis=0)
    oracle_py.cv_from_bv(p, hb)
    oracle_py.properties(p, hb)
    got = gpu_rhs(p, hb, faces)
    oracle_py.rhs(p, hb, faces)
    assert helpers.rel_err(got, hb.a["dq"]) < 1e-12


@pytest.mark.parametrize("scheme,rec", [(abi.INV_HLLC, abi.REC_WENO5), (abi.INV_AUSMP, abi.REC_MUSCL), (abi.INV_WENO5_CH, abi.REC_MUSCL)],
                         ids=["hllc_weno5", "ausm_muscl", "weno5_ch"])
def test_five_species_steps(scheme, rec):
    import torch
    import cb200
    from cb200.field import DeviceBlock
    mech = helpers.sub_mechanism(mechmod.load_json(GOLD), ("H2", "O2", "HO2", "H", "N2"))
    c = cases.h2_air_box(mech, n_nodes=15, seed=5, scheme=scheme, reconstruction=rec)
    p, hb, faces = c.param, c.blocks[0], c.faces[0]
    y = hb.a["sv"] + np.random.default_rng(5).uniform(0, 0.02, hb.a["sv"].shape)
    hb.a["sv"][...] = y / y.sum(axis=0)
    oracle_py.cv_from_bv(p, hb)
    oracle_py.boundary(p, hb, faces)
    oracle_py.properties(p, hb)
    dev = DeviceBlock(hb)
    ctx = cb200.Context(p)
    ctx.bind(0, dev.view(), faces)
    for _ in range(3):
        ctx.rk3_step(2e-9)
        oracle_py.rk3_step(p, [hb], [faces], 2e-9)
    torch.cuda.synchronize()
    out = dev.to_host(["cv", "bv", "sv"])
    ctx.close()
    g = hb.ngg
    sl = (slice(None), slice(g, -g), slice(g, -g), slice(g, -g))
    for n in out:
        assert helpers.rel_err(out[n][sl], hb.a[n][sl]) < 3e-12, n  # the bar of the step tests
