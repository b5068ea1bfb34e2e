"""AUSM+ and HLLC fluxes next to nodes whose sound speed leaves the range of the fast reciprocal square
root, against the oracle: a pressure of exactly zero (no sound speed; the flux between it and a side of
positive pressure is finite), pressures whose product with the density is subnormal (a sound speed of
at most 1e-153, nothing beside the other side's whatever its digits), and for AUSM+ a node of negative
density and pressure, whose quotient is positive.  The odd nodes are isolated, so that first-order and
MUSCL (minmod) states take their values exactly."""
import os

import numpy as np
import pytest

import cb200
import helpers
from cb200 import abi, cases, mech as mechmod
from cb200.field import DeviceBlock

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")


def odd_nodes(hb, values, seed):
    """Isolated interior nodes (no two of them neighbours), one value of `values` after the other."""
    rng = np.random.default_rng(seed)
    g = hb.ngg
    at = [(k, j, i) for k in range(g, g + hb.mz, 3) for j in range(g, g + hb.my, 3) for i in range(g, g + hb.mx, 3)
          if rng.random() < 0.5]
    assert len(at) > 2 * len(values)
    return [(n, values[a % len(values)]) for a, n in enumerate(at)]


def compare(p, hb, faces):
    import torch
    import oracle_py
    dev = DeviceBlock(hb)
    ctx = cb200.Context(p)
    ctx.bind(0, dev.view(), faces)
    ctx.rhs(0, abi.RHS_INVISCID)
    torch.cuda.synchronize()
    got = dev.to_host(["dq"])["dq"]
    ctx.close()
    oracle_py.rhs(p, hb, faces, abi.RHS_INVISCID)
    assert np.isfinite(hb.a["dq"]).all()
    assert np.isfinite(got).all()
    assert helpers.rel_err(got, hb.a["dq"]) < 1e-12  # the bar of the parity tests


@pytest.mark.parametrize("rec", [abi.REC_FIRST, abi.REC_MUSCL], ids=["first", "muscl"])
@pytest.mark.parametrize("scheme", [abi.INV_AUSMP, abi.INV_HLLC], ids=["ausm", "hllc"])
def test_air(oracle_lib, scheme, rec):
    p, hb, faces = helpers.curvilinear_air_case(35, 12, 11, scheme=scheme, reconstruction=rec, seed=9)
    bv = hb.a["bv"]
    for (k, j, i), v in odd_nodes(hb, [0.0, 1e-310, 1e-308, 1e-200], 1):
        bv[4, k, j, i] = v
        bv[5, k, j, i] = 0.0
    cases.fill_cv_air(hb)
    compare(p, hb, faces)


def test_negative_density_and_pressure(oracle_lib):
    p, hb, faces = helpers.curvilinear_air_case(35, 12, 11, scheme=abi.INV_AUSMP, reconstruction=abi.REC_FIRST, seed=10)
    for (k, j, i), v in odd_nodes(hb, [-1.0], 2):
        hb.a["bv"][0, k, j, i] *= v
        hb.a["bv"][4, k, j, i] *= v
    cases.fill_cv_air(hb)
    compare(p, hb, faces)


@pytest.mark.parametrize("scheme", [abi.INV_AUSMP, abi.INV_HLLC], ids=["ausm", "hllc"])
def test_mixture(oracle_lib, scheme):
    mech = mechmod.load_json(os.path.join(GOLD, "h2_li2004.json"))
    c = cases.h2_air_box(mech, n_nodes=14, scheme=scheme, reconstruction=abi.REC_MUSCL, viscous_order=0, reaction=False)
    p, hb, faces = c.param, c.blocks[0], c.faces[0]
    for (k, j, i), v in odd_nodes(hb, [0.0, 1e-310], 3):
        hb.a["bv"][4, k, j, i] = v
    compare(p, hb, faces)


@pytest.mark.parametrize("scheme", [abi.INV_AUSMP, abi.INV_HLLC], ids=["ausm", "hllc"])
def test_two_temperatures(oracle_lib, scheme):
    path = os.path.join(GOLD, "air5_park.json")
    mech, tt = mechmod.load_json(path), mechmod.load_two_temperature_json(path)
    c = cases.air5_box_2t(mech, tt, n_nodes=12, reaction=False, scheme=scheme, reconstruction=abi.REC_MUSCL)
    p, hb, faces = c.param, c.blocks[0], c.faces[0]
    oracle_lib.cv_from_bv(p, hb)
    for (k, j, i), v in odd_nodes(hb, [0.0, 1e-310], 4):
        hb.a["bv"][4, k, j, i] = v
    compare(p, hb, faces)
