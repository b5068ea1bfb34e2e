"""Walls and farfield faces on blocks of two and three nodes across, an outflow opposite, against the
oracle, which takes the layers of a face node in order: with two nodes the node inside lies on the
opposite boundary and is moved onto the face itself, so that the ghosts mirror the state that the fill
has just written there."""
import os

import numpy as np
import pytest

import cb200
import helpers
from cb200 import abi, cases, mech as mechmod
from cb200.field import DeviceBlock, face

pytestmark = pytest.mark.gpu
AIR5 = os.path.join(os.path.dirname(__file__), "golden", "air5_park.json")


def pair(dims, d, s, kind, **state):
    """The face under test on side s of direction d, an outflow on the other side."""
    out = []
    for side in (-1, 1):
        start, end = [0, 0, 0], [m - 1 for m in dims]
        start[d] = end[d] = 0 if side < 0 else dims[d] - 1
        out.append(face(kind, d, s, start, end, **state) if side == s else face(abi.BC_OUTFLOW, d, side, start, end))
    return out


def check(oracle, p, hb, faces, names):
    import torch
    first = None
    for _ in range(4):
        dev = DeviceBlock(hb)
        ctx = cb200.Context(p)
        ctx.bind(0, dev.view(), faces)
        ctx.boundary(0)
        torch.cuda.synchronize()
        out = dev.to_host(names)
        ctx.close()
        first = first or out
        assert all(np.array_equal(out[n], first[n], equal_nan=True) for n in out)
    oracle.boundary(p, hb, faces)
    for n in names:
        assert np.isfinite(hb.a[n]).all()
        assert helpers.rel_err(first[n], hb.a[n]) < 1e-12  # the bar of the step tests: T_ve is an inversion


@pytest.mark.parametrize("kind", ["isothermal", "adiabatic", "farfield"])
@pytest.mark.parametrize("s", [-1, 1])
@pytest.mark.parametrize("d", [0, 1, 2])
@pytest.mark.parametrize("m", [2, 3])
def test_air(oracle_lib, m, d, s, kind):
    dims = [35, 9, 8]
    dims[d] = m
    p, hb, _ = helpers.curvilinear_air_case(*dims, scheme=abi.INV_HLLC, bc="outflow", seed=sum(dims))
    if kind == "farfield":
        faces = pair(dims, d, s, abi.BC_FARFIELD, rho=0.9, u=0.5, v=-0.3, w=0.4, p=1.05, T=1.05 / (0.9 * cases.R_AIR))
    else:
        faces = pair(dims, d, s, abi.BC_WALL, wall_temperature=0.8 / cases.R_AIR if kind == "isothermal" else 0.0)
    check(oracle_lib, p, hb, faces, ["bv", "cv"])


@pytest.mark.parametrize("m", [2, 3])
def test_two_temperature_wall(oracle_lib, m):
    from cb200.field import HostBlock
    mech, tt = mechmod.load_json(AIR5), mechmod.load_two_temperature_json(AIR5)
    c = cases.air5_box_2t(mech, tt, n_nodes=12)
    p, box = c.param, c.blocks[0]
    dims = (12, m, 12)
    hb = HostBlock(*dims, box.ngg, box.specs)
    for n, a in hb.a.items():
        a[...] = box.a[n][:, :a.shape[1], :a.shape[2], :a.shape[3]]
    oracle_lib.cv_from_bv(p, hb)
    check(oracle_lib, p, hb, pair(dims, 1, 1, abi.BC_WALL, wall_temperature=900.0, wall_temperature_ve=700.0),
          ["bv", "cv", "sv", "temperature_ve"])
