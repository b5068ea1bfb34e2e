"""Outflow faces that fill in one launch, and those that must not, against the oracle, which fills the
faces one after the other: a back-pressure face opposite an outflow face on blocks of at most as many
nodes across as there are ghost layers (its reads are the other face's ghosts) and on the first that
are thicker; more faces than one launch takes; sub-faces that touch and that overlap; faces extended
into the tangential ghosts (2nd-order viscous terms).  The bar is the one of the ghost-fill tests."""
import numpy as np
import pytest

import cb200
import helpers
from cb200 import abi
from cb200.field import DeviceBlock, face

pytestmark = pytest.mark.gpu


def whole(dims, d, s, p=0.0, lo=None, hi=None):
    start, end = list(lo or (0, 0, 0)), list(hi or (m - 1 for m in dims))
    start[d] = end[d] = 0 if s < 0 else dims[d] - 1
    return face(abi.BC_OUTFLOW, d, s, start, end, p=p)


def check(oracle, dims, faces, viscous=0):
    import torch
    p, hb, _ = helpers.curvilinear_air_case(*dims, scheme=abi.INV_HLLC, viscous_order=viscous, bc="outflow", seed=sum(dims))
    first = None
    for _ in range(4):
        dev = DeviceBlock(hb)
        ctx = cb200.Context(p)
        ctx.bind(0, dev.view(), faces)
        ctx.boundary(0)
        torch.cuda.synchronize()
        out = dev.to_host(["bv", "cv"])
        ctx.close()
        first = first or out
        assert all(np.array_equal(out[n], first[n]) for n in out)
    oracle.boundary(p, hb, faces)
    for n in ("bv", "cv"):
        assert np.isfinite(hb.a[n]).all()
        assert helpers.rel_err(first[n], hb.a[n]) < 1e-13


@pytest.mark.parametrize("left", [0.0, 1.05], ids=["outflow", "back_pressure"])
@pytest.mark.parametrize("d", [0, 1, 2])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5])
def test_back_pressure_across_a_thin_block(oracle_lib, m, d, left):
    dims = [67, 9, 8]
    dims[d] = m
    check(oracle_lib, dims, [whole(dims, d, -1, p=left), whole(dims, d, 1, p=0.95)])
    check(oracle_lib, dims, [whole(dims, d, 1, p=0.95), whole(dims, d, -1, p=left)])


@pytest.mark.parametrize("viscous", [0, 2])
def test_more_faces_than_a_launch_takes(oracle_lib, viscous):
    dims = (18, 13, 11)
    faces = []
    for d in range(3):
        t = (d + 1) % 3
        for s in (-1, 1):
            mid, lo, hi = dims[t] // 2, [0, 0, 0], [m - 1 for m in dims]
            lo[t], hi[t] = mid + 1, mid
            faces += [whole(dims, d, s, hi=hi), whole(dims, d, s, p=0.9 + 0.01 * d, lo=lo)]
    check(oracle_lib, dims, faces, viscous)


@pytest.mark.parametrize("gap", [1, 0, -2], ids=["touch", "share_a_line", "overlap"])
def test_sub_faces_of_one_side(oracle_lib, gap):
    dims = (15, 20, 9)
    cut = 9
    faces = [whole(dims, 0, 1, hi=(0, cut, 8)), whole(dims, 0, 1, p=0.93, lo=(0, cut + gap, 0)), whole(dims, 0, -1, p=1.1)]
    check(oracle_lib, dims, faces)
