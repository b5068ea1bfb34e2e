"""Batched closed blocks (cb2_block_batch_advance): uneven 2-D and 3-D periodic air blocks, every phase of
a step in one launch over all of them, must give, block by block, the same bits as cb2_rk3_step on that
block, with fixed and CFL steps, whatever other blocks share the batch (failing ones among them) and
whatever tile width is set or tuned."""
import numpy as np
import pytest

import cb200
from cb200 import abi
from cb200.field import DeviceBlock

import helpers

pytestmark = pytest.mark.gpu

DIMS = [(20, 18, 16), (30, 12, 10), (16, 14, 1), (12, 12, 12)]


def _sync():
    import torch
    torch.cuda.synchronize()


def _blocks(oracle, scheme, rec, dims=DIMS, seed=21):
    out = []
    for a, d in enumerate(dims):
        p, hb, faces = helpers.curvilinear_air_case(*d, scheme=scheme, reconstruction=rec, viscous_order=0,
                                                    bc="periodic", seed=seed + a)
        if d[2] == 1:
            # a closed 2-D block: periodic i and j faces, the k direction collapsed
            p.dim = 2
            faces = [f for f in faces if f.face < 2]
        oracle.boundary(p, hb, faces)
        out.append((p, hb, faces))
    return out


def _reference(p, hb, faces, steps, dt):
    dev = DeviceBlock(hb)
    ctx = cb200.Context(p)
    ctx.bind(0, dev.view(), faces)
    t = 0.0
    for _ in range(steps):
        t += ctx.rk3_step(dt, fixed_dt=dt > 0)
    _sync()
    return dev.to_host(["cv", "bv"]), t


def _batch(ctx, blocks, steps, dt, t_end=1e30):
    devs = [DeviceBlock(hb) for _, hb, _ in blocks]
    cases = (abi.BlockCase * len(blocks))()
    for c, d in zip(cases, devs):
        c.zone = d.view()
        c.time, c.t_end, c.dt = 0.0, t_end, dt
    ctx.block_batch_advance(cases, steps)
    _sync()
    return devs, cases


@pytest.mark.parametrize("scheme,rec", [(abi.INV_AUSMP, abi.REC_WENO7), (abi.INV_HLLC, abi.REC_WENO5)],
                         ids=["ausm_weno7", "hllc_weno5"])
@pytest.mark.parametrize("cfl", [False, True], ids=["fixed_dt", "cfl_dt"])
def test_batch_matches_block_path(oracle_lib, scheme, rec, cfl):
    blocks = _blocks(oracle_lib, scheme, rec)
    p0 = blocks[0][0]
    dts = [0.0 if cfl else 0.2 * oracle_lib.cfl_dt(p, hb) for p, hb, _ in blocks]
    ctx = cb200.Context(p0)
    devs = [DeviceBlock(hb) for _, hb, _ in blocks]
    cases = (abi.BlockCase * len(blocks))()
    for c, d, dt in zip(cases, devs, dts):
        c.zone = d.view()
        c.time, c.t_end, c.dt = 0.0, 1e30, dt
    ctx.block_batch_advance(cases, 4)
    _sync()
    for (p, hb, faces), d, c, dt in zip(blocks, devs, cases, dts):
        ref, t_ref = _reference(p, hb, faces, 4, dt)
        out = d.to_host(["cv", "bv"])
        assert c.steps == 4 and c.status == 0
        assert c.time == t_ref
        for n in ("cv", "bv"):
            assert np.array_equal(out[n], ref[n]), (hb.mx, hb.my, hb.mz, n)


def _cases_for(blocks, dt):
    devs = [DeviceBlock(hb) for _, hb, _ in blocks]
    cases = (abi.BlockCase * len(blocks))()
    for c, d in zip(cases, devs):
        c.zone = d.view()
        c.time, c.t_end, c.dt = 0.0, 1e30, dt
    return cases, devs


def test_batch_result_independent_of_company_and_tiles(oracle_lib):
    blocks = _blocks(oracle_lib, abi.INV_AUSMP, abi.REC_WENO7)
    dt = 0.2 * min(oracle_lib.cfl_dt(p, hb) for p, hb, _ in blocks)
    ctx = cb200.Context(blocks[0][0])
    alone, _ = _batch(ctx, blocks[1:2], 3, dt)
    ref = alone[0].to_host(["cv"])["cv"]
    for w in (4, 8, 16):
        ctx.block_batch_set_schedule(w, 8)
        for company in ((1,), (0, 1, 2, 3), (2, 1), (3, 1, 0, 1)):
            together, cases = _batch(ctx, [blocks[c] for c in company], 3, dt)
            for c, d in zip(company, together):
                if c == 1:
                    assert np.array_equal(d.to_host(["cv"])["cv"], ref), (w, company)
    tune_cases, keep = _cases_for(blocks, dt)
    ni, cs = ctx.block_batch_autotune(tune_cases)
    assert ni in (4, 8, 16) and cs == 8  # the cluster size is the one last set
    # tuning touched only the residual scratch dq
    for (_, hb, _), d in zip(blocks, keep):
        assert np.array_equal(d.to_host(["cv"])["cv"], hb.a["cv"])


def test_autotune_times_the_residual_of_every_block(oracle_lib):
    """Blocks at or past their end time too: each candidate width leaves every block's residual in dq."""
    blocks = _blocks(oracle_lib, abi.INV_AUSMP, abi.REC_WENO7)
    ctx = cb200.Context(blocks[0][0])
    cases, devs = _cases_for(blocks, 1e-3)
    for c, (t, t_end) in zip(cases, ((0.0, 0.0), (0.0, 1.0), (2.0, 1.0), (0.5, 0.5))):
        c.time, c.t_end = t, t_end
    ctx.block_batch_autotune(cases)
    for (p, hb, faces), d in zip(blocks, devs):
        one = DeviceBlock(hb)
        path = cb200.Context(p)
        path.bind(0, one.view(), faces)
        path.rhs(0)
        _sync()
        assert np.array_equal(d.to_host(["dq"])["dq"], one.to_host(["dq"])["dq"]), (hb.mx, hb.my, hb.mz)
        path.close()


def test_batch_stops_each_block_at_its_end_time(oracle_lib):
    blocks = _blocks(oracle_lib, abi.INV_HLLC, abi.REC_WENO5)[:3]
    ctx = cb200.Context(blocks[0][0])
    devs = [DeviceBlock(hb) for _, hb, _ in blocks]
    cases = (abi.BlockCase * 3)()
    dt = 0.2 * min(oracle_lib.cfl_dt(p, hb) for p, hb, _ in blocks)
    for c, d, n in zip(cases, devs, (2.5, 4.5, 7.5)):
        c.zone = d.view()
        c.time, c.t_end, c.dt = 0.0, n * dt, dt
    ctx.block_batch_advance(cases, 100)
    assert [c.steps for c in cases] == [3, 5, 8]
    assert all(c.status == abi.BLOCK_DONE for c in cases)


@pytest.mark.parametrize("kind", ["cfl", "update"])
def test_batch_reports_failed_blocks(oracle_lib, kind):
    """A block whose CFL step is not a number stops before it; one whose update leaves the physical range
    runs on and is reported; the others do not notice."""
    blocks = _blocks(oracle_lib, abi.INV_AUSMP, abi.REC_WENO7)
    bad, steps = 1, 3
    dts = [0.0 if kind == "cfl" else 0.2 * oracle_lib.cfl_dt(p, hb) for p, hb, _ in blocks]
    if kind == "cfl":
        hb = blocks[bad][1]
        hb.a["bv"][5, hb.ngg + 2, hb.ngg + 3, hb.ngg + 4] = np.nan
    else:
        dts[bad] *= 1e4
    cases, devs = _cases_for(blocks, 0.0)
    for c, dt in zip(cases, dts):
        c.dt = dt
    ctx = cb200.Context(blocks[0][0])
    ctx.block_batch_advance(cases, steps)
    _sync()
    assert cases[bad].status == abi.BLOCK_FAILED
    if kind == "cfl":
        assert cases[bad].steps == 0 and cases[bad].time == 0.0 and cases[bad].last_dt == 0.0
        assert np.array_equal(devs[bad].to_host(["cv"])["cv"], blocks[bad][1].a["cv"])
    else:
        assert cases[bad].steps == steps
    for i, ((p, hb, faces), d, c) in enumerate(zip(blocks, devs, cases)):
        if i == bad:
            continue
        ref, t = _reference(p, hb, faces, steps, dts[i])
        assert (c.steps, c.status, c.time) == (steps, 0, t)
        assert np.array_equal(d.to_host(["cv"])["cv"], ref["cv"]), i


def test_batch_rejects_unsupported_settings(oracle_lib):
    p, hb, faces = helpers.curvilinear_air_case(12, 12, 12, scheme=abi.INV_WENO5_CH, reconstruction=abi.REC_MUSCL,
                                                viscous_order=0, bc="periodic", seed=3)
    ctx = cb200.Context(p)
    d = DeviceBlock(hb)
    cases = (abi.BlockCase * 1)()
    cases[0].zone = d.view()
    cases[0].t_end = 1.0
    with pytest.raises(cb200.CB2Error) as e:
        ctx.block_batch_advance(cases, 1)
    assert e.value.code == abi.ERR_UNSUPPORTED
