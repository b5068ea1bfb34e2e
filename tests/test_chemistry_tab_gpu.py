"""The block chemistry kernel on a repacked mechanism against the oracle: sizes around the edges of
its tiles of 128 nodes of a k plane, temperatures in both ranges of the NASA7 fits, at their middle
and beyond their ends, absent species, five species, a species with a middle temperature of its own,
third bodies that are absent, the longest mechanism and the longest side of a reaction that fit a table,
and the mechanisms that do not (more than 24 reactions, more than eight reactants), which run the
generic kernel."""
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


def mechanism(kind):
    h2 = mechmod.load_json(GOLD)
    d = copy.deepcopy(h2.d)
    ns, nr = h2.ns, h2.nr
    if kind in ("long", "full"):  # the first reactions again: 27, 24
        more = 8 if kind == "long" else 5
        for name in abi.MECH_INT + abi.MECH_REAC:
            a = np.asarray(d[name]).reshape(nr, -1)
            d[name] = np.concatenate([a, a[:more]]).reshape(-1).tolist()
        d["n_reac"] = nr + more
    elif kind in ("steep", "eight"):  # H + O2 -> O + OH with ten H on the left; with seven
        a = np.asarray(d["stoi_f"]).reshape(nr, ns)
        a[0, list(h2.species).index("H")] = 10 if kind == "steep" else 7
        d["stoi_f"] = a.reshape(-1).tolist()
    elif kind == "five":
        return helpers.sub_mechanism(h2, ("H", "O2", "O", "OH", "HO2"))
    elif kind == "five_h2":
        return helpers.sub_mechanism(h2, ("O", "H2", "OH", "O2", "H"))
    elif kind == "middles":  # a middle temperature of its own
        d["t_mid"][3] = 1100.0
    elif kind == "no_body":  # the only third body of every such reaction is a species that is not there
        a = np.zeros((nr, ns))
        a[:, 1] = 1.0
        d["third_body_coeff"] = a.reshape(-1).tolist()
        d["reac_type"] = [5 if t > 5 else t for t in d["reac_type"]]  # Troe's form has no value there
    elif kind == "irreversible":  # no backward rate for some
        d["reac_type"][1] = d["reac_type"][16] = 0
    elif kind == "explicit":  # every backward rate from its own Arrhenius constants
        d["rev_type"] = [1] * nr
    return mechmod.MechStruct(d)


def block(mech, dims, seed):
    rng = np.random.default_rng(seed)
    g = 3
    specs = array_specs(*dims, g, 5 + mech.ns, mech.ns, reaction=True)
    b = HostBlock(*dims, g, specs)
    shape = b.a["bv"][0].shape
    y = rng.uniform(0, 1, (mech.ns,) + shape) ** 4
    y[1][rng.uniform(0, 1, shape) < 0.2] = 0.0  # a species that is not there
    y /= y.sum(axis=0)
    t = rng.choice([180.0, 250.0, 300.0, 999.0, 1000.0, 1001.0, 1500.0, 3400.0, 3600.0, 5200.0], shape)
    b.a["sv"][...] = y
    b.a["bv"][0] = rng.uniform(0.05, 2.0, shape)
    b.a["bv"][5] = t
    b.a["jac"][0] = rng.uniform(0.5, 2.0, shape)
    b.a["dq"][...] = 0
    p = cases.make_param(n_var=5 + mech.ns, n_spec=mech.ns, inviscid_scheme=abi.INV_HLLC, reconstruction=abi.REC_WENO5,
                         rho_ref=1.0, v_ref=700.0, mech=mech.ptr())
    p.reaction = 1
    return p, b


@pytest.mark.parametrize("dims,kind", [((1, 1, 1), "h2"), ((127, 1, 1), "h2"), ((43, 3, 2), "h2"), ((64, 2, 3), "h2"),
                                       ((17, 23, 5), "h2"), ((17, 5, 2), "irreversible"), ((17, 5, 2), "explicit"),
                                       ((17, 5, 2), "long"),
                                       ((17, 5, 2), "steep"), ((17, 5, 2), "full"), ((17, 5, 2), "eight"),
                                       ((17, 5, 2), "five"), ((43, 3, 2), "five_h2"), ((17, 5, 2), "middles"),
                                       ((17, 5, 2), "no_body")])
def test_chemistry_against_oracle(dims, kind):
    import torch
    import cb200
    from cb200.field import DeviceBlock
    mech = mechanism(kind)
    p, hb = block(mech, dims, seed=sum(dims))
    dev = DeviceBlock(hb)
    ctx = cb200.Context(p)
    ctx.bind(0, dev.view(), [])
    ctx.rhs(0, abi.RHS_CHEMISTRY)
    torch.cuda.synchronize()
    got = dev.to_host(["dq", "reaction_timeScale"])
    ctx.close()
    oracle_py.rhs(p, hb, [], abi.RHS_CHEMISTRY)
    ref = hb.a["dq"]
    # rates are exponentials of arguments up to about 150: 150 ulp of the rate of each reaction,
    # measured against the largest source of the node
    scale = np.abs(ref[5:]).max(axis=0)
    assert np.isfinite(got["dq"]).all() and np.isfinite(ref).all()
    assert (np.abs(got["dq"][5:] - ref[5:]) <= 5e-13 * scale + 1e-300).all()
    a, b = (x[0][hb.ngg:hb.ngg + dims[2], hb.ngg:hb.ngg + dims[1], hb.ngg:hb.ngg + dims[0]]
            for x in (got["reaction_timeScale"], hb.a["reaction_timeScale"]))
    assert (np.abs(a - b) <= 1e-11 * np.abs(b)).all()
