"""The rule that lets outflow faces of a block fill in one launch (csrc/outflow_apart.h), against the
nodes that the fills write and read: faces it calls apart share no ghost node that one writes and the
other writes or reads.  Blocks from one node to more than the ghost layers along every direction, whole
faces, sub-faces that touch, overlap or leave the block, with and without a back pressure."""
import ctypes as C
import itertools
import os
import random
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = """
#include "outflow_apart.h"
extern "C" int apart(const int *ext, int ngg, const int *a, const int *b) {
  auto f = [](const int *q) { return cb2::OutflowRange{q[0], q[1], {q[2], q[3], q[4]}, {q[5], q[6], q[7]}, q[8] != 0}; };
  return cb2::outflow_apart(ext, ngg, f(a), f(b));
}
"""


@pytest.fixture(scope="module")
def apart(tmp_path_factory):
    d = tmp_path_factory.mktemp("apart")
    (d / "shim.cpp").write_text(SHIM)
    cxx = shutil.which("g++") or shutil.which("c++")
    assert cxx, "no host compiler"
    subprocess.run([cxx, "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(REPO, "corefl-cpc_b200", "csrc"),
                    str(d / "shim.cpp"), "-o", str(d / "shim.so")], check=True)
    fn = C.CDLL(str(d / "shim.so")).apart

    def call(ext, ngg, a, b):
        flat = [(C.c_int * 9)(f["face"], f["dir"], *f["start"], *f["end"], int(f["back"])) for f in (a, b)]
        return bool(fn((C.c_int * 3)(*ext), ngg, *flat))

    return call


def face(ext, d, s, lo=None, hi=None, back=False):
    start, end = list(lo or (0, 0, 0)), list(hi or (e - 1 for e in ext))
    start[d] = end[d] = 0 if s < 0 else ext[d] - 1
    return {"face": d, "dir": s, "start": start, "end": end, "back": back}


def touched(f, ngg):
    """(nodes written, nodes read) of one face's fill (k_bc_outflow)."""
    write, read = set(), set()
    for n in itertools.product(*(range(a, b + 1) for a, b in zip(f["start"], f["end"]))):
        def at(m):
            return tuple(c + (m * f["dir"] if d == f["face"] else 0) for d, c in enumerate(n))
        read.add(n)
        for gl in range(1, ngg + 1):
            write.add(at(gl))
            if f["back"]:
                read.update((at(-gl), at(-1)))
    return write, read


def independent(a, b, ngg):
    (wa, ra), (wb, rb) = touched(a, ngg), touched(b, ngg)
    return not (wa & wb or wa & rb or wb & ra)


@pytest.mark.parametrize("ngg", [3, 4])
def test_faces_called_apart_do_not_touch(apart, ngg):
    rng = random.Random(ngg)
    n_apart = 0
    for _ in range(4000):
        ext = [rng.choice((1, 2, 3, 4, 5, 7)) for _ in range(3)]

        def any_face():
            d, s = rng.randrange(3), rng.choice((-1, 1))
            f = face(ext, d, s, back=rng.random() < 0.5)
            for t in range(3):
                if t != d and rng.random() < 0.6:
                    f["start"][t], f["end"][t] = sorted(rng.randint(-1 if rng.random() < 0.1 else 0, ext[t] - 1) for _ in range(2))
            if rng.random() < 0.05:
                f["start"][d] = f["end"][d] = rng.randrange(ext[d])
            return f

        a, b = any_face(), any_face()
        if apart(ext, ngg, a, b):
            n_apart += 1
            assert independent(a, b, ngg), (ext, ngg, a, b)
    assert n_apart > 1000


@pytest.mark.parametrize("ngg", [3, 4])
def test_whole_faces_of_a_block_are_apart(apart, ngg):
    """The merged launch stays for the blocks it is made for: whole faces, a back pressure on any of
    them where the block has more than ngg nodes across."""
    ext = (ngg + 1, ngg + 2, 9)
    for back in (False, True):
        faces = [face(ext, d, s, back=back) for d in range(3) for s in (-1, 1)]
        assert all(apart(ext, ngg, a, b) for a, b in itertools.combinations(faces, 2))
    thin = (ngg, 8, 8)
    left, right = face(thin, 0, -1), face(thin, 0, 1, back=True)
    assert not apart(thin, ngg, left, right)
    assert apart(thin, ngg, face(thin, 0, -1), face(thin, 0, 1))
