"""Bonds that went through a pickle of another process (spawned workers, torch.save) are the bonds they were."""
import copy
import os
import pickle
import subprocess
import sys

import pytest

import cytnx_b200 as c
from cytnx_b200.unitensor import layout_for

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MAKE = """
import pickle, sys
import cytnx_b200 as c
from cytnx_b200.unitensor import layout_for
b = c.Bond(c.BD_KET, [[0], [1], [2]], [2, 3, 1])
layout_for([b, b.redirect()])  # takes the bond's keys
b._sectors()
sys.stdout.buffer.write(pickle.dumps((b, b.redirect())))
"""


def fresh():
    return c.Bond(c.BD_KET, [[0], [1], [2]], [2, 3, 1])


@pytest.fixture(scope="module")
def travelled():
    out = subprocess.run([sys.executable, "-c", MAKE], cwd=ROOT, env={**os.environ, "PYTHONHASHSEED": "12345"},
                         capture_output=True, check=True).stdout
    return pickle.loads(out)


def test_keys_equal_those_of_a_fresh_bond(travelled):
    b, r = travelled
    f = fresh()
    for x, y in ((b, f), (r, f.redirect())):
        assert x == y and x._id() == y._id() and x._sectors() == y._sectors()
        assert hash(x._id()) == hash(y._id()) and hash(x._sectors()) == hash(y._sectors())
    assert layout_for([b, r]) is layout_for([f, f.redirect()])
    assert not b._degs.flags.writeable and not b._qnums.flags.writeable


def test_contract_accepts_it(travelled):
    b, _ = travelled
    f = fresh()
    A = c.UniTensor([f.redirect(), b], labels=["a", "b"], rowrank=1, device=c.Device.cpu)
    B = c.UniTensor([f.redirect(), f], labels=["b", "d"], rowrank=1, device=c.Device.cpu)
    with pytest.raises(c.CytnxError, match="CUDA devices only"):  # past the bond checks, and no further on a CPU tensor
        c.Contract(A, B)


def test_copies_and_a_state_without_keys():
    f = fresh()
    f._id()
    assert copy.deepcopy(f) == f and copy.copy(f)._id() == f._id()
    old = {k: v for k, v in f.__dict__.items() if k not in ("_idc", "_secc")}  # as written before bonds kept keys
    b = c.Bond.__new__(c.Bond)
    b.__setstate__(dict(old))
    assert b._id() == f._id()
