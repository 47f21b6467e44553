"""Poseidon2.same_as: two handles are one permutation when field, exponent,
rounds and every constant agree, whichever way the handles were made (host
constants only: runs without a GPU)."""

from __future__ import annotations

import numpy as np
import pytest

from zorch_gb300.commit import Poseidon2, koalabear16_params
from zorch_gb300.field import BABYBEAR, KOALABEAR


def _parts(orc):
    return list(orc.Poseidon2.babybear16().export_canonical())


def test_equal_constants_are_one_permutation(orc):
    a = Poseidon2.from_params(BABYBEAR, 7, *_parts(orc))
    assert a.same_as(a) and a.same_as(Poseidon2.from_params(BABYBEAR, 7, *_parts(orc)))
    assert a.same_as(Poseidon2.builtin()) and Poseidon2.builtin().same_as(a)
    kb = orc.load_koalabear_fixture()
    assert koalabear16_params(kb).same_as(koalabear16_params(kb))


@pytest.mark.parametrize("which", ["ext_init", "ext_term", "int_rc", "diag", "alpha", "rounds_f",
                                   "rounds_p", "j", "field", "instance"])
def test_any_difference_is_another_permutation(orc, which):
    a = Poseidon2.from_params(BABYBEAR, 7, *_parts(orc))
    ei, et, ir, dg = (x.astype(np.uint32).copy() for x in _parts(orc))
    field, alpha, j = BABYBEAR, 7, 1
    if which in ("ext_init", "ext_term", "int_rc", "diag"):
        x = {"ext_init": ei, "ext_term": et, "int_rc": ir, "diag": dg}[which].reshape(-1)
        x[-1] = (int(x[-1]) + 1) % BABYBEAR.p
    elif which == "alpha":
        alpha = 5
    elif which == "rounds_f":
        ei, et = ei[:-1], et[:-1]
    elif which == "rounds_p":
        ir = ir[:-1]
    elif which == "j":
        j = 2
    elif which == "field":
        field = KOALABEAR
    b = (koalabear16_params(orc.load_sp1_fixture()) if which == "instance"
         else Poseidon2.from_params(field, alpha, ei, et, ir, dg, j))
    assert not a.same_as(b) and not b.same_as(a)
    if which == "instance":
        assert not b.same_as(koalabear16_params(orc.load_koalabear_fixture()))
