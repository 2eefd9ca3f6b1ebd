"""The projector by counted signs, which the Lanczos update and project_c share, against the oracle's sum over the stabiliser on
vectors that are not symmetric: diagonal groups (orbitals kept or cleared), one of 40 operations (every operation of D2h
five times: two ballots), a group that permutes orbitals (the sum), and signs that belong to no representation (neither kept
nor cleared: the sum).  Tolerance 1e-14 of the largest entry: a mean of at most 64 values."""
import numpy as np
import pytest

import asr_b200 as A
from oracle import oracle as O
from tests import cases as K

pytestmark = pytest.mark.gpu


def _case(name):
    c = K.cubic("bcc", 3, 2, (0.5, 0.5), group="d4h" if name == "d4h" else "d2h", maxlevel=2, maxrank=1)
    if name == "d2h_five_times":
        c["perm"] = np.asfortranarray(np.concatenate([c["perm"]] * 5, axis=1))
        c["dmat"] = np.asfortranarray(np.concatenate([c["dmat"]] * 5, axis=2))
    return c


@pytest.mark.parametrize("name,orbs", [("d2h", range(1, 10)), ("d2h_five_times", (1, 2, 6)), ("d4h", (1, 3, 5))])
def test_projection_of_any_vector(name, orbs):
    gop, oop = K.build_both(_case(name), A.build_augcls_operator, O.OracleOp)
    rng = np.random.default_rng(2)
    x = rng.standard_normal(gop.dim) + 1j * rng.standard_normal(gop.dim)

    def same():
        pg, po = gop.project_c(x), oop.project_c(x)
        assert np.max(np.abs(pg - po)) <= 1e-14 * np.max(np.abs(x))
        return po
    for l0 in orbs:
        for op in (gop, oop):
            op.set_start(l0)
        assert np.max(np.abs(same() - x)) > 0.1   # it does something
    for _ in range(3):
        chi = np.where(rng.random(gop.nop) < 0.5, -1.0, 1.0)
        chi[0] = 1.0
        for op in (gop, oop):
            op.set_chi(chi)
        same()
