"""The scaled Chebyshev steps at the edges of their tiles against the oracle: one to five octets of vector pairs (the last
block of vectors partly filled), fewer sites than a thread block, both moment schemes.  Tolerances: FP64 1e-11 relative (200
steps' worth of rounding of a stable recurrence, against moments of order 1), FP32 2e-5 (its storage rounding)."""
import numpy as np
import pytest

from asr_b200 import kpm
from asr_b200 import synthetic as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("fp32", 2e-5)])
@pytest.mark.parametrize("nvec", [1, 16, 17, 33, 64, 67])
def test_moments_of_any_number_of_vectors(nvec, precision, tol):
    nbr, spc, bvec, _ = kpm.fcc_supercell(3, [0.6, 0.3, 0.1], None, 2)
    block, block0 = S.sk_blocks(bvec, 2)
    c, d, o, e = S.plain_params(S.draw_species(3, 2))
    e = e + 0.05
    sc = kpm.Supercell(nbr, spc, c, d, o, e, block, block0)
    for doubling in (False, True):
        mu = sc.kpm_moments(0.1, 9.0, 13, nvec, seed=3, v0=5, precision=precision, doubling=doubling)
        mo = O.kpm_moments(nbr, spc, c, d, o, e, block, block0, 0.1, 9.0, 13, 5, nvec, 3)
        assert np.max(np.abs(mu - mo)) <= tol
