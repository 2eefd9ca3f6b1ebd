"""A uniform d with orbitals of zero or hardly any d: the step kernels, which fold d into the bond blocks and divide it out
again for the adjoint, against the route that never does (d of one species off by 1e-14, so that it counts as species
dependent).  Tolerances: chains of depth 9 at Im z = 0.1 carry the 1e-14 and the reordered sums to 1e-11 of the largest entry
at most; a single orbital's d gradient, where it is not zero, to 1e-6 of its own."""
import numpy as np
import pytest

import asr_b200 as A
from asr_b200 import chains as CH
from asr_b200 import synthetic as S
from tests import cases as K

pytestmark = pytest.mark.gpu

ZERO, TINY, SMALL = 6, 7, 8   # orbitals of d = 0, far below and just above what is divided out


def _specs(d_small, o, split):
    sp = S.draw_species(2, 3)
    specs = []
    for orb, nlev in ((1, 9), (7, 8), (4, 9)):
        ed = S.edc_params(sp, 1) if o == 0.0 else S.edc_params_o(sp, S.draw_o(2, 3, o), 1)
        d = ed["d"].copy(order="F")
        d[ZERO], d[TINY], d[SMALL] = 0.0, d_small, 3e-8
        if split:
            d[0, 1] *= 1.0 + 1e-14
        specs.append(CH.ChainSpec(c=ed["c"], d=d, o=ed["o"], e=ed["e"], pa=ed["pa"], pb=ed["pb"], frozen_sp=1, start_orb=orb, nlev=nlev))
    return specs


@pytest.mark.parametrize("o", [0.0, 0.15])
@pytest.mark.parametrize("d_small", [1e-9, 1e-200])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("fp32", 1e-3)])
@pytest.mark.parametrize("stride", [0, 3])
def test_small_d(o, d_small, precision, tol, stride):
    c = K.cubic("bcc", 3, 2, (0.5, 0.5), group="d2h", maxlevel=2, maxrank=1)
    op = A.build_augcls_operator(c["graph"], c["model"], c["cls"], c["perm"], c["dmat"], 1, 2, maxrank=1, flippable=c["flippable"])
    z = np.linspace(-0.5, 0.3, 20) + 0.1j
    rng = np.random.default_rng(5)
    w = rng.standard_normal((20, 3)) + 1j * rng.standard_normal((20, 3))
    res = []
    for split in (False, True):
        specs = _specs(d_small, o, split)
        run = A.chains_run(op, specs, z, precision=precision)["g"]
        g, m, grad = CH.chains_adjoint_ext(op, specs, z, w, 0.0, "hull", precision, stride=stride)
        res.append((run, g, grad))
    for x, y in zip(res[0], res[1]):
        assert np.all(np.isfinite(x))
        assert np.max(np.abs(x - y)) <= tol * np.max(np.abs(y))
    if precision == "fp64":
        for l in (TINY, SMALL):
            x, y = res[0][2][:, 1, :, l], res[1][2][:, 1, :, l]
            assert np.max(np.abs(x - y)) <= 1e-6 * np.max(np.abs(y))
