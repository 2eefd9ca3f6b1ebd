"""The Lanczos update's projection by the stabiliser's signs (diagonal groups) and by the sum over its operations (the others):
the chains live in the symmetric subspace, so projecting every level changes them by rounding only.  Tolerance 1e-9 of the
largest entry: 12 levels of 1e-16 errors, at most 1e2 a level between converged directions, over an imaginary part of a tenth."""
import numpy as np
import pytest

import asr_b200 as A
from asr_b200 import synthetic as S
from tests import cases as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group,orbs", [("d2h", (1, 2, 3, 4, 5, 6, 7, 8, 9)), ("d4h", (1, 3, 5))])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-9), ("fp32", 2e-4)])
def test_projected_chains(group, orbs, precision, tol):
    c = K.cubic("bcc", 3, 2, (0.5, 0.5), group=group, maxlevel=3, maxrank=2)
    op = A.build_augcls_operator(c["graph"], c["model"], c["cls"], c["perm"], c["dmat"], 1, 3, maxrank=2, flippable=c["flippable"])
    ed = S.edc_params(S.draw_species(2, 1), 1)
    specs = [A.ChainSpec(c=ed["c"], d=ed["d"], o=ed["o"], e=ed["e"], pa=ed["pa"], pb=ed["pb"], frozen_sp=1, start_orb=l0, nlev=12)
             for l0 in orbs]
    z = np.linspace(-0.6, 0.4, 33) + 0.1j
    on = A.chains_run(op, specs, z, precision=precision, project=True)["g"]
    off = A.chains_run(op, specs, z, precision=precision, project=False)["g"]
    assert np.max(np.abs(on - off)) <= tol * np.max(np.abs(off))
