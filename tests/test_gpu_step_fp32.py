"""The FP32 step's two row gathers (operations that move no orbital, and those that do) and its flip links (up to two looked up
once, more again for each orbital) against the FP64 step on the same chains.  Tolerance 2e-4 of the largest: 8 levels of
products rounded to 6e-8, sums of 19 x 9 terms, over an imaginary part of a tenth of the band."""
import numpy as np
import pytest

import asr_b200 as A
from asr_b200 import synthetic as S
from tests import cases as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice,nsp,group", [("bcc", 2, "d2h"), ("bcc", 2, "d4h"), ("fcc", 3, "d2h"), ("bcc", 3, "d4h"),
                                               ("bcc", 5, "d2h")])
def test_fp32_step(lattice, nsp, group):
    conc = tuple((nsp - q) / (nsp * (nsp + 1) / 2) for q in range(nsp))
    c = K.cubic(lattice, 3, nsp, conc, group=group, maxlevel=2, maxrank=1)
    op = A.build_augcls_operator(c["graph"], c["model"], c["cls"], c["perm"], c["dmat"], 1, 2, maxrank=1, flippable=c["flippable"])
    ed = S.edc_params(S.draw_species(nsp, 1), 1)
    specs = [A.ChainSpec(c=ed["c"], d=ed["d"], o=ed["o"], e=ed["e"], pa=ed["pa"], pb=ed["pb"], frozen_sp=f, start_orb=l0, nlev=8)
             for l0, f in ((1, 1), (3, 0), (5, 1))]
    z = np.linspace(-0.6, 0.4, 40) + 0.1j
    g64 = A.chains_run(op, specs, z, precision="fp64")["g"]
    g32 = A.chains_run(op, specs, z, precision="fp32")["g"]
    assert np.max(np.abs(g32 - g64)) <= 2e-4 * np.max(np.abs(g64))
