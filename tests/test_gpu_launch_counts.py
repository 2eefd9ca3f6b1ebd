"""The context's launch counter against the kernels of each form of a chain step and of a reverse level, for one tile: two
kernels to start a batch, the step and the Lanczos update per level (a reduction where the step is several kernels), the
depth test, the fractions, the depths; the adjoint's start, fraction adjoint and gradient sum."""
import numpy as np
import pytest

import asr_b200 as A
from asr_b200 import chains as CH
from asr_b200 import synthetic as S
from tests import cases as K

pytestmark = pytest.mark.gpu

N = 9   # levels


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("o", [0.0, 0.15])
@pytest.mark.parametrize("uniform", [True, False])
def test_counter(precision, o, uniform):
    c = K.cubic("bcc", 3, 2, (0.5, 0.5), group="d2h", maxlevel=2, maxrank=1)
    ctx = A.Context(0)
    op = A.build_augcls_operator(c["graph"], c["model"], c["cls"], c["perm"], c["dmat"], 1, 2, maxrank=1, flippable=c["flippable"],
                                 ctx=ctx)
    sp = S.draw_species(2, 1)
    ed = S.edc_params(sp, 1) if o == 0.0 else S.edc_params_o(sp, S.draw_o(2, 1, o), 1)
    d = ed["d"].copy(order="F")
    if not uniform:
        d[0, 1] *= 1.1
    specs = [A.ChainSpec(c=ed["c"], d=d, o=ed["o"], e=ed["e"], pa=ed["pa"], pb=ed["pb"], frozen_sp=1, start_orb=1, nlev=N)]
    z = np.linspace(-0.5, 0.3, 20) + 0.1j
    fp64 = precision == "fp64"
    step = (1 if not o else 3 if fp64 else 6) if uniform else (7 if o else 3)
    level = step + 1 + (0 if uniform and (fp64 or not o) else 1)

    def counted(f):
        n = ctx.launches()
        f()
        return ctx.launches() - n
    assert counted(lambda: A.chains_run(op, specs, z, precision=precision)) == 2 + N * level + 2
    assert counted(lambda: A.chains_run(op, specs, z, depth_tol=1e-300, precision=precision)) == 2 + N * level + 1 + 2
    if not o:
        for tail, k in (("bp", 2), ("hull", 1)):
            assert counted(lambda: A.chains_run(op, specs, z, mode="plain", tail=tail, precision=precision)) == 2 + N * level + 1 + k
    fused = uniform and not o
    apply = (3 if uniform and fp64 else 5 if uniform else 7) if o else (1 if uniform else 3)
    level = (2 + 4) if fused else (apply + 2) + (apply + 7)
    w = np.ones((20, 1), complex)
    assert counted(lambda: CH.chains_adjoint_ext(op, specs, z, w, 0.0, "hull", precision)) == 3 + N * level
    assert counted(lambda: CH.chains_adjoint_ext(op, specs, z, w, 0.0, "hull", precision, stride=3)) == 3 + N * (level + apply + 2)
    op.free()
    ctx.close()
