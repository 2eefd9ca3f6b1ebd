"""The gradient kernel at the edges of its forms: three, five and eight species' accumulators, classes that lack a species,
node counts that leave a block of 64 nearly empty, frozen and free start sites, both operator forms.  Against central
differences (Richardson-extrapolated, truncation O(h^4)) of the CUDA forward; the tolerance is that of the other adjoint
tests: the rounding of a difference of two losses of order one, 1e-16 / 1e-5, with two digits to spare, over entries of at
least 1e-2 of the largest."""
import numpy as np
import pytest

from asr_b200 import augcls as A
from asr_b200 import autograd as AG
from asr_b200 import chains as CH
from asr_b200 import synthetic as S
from tests import cases as K
from tests.test_gpu_adjoint_general import KIND, _central, _perturbed

pytestmark = pytest.mark.gpu


def _case(name):
    if name == "l21":
        return S.heusler_case(4, 2, 4, 2, 1), 2
    nsp = int(name[3:])
    conc = [(nsp - q) / (nsp * (nsp + 1) / 2) for q in range(nsp)]
    case = K.cubic("bcc", 3, nsp, tuple(conc), group="d2h", maxlevel=2, maxrank=1)
    return case, 2


@pytest.mark.parametrize("name,o,frozen", [("bcc3", 0.0, True), ("bcc5", 0.0, False), ("bcc6", 0.0, True), ("bcc5", 0.15, True),
                                           ("bcc6", 0.15, False), ("l21", 0.0, True), ("l21", 0.15, True)])
def test_gradient_of_every_species(name, o, frozen):
    case, levels = _case(name)
    op = A.build_augcls_operator(case["graph"], case["model"], case["cls"], case["perm"], case["dmat"], 1, levels, maxrank=1,
                                 flippable=case["flippable"])
    nsp = case["model"].nsp
    kap = int(case["cls"][0]) - 1
    cen = int(case["model"].spc[0, kap])
    sp = S.draw_species(nsp, 3)
    specs = []
    for orb, nlev in ((1, 9), (4, 11)):
        ed = S.edc_params(sp, cen) if o == 0.0 else S.edc_params_o(sp, S.draw_o(nsp, 3, o), cen)
        e = np.asfortranarray(0.05 * np.cos(np.arange(nsp)[None, :] + 0.3 * orb) * np.ones((9, 1)))
        specs.append(CH.ChainSpec(c=ed["c"], d=ed["d"], o=ed["o"], e=e, pa=ed["pa"], pb=ed["pb"], frozen_sp=cen if frozen else 0,
                                  start_orb=orb, nlev=nlev))
    z = np.linspace(-0.5, 0.3, 5) + 0.1j
    rng = np.random.default_rng(5)
    w = rng.standard_normal((5, 2)) + 1j * rng.standard_normal((5, 2))
    g, _, grad = CH.chains_adjoint_ext(op, specs, z, w, 0.0, "hull")

    def loss(s):
        return np.sum(w * CH.chains_run(op, s, z, "edc", 0.0, "hull", "fp64")["g"])
    orbits = AG.orbital_orbits(case["dmat"])
    for q in range(2):
        scale = np.max(np.abs(grad[q]))
        for s in range(nsp):
            for kind in ("c", "d", "pa", "e") + (("o",) if o else ()):
                orbit = orbits[int(rng.integers(len(orbits)))]
                fd = _central(lambda h: loss(_perturbed(specs, q, kind, orbit, s, h)))
                adj = np.sum(grad[q, KIND[kind], s, orbit])
                assert abs(adj - fd) <= 1e-6 * max(abs(fd), 1e-2 * scale), (q, s, kind, orbit, adj, fd)
    g32, _, grad32 = CH.chains_adjoint_ext(op, specs, z, w, 0.0, "hull", precision="fp32")
    assert np.max(np.abs(grad32 - grad)) < 1e-3 * np.max(np.abs(grad))
