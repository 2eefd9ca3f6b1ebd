"""Operators of many site classes, whose diagonal weights do not fit into shared memory beside the bond blocks: classes that are
all alike give the bits of the operator with one class, in the chains, the general operator and the adjoints, and the
oracle's coefficients (1e-9 relative, the reference's own for them).  Row counts (class, state) + species on both sides of
the limit; 127 classes of 7 species are the most that the node tables hold with 889 rows."""
import numpy as np
import pytest

import asr_b200 as A
from asr_b200 import chains as CH
from asr_b200 import synthetic as S
from oracle import oracle as O
from tests import cases as K

pytestmark = pytest.mark.gpu


def _case(ncls, nsp):
    conc = np.array([(nsp - q) / (nsp * (nsp + 1) / 2) for q in range(nsp)])
    c = K.cubic("fcc", 4, nsp, tuple(conc), group="identity", maxlevel=1, maxrank=1)
    m = c["model"]
    rep = lambda x: np.asfortranarray(np.repeat(x, ncls, axis=-1))
    c["model"] = S.ClassModel(nsp=m.nsp, nsc=rep(m.nsc), spc=rep(m.spc), conc=rep(m.conc), block=m.block, block0=m.block0)
    c["cls"] = (1 + np.arange(c["graph"].n, dtype=np.int32) % ncls).astype(np.int32)
    c["stype"] = np.ones(c["graph"].n, np.int32)
    return c


def _build(c):
    return A.build_augcls_operator(c["graph"], c["model"], c["cls"], c["perm"], c["dmat"], 1, 1, maxrank=1, flippable=c["flippable"], stype=c["stype"])


@pytest.mark.parametrize("ncls,nsp", [(60, 3), (100, 4), (101, 4), (127, 7)])
def test_many_like_classes(ncls, nsp):
    one, many = _build(_case(1, nsp)), _build(_case(ncls, nsp))
    assert one.nn == many.nn
    z = np.linspace(-0.5, 0.3, 20) + 0.1j
    sp = S.draw_species(nsp, 3)
    rng = np.random.default_rng(5)
    w = rng.standard_normal((20, 2)) + 1j * rng.standard_normal((20, 2))
    for o in (0.0, 0.15):
        specs = []
        for frozen in (0, 1):
            ed = S.edc_params(sp, 1) if o == 0.0 else S.edc_params_o(sp, S.draw_o(nsp, 3, o), 1)
            specs.append(CH.ChainSpec(c=ed["c"], d=ed["d"], o=ed["o"], e=ed["e"], pa=ed["pa"], pb=ed["pb"], frozen_sp=frozen,
                                      start_orb=5, nlev=8))
        g1, gm = (A.chains_run(op, specs, z)["g"] for op in (one, many))
        assert np.array_equal(g1, gm)
        r1, rm = (CH.chains_adjoint_ext(op, specs, z, w, 0.0, "hull") for op in (one, many))
        assert np.array_equal(r1[0], rm[0]) and np.array_equal(r1[2], rm[2])


def test_many_classes_match_the_oracle():
    c = _case(127, 7)
    gop = _build(c)
    oop = O.OracleOp(c["graph"], c["model"], c["cls"], c["perm"], c["dmat"], 1, 1, 1, c["flippable"], c["stype"])
    ed = S.edc_params(S.draw_species(7, 2), 1)
    zs = np.linspace(-0.6, 0.4, 9) + 0.05j
    for op in (gop, oop):
        op.set_params(ed["c"], ed["d"], ed["o"], ed["e"])
        op.freeze_site(1, 1)
        op.set_start(5)
    g, m, a, b = A.edc_green_blk(gop, ed, zs, 5, 10)
    go, mo, ao, bo = oop.edc_green_blk(ed, zs, 5, 10)
    assert np.array_equal(m, mo)
    for x, y in ((g, go), (a, ao), (b, bo)):
        assert np.max(np.abs(x - y)) <= 1e-9 * np.max(np.abs(y))
