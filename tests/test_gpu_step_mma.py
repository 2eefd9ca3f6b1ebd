"""The FP64 tensor-core step at the edges of its tiles: the octets of lanes a tile computes (one to four, with idle lanes in
the last), operators with fewer nodes than a thread block, signed and permuting links, and more than 32 neighbour slots, against
the oracle.  Tolerance: 1e-9 relative, the reference's own for recursion coefficients (an edc chain of depth 10 amplifies
the 1e-16 of a reordered product sum by far less)."""
import numpy as np
import pytest

import asr_b200 as A
from asr_b200 import synthetic as S
from oracle import oracle as O
from tests import cases as K

pytestmark = pytest.mark.gpu

CASES = {
    "signs": lambda: K.cubic("bcc", 3, 2, (0.5, 0.5), group="d2h", maxlevel=2, maxrank=1),
    "permutations": lambda: K.cubic("fcc", 3, 3, (0.5, 0.3, 0.2), group="d4h", maxlevel=1, maxrank=1),
}


@pytest.fixture(scope="module", params=sorted(CASES))
def pair(request):
    gop, oop = K.build_both(CASES[request.param](), A.build_augcls_operator, O.OracleOp)
    ed = S.edc_params(S.draw_species(gop.nsp, 2), 1)
    for op in (gop, oop):
        op.set_params(ed["c"], ed["d"], ed["o"], ed["e"])
        op.freeze_site(1, 1)
        op.set_start(5)
    return gop, oop, ed


@pytest.mark.parametrize("nz", [1, 7, 8, 9, 16, 17, 24, 25, 32, 33, 41])
def test_octets_match_the_oracle_and_each_other(pair, nz):
    gop, oop, ed = pair
    zs = np.linspace(-0.6, 0.4, 41) + 0.05j
    g, m, a, b = A.edc_green_blk(gop, ed, zs[:nz], 5, 10)
    go, mo, ao, bo = oop.edc_green_blk(ed, zs[:nz], 5, 10)
    assert np.array_equal(m, mo)
    for x, y in ((g, go), (a, ao), (b, bo)):
        assert np.max(np.abs(x - y)) <= 1e-9 * np.max(np.abs(y))
    full = A.edc_green_blk(gop, ed, zs, 5, 10)
    assert np.array_equal(g, full[0][:nz]) and np.array_equal(a, full[2][:, :nz])   # a lane's bits in any tile


def test_more_neighbour_slots_than_lanes():
    c = S.cubic_case("fcc", 4, 2, [0.5, 0.5], seed=1, group="d2h", r2max=8)   # 54 slots
    fl = np.ones(c["graph"].n, np.int32)
    fl[0] = 0
    c.update(maxlevel=1, maxrank=1, flippable=fl)
    gop, oop = K.build_both(c, A.build_augcls_operator, O.OracleOp)
    assert gop.nslot > 32
    par = K.general_params(2)
    x = np.random.default_rng(1).uniform(-0.5, 0.5, (gop.dim, 2))
    for op in (gop, oop):
        op.set_params(*par)
    y = gop.apply(x)
    for j in range(2):
        yo = oop.apply(x[:, j])
        assert np.max(np.abs(y[:, j] - yo)) <= 1e-12 * np.max(np.abs(yo))


@pytest.mark.parametrize("nz", [5, 16, 20, 33])
def test_general_operator_octets(pair, nz):
    """H = E + h - h o h + X(z) at uniform d (two tensor-core passes with the random operator between them)."""
    gop, oop, _ = pair
    sp = S.draw_species(gop.nsp, 4)
    ed = S.edc_params_o(sp, S.draw_o(gop.nsp, 4, 0.2), 1)
    zs = np.linspace(-0.5, 0.3, nz) + 0.05j
    for op in (gop, oop):
        op.set_params(ed["c"], ed["d"], ed["o"], ed["e"])
    try:
        g, m, a, b = A.edc_green_blk(gop, ed, zs, 5, 10)
        go, mo, ao, bo = oop.edc_green_blk(ed, zs, 5, 10)
        assert np.array_equal(m, mo)
        for x, y in ((g, go), (a, ao), (b, bo)):
            assert np.max(np.abs(x - y)) <= 1e-9 * np.max(np.abs(y))
    finally:
        for op in (gop, oop):
            op.set_params(*[pair[2][k] for k in ("c", "d", "o", "e")])
