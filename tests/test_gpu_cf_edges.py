"""The fraction kernels at the edges of their forms against the oracle: one thread per (energy, chain) below 8 energies and
one block per chain from there on, chains from one level to the device maximum, and the warp's sectioned Beer-Pettifor
asymptote of real chains.  Tolerances: 1e-10 relative for complex fractions (as on the golden chains), 1e-9 for real ones."""
import numpy as np
import pytest

import asr_b200 as A
from asr_b200 import synthetic as S
from oracle import oracle as O
from tests import cases as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tail", ["hull", "avg2", "bp", "none"])
@pytest.mark.parametrize("nz", [1, 7, 8, 130])
def test_fractions_of_every_depth(tail, nz):
    rng = np.random.default_rng(5)
    ms = np.array([1, 2, 3, 9, 31, 32, 33, 128], np.int32) if tail != "bp" else np.array([1, 2, 3, 9, 24], np.int32)
    ld, nc = int(ms.max()), ms.size
    # coefficients that settle, as a recursion's do
    fade = np.exp(-0.3 * np.arange(ld))[:, None]
    a = -0.1 - 0.05j + fade * (rng.uniform(-0.3, 0.3, (ld, nc)) + 1j * rng.uniform(-0.05, 0.0, (ld, nc)))
    b = 0.3 + 0.02j + fade * rng.uniform(-0.1, 0.1, (ld, nc))
    z = np.linspace(-0.9, 0.8, nz)[:, None] + 0.05j + 0.01 * np.arange(nc)[None, :]
    g = A.cf_species(a, b, ms, z, tail)
    for c in range(nc):
        for j in range(0, nz, max(1, nz // 5)):
            go = O.cf_species(a[:, c], b[:, c], int(ms[c]), z[j, c], tail)[0]
            assert abs(g[j, c] - go) <= 1e-10 * abs(go), (ms[c], j)


@pytest.mark.parametrize("depth", [2, 3, 9, 16])
def test_real_beer_pettifor(depth):
    gop, oop = K.build_both(K.cubic("bcc", 3, 2, (0.5, 0.5), group="d2h", maxlevel=2, maxrank=1), A.build_augcls_operator, O.OracleOp)
    c, d, o, e = S.plain_params(S.draw_species(2, 3))
    specs = [A.ChainSpec(c=c, d=d, o=o, e=e, start_orb=l0, nlev=depth) for l0 in (1, 4, 9)]
    z = np.linspace(-1.2, 0.8, 33) + 0.02j
    g = A.chains_run(gop, specs, z, mode="plain", tail="bp")["g"]
    oop.set_params(c, d, o, e)
    for q, l0 in enumerate((1, 4, 9)):
        oop.set_start(l0)
        v0 = np.zeros(oop.dim)
        v0[l0 - 1] = 1.0
        ao, bo, no = oop.lanczos(v0, depth)
        go, _ = O.terminated_green(ao, bo, no, z, "beer-pettifor")
        assert np.max(np.abs(g[:, q] - go)) <= 1e-9 * np.max(np.abs(go))
