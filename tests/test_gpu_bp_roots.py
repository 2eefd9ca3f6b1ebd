"""Beer-Pettifor tails whose spectra are followed by simultaneous root finding, against the oracle's fractions: depths around the
warp's 32 roots a pass and up to the device maximum, coefficients of very different size, chains that settle fast, slowly and
not at all (hull fallback), and a chain that falls apart.  Tolerance 1e-9 relative: the iteration stops at 1e-12, errors left
by a contraction of up to 0.95 are 2e-11, and a fraction at Im z = 0.05 bandwidths magnifies them by up to 1 / 0.05."""
import numpy as np
import pytest

import asr_b200 as A
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def chains(fade, scale, ms):
    rng = np.random.default_rng(11)
    ld, nc = int(ms.max()), ms.size
    f = np.exp(-fade * np.arange(ld))[:, None]
    a = -0.1 - 0.05j + f * (rng.uniform(-0.3, 0.3, (ld, nc)) + 1j * rng.uniform(-0.05, 0.0, (ld, nc)))
    b = 0.3 + 0.02j + f * rng.uniform(-0.1, 0.1, (ld, nc))
    return scale * a, scale * b


@pytest.mark.parametrize("fade", [0.3, 0.05, 0.0])
@pytest.mark.parametrize("scale", [1.0, 3.7e5, 2.9e-6])
def test_tails_of_every_depth(fade, scale):
    ms = np.array([2, 3, 5, 17, 31, 32, 33, 48, 64, 65, 128], np.int32)
    a, b = chains(fade, scale, ms)
    nz = 9
    z = scale * (np.linspace(-0.9, 0.8, nz)[:, None] + 0.05j + 0.01 * np.arange(ms.size)[None, :])
    g = A.cf_species(a, b, ms, z, "bp")
    for c in range(ms.size):
        for j in range(0, nz, 4):
            go = O.cf_species(a[:, c], b[:, c], int(ms[c]), z[j, c], "bp")[0]
            assert abs(g[j, c] - go) <= 1e-9 * abs(go), (ms[c], j)


def test_decoupled_chain():
    ms = np.array([9], np.int32)
    a, b = chains(0.3, 1.0, ms)
    b[3] = 0.0
    z = np.linspace(-0.9, 0.8, 9)[:, None] + 0.05j
    g = A.cf_species(a, b, ms, z, "bp")
    for j in range(9):
        go = O.cf_species(a[:, 0], b[:, 0], 9, z[j, 0], "bp")[0]
        assert abs(g[j, 0] - go) <= 1e-9 * abs(go)
