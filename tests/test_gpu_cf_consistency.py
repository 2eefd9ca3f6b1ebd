"""Fractions of the same chain in calls of any size, and chains whose diagonal carries a common offset.  A fraction has the same
bits however many energies share the call.  An offset c moves the energies with it: what is left is the rounding of the
coefficients, 1.1e-16 c, over Im z = 0.05 and, for a Beer-Pettifor tail, a fixed point that gains at most a factor 1 - 0.95 an
iteration: 1.1e-16 / 0.05 / 0.05 c = 5e-14 c, next to the 1e-12 at which the iteration stops."""
import numpy as np
import pytest

import asr_b200 as A
from tests.test_gpu_bp_roots import chains

pytestmark = pytest.mark.gpu

MS = np.array([1, 2, 3, 9, 16, 31, 32, 33, 64, 128], np.int32)


@pytest.mark.parametrize("tail", ["hull", "bp", "avg2", "none"])
@pytest.mark.parametrize("fade", [0.3, 0.05])
def test_bits_do_not_depend_on_the_energies(tail, fade):
    a, b = chains(fade, 1.0, MS)
    z = np.linspace(-0.9, 0.8, 16)[:, None] + 0.05j + 0.01 * np.arange(MS.size)[None, :]
    g = A.cf_species(a, b, MS, z, tail)
    for n in (1, 3, 7, 8, 9):
        assert np.array_equal(A.cf_species(a, b, MS, z[:n], tail), g[:n])


@pytest.mark.parametrize("tail", ["hull", "bp"])
@pytest.mark.parametrize("c", [1e1, 1e3, 1e4])
def test_common_offset(tail, c):
    ms = MS[2:]
    a, b = chains(0.3, 1.0, ms)
    z = np.linspace(-0.9, 0.8, 9)[:, None] + 0.05j + 0.01 * np.arange(ms.size)[None, :]
    g = A.cf_species(a, b, ms, z, tail)
    gc = A.cf_species(a + c, b, ms, z + c, tail)
    assert np.max(np.abs(gc - g) / np.abs(g)) <= 1e-12 + 5e-14 * c
