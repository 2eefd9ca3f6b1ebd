"""The link choice, which selects no kernel, is not timed by the autotuner, and is kept where it is set."""
import numpy as np
import pytest

import asr_b200 as A
from asr_b200 import synthetic as S
from tests import cases as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_link_choice_is_not_timed(precision):
    c = K.cubic("bcc", 3, 2, (0.5, 0.5), group="d2h", maxlevel=2, maxrank=1)
    op = A.build_augcls_operator(c["graph"], c["model"], c["cls"], c["perm"], c["dmat"], 1, 2, maxrank=1, flippable=c["flippable"])
    ed = S.edc_params(S.draw_species(2, 1), 1)
    spec = A.ChainSpec(c=ed["c"], d=ed["d"], o=ed["o"], e=ed["e"], pa=ed["pa"], pb=ed["pb"], frozen_sp=1, start_orb=1, nlev=8)
    A.set_tuning(op, precision, 16, 4, "fixed-offset")
    assert A.tuning(op, precision)["link_gather"] == "fixed-offset"
    tune = A.autotune(op, [spec], np.linspace(-0.5, 0.3, 40) + 0.1j, precision, levels=4)
    assert tune["link_gather"] == "general" and tune["ms_link"] == [-1.0, -1.0]
    assert A.tuning(op, precision)["link_gather"] == "general"
