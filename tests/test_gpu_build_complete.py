"""A build returns with every table written: nothing of it is left on its stream, although another stream keeps the device
busy, and the first call on another stream gives the bits of a call on the build's own."""
import numpy as np
import pytest
import torch

import asr_b200 as A
from asr_b200 import synthetic as S
from tests import cases as K

pytestmark = pytest.mark.gpu


def _build(ctx):
    c = K.cubic("fcc", 4, 3, (0.5, 0.3, 0.2), group="d2h", maxlevel=2, maxrank=1)
    return A.build_augcls_operator(c["graph"], c["model"], c["cls"], c["perm"], c["dmat"], 1, 2, maxrank=1, flippable=c["flippable"], ctx=ctx)


def _run(op):
    ed = S.edc_params(S.draw_species(3, 1), 1)
    spec = A.ChainSpec(c=ed["c"], d=ed["d"], o=ed["o"], e=ed["e"], pa=ed["pa"], pb=ed["pb"], frozen_sp=1, start_orb=5, nlev=10)
    return A.chains_run(op, [spec], np.linspace(-0.5, 0.3, 33) + 0.05j)["g"]


def test_build_is_complete_on_return():
    ctx = A.Context(0)
    op = _build(ctx)
    ref = _run(op)
    op.free()
    s1, s2, busy = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Stream()
    x = torch.ones(1 << 30, device="cuda")   # a pass over it takes a millisecond and fills every SM
    torch.cuda.synchronize()
    for _ in range(3):
        with torch.cuda.stream(busy):
            for _ in range(400):
                x.mul_(1.0)
        ctx.set_stream(s1.cuda_stream)
        op = _build(ctx)
        assert s1.query()
        ctx.set_stream(s2.cuda_stream)
        assert np.array_equal(_run(op), ref)
        op.free()
        torch.cuda.synchronize()
    ctx.set_stream(None)
    ctx.close()
