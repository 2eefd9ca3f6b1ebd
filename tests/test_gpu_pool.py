"""The context's pool of call temporaries: calls of different sizes in turn, from two contexts in two threads and on a caller's
stream, give the results of the first call bit for bit; what the pool keeps is bounded and goes back with the context."""
import threading

import numpy as np
import pytest
import torch

import asr_b200 as A
from asr_b200 import synthetic as S
from tests import cases as K

pytestmark = pytest.mark.gpu


def _op(ctx):
    c = K.cubic("bcc", 3, 2, (0.5, 0.5), group="d2h", maxlevel=2, maxrank=1)
    op = A.build_augcls_operator(c["graph"], c["model"], c["cls"], c["perm"], c["dmat"], 1, 2, maxrank=1, flippable=c["flippable"], ctx=ctx)
    ed = S.edc_params(S.draw_species(2, 1), 1)
    specs = [A.ChainSpec(c=ed["c"], d=ed["d"], o=ed["o"], e=ed["e"], pa=ed["pa"], pb=ed["pb"], frozen_sp=1, start_orb=l0, nlev=12)
             for l0 in range(1, 10)]
    return op, specs


def test_pool_reuse_threads_streams():
    z = np.linspace(-0.6, 0.4, 70) + 0.02j
    got = [None, None]

    def work(k):
        ctx = A.Context(0)
        op, specs = _op(ctx)
        first = A.chains_run(op, specs, z)["g"]
        ok = True
        stream = torch.cuda.Stream()
        for q, n in enumerate((70, 3, 33, 70, 1, 70)):
            ctx.set_stream(stream.cuda_stream if q % 2 else None)
            g = A.chains_run(op, specs, z[:n])["g"]
            ok = ok and np.array_equal(g, first[:n])
            gr = A.chains_adjoint(op, specs[:2], z[:n], np.ones((n, 2), complex))[0]
            ok = ok and np.array_equal(gr, first[:n, :2])
        ctx.set_stream(None)
        op.free()
        ctx.close()
        got[k] = (ok, first)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert got[0][0] and got[1][0] and np.array_equal(got[0][1], got[1][1])


def test_pool_is_bounded_and_given_back():
    torch.cuda.synchronize()
    free0, total = torch.cuda.mem_get_info()
    ctx = A.Context(0)
    op, specs = _op(ctx)
    A.chains_run(op, specs, np.linspace(-0.6, 0.4, 400) + 0.02j)
    held, _ = torch.cuda.mem_get_info()
    assert free0 - held <= total // 8 + (64 << 20)
    op.free()
    ctx.close()
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] <= 64 << 20
