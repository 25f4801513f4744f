"""Encryption and setup run part of their work on a second stream of the context: a call must still be ordered
on the caller's stream as a whole -- behind what produces its inputs, before what reads or overwrites them
afterwards -- for calls in which the two parts share the SMs and calls in which they do not."""
import numpy as np
import pytest

from oracle.ffi import Oracle, canon
from tests.conftest import seeds

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402


@pytest.mark.parametrize("n,l,batch", [(1024, 57, 1), (1024, 57, 4), (1024, 57, 16), (2048, 9, 3), (4096, 130, 2)])
def test_calls_are_ordered_on_their_stream(n, l, batch, rng, oracle_built):
    O = Oracle(n, l)
    ctxs = [cf.Context(n, l) for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    sa, ss, se = (seeds(rng, 1) for _ in range(3))
    rmpk, rmsk = O.setup(sa[0], ss[0], se[0])
    work = torch.randn(2048, 2048, device="cuda")
    torch.cuda.synchronize()
    steps = []
    for k in range(4):
        c, st = ctxs[k % 2], streams[k % 2]
        s2, s3 = seeds(rng, batch), seeds(rng, batch)
        xs = rng.integers(0, 5, (batch, l), dtype=np.uint32)
        src = cf.to_dev(xs)
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            x = torch.zeros_like(src)
            for _ in range(5):
                work @ work  # the inputs arrive late
            mpk, msk = c.setup(sa, ss, se, stream=st)
            x.copy_(src)
            ct = c.encrypt(x, mpk, s2, s3, stream=st)
            got, key = ct.clone(), msk.clone()
            for t in (x, mpk, msk, ct):
                t.zero_()
        steps.append((got, key, s2, s3, xs))
    torch.cuda.synchronize()
    for got, key, s2, s3, xs in steps:
        assert (cf.u32(key) == canon(rmsk)).all()
        for b in range(batch):
            assert (cf.u32(got)[b] == canon(O.encrypt(xs[b], rmpk, s2[b], s3[b]))).all(), b
    for c, st in zip(ctxs, streams):
        c.sync(st)
        c.close()
