"""While a capture that holds a call of a context is open, the context's other calls run on other streams
as before: the second stream of encryption and setup, which the capture has taken in, does not tie them to it."""
import numpy as np
import pytest

from oracle.ffi import Oracle, canon
from tests.conftest import seeds

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402


@pytest.mark.parametrize("n,l", [(256, 9), (1024, 140)])
def test_calls_beside_an_open_capture(n, l, rng, oracle_built):
    O, c = Oracle(n, l), cf.Context(n, l)
    sa, ss, se = (seeds(rng, 1) for _ in range(3))
    rmpk, rmsk = O.setup(sa[0], ss[0], se[0])
    x0 = rng.integers(0, 5, (1, l), dtype=np.uint32)
    x, s2, s3 = cf.to_dev(x0), seeds(rng, 1), seeds(rng, 1)
    mpk, msk = c.setup(sa, ss, se)
    ct = c.encrypt(x, mpk, s2, s3)
    mpk2, msk2, ct2, ct3 = torch.zeros_like(mpk), torch.zeros_like(msk), torch.zeros_like(ct), torch.zeros_like(ct)
    cap, st = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=cap, capture_error_mode="relaxed"):
        c.encrypt(x, mpk, s2, s3, ct=ct, stream=cap)  # not replayed: its seeds are the host's
        c.setup(sa, ss, se, mpk=mpk2, msk=msk2, stream=st)
        c.encrypt(x, mpk2, s2, s3, ct=ct2, stream=st)
        c.encrypt(x, mpk, s2, s3, ct=ct, stream=cap)
    c.encrypt(x, mpk2, s2, s3, ct=ct3, stream=st)
    st.synchronize()
    want = canon(O.encrypt(x0[0], rmpk, s2[0], s3[0]))
    assert (cf.u32(msk2) == canon(rmsk)).all() and (cf.u32(mpk2) == canon(rmpk)).all()
    assert (cf.u32(ct2)[0] == want).all() and (cf.u32(ct3)[0] == want).all()
    c.sync()
    c.close()
