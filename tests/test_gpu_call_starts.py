"""Where the CPU-mapping sampler's calls start: the walk (few calls, or small rings) and the table of
call ends (128 calls or more at rings wide enough for its windows), at the edges of that rule, of the
walk's tiles of 8,192 refills and of the groups of 16 calls, and with streams of different lengths in
one run (a heterogeneous batch).  Every sample must equal the oracle's."""
import numpy as np
import pytest

from oracle.ffi import Oracle, canon
from tests.conftest import seeds

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402


@pytest.mark.parametrize("sig", [0, 1, 2])
@pytest.mark.parametrize("n,calls", [(16, 700), (256, 200), (1024, 127), (1024, 128), (1024, 200), (2048, 333), (4096, 129),
                                     (8192, 144), (4096, 3), (512, 128), (512, 144), (512, 145), (1024, 785), (1024, 1024)])
def test_streams_equal_the_oracle(sig, n, calls, rng, oracle_built):
    c = cf.Context(n, 4)
    keys = seeds(rng, 3)
    got = cf.u32(c.sample_cpu_map(sig, keys, calls))
    c.sync()
    O = Oracle(n, 4)
    for i in range(3):
        ref, _ = O.gauss(sig, keys[i], calls)
        assert (got[i] == canon(ref)).all(), i
    c.close()


def test_mixed_lengths_equal_their_oracle(rng, oracle_built):
    n, l = [1024, 2048, 2048, 4096, 2048], [64, 200, 5, 90, 31]
    b = cf.Batch(n, l)
    sa, se, s2, s3 = (seeds(rng, len(n)) for _ in range(4))
    b.setup(sa, None, se)
    xs = [rng.integers(0, 5, k, dtype=np.int64) for k in l]
    ys = [rng.integers(-16, 17, k, dtype=np.int64) for k in l]
    out = b.bind(cf.to_dev(b.pack(xs).astype(np.uint32)), cf.to_dev(b.pack(ys).astype(np.int32)),
                 cf.bytes_to_dev(s2), cf.bytes_to_dev(s3))
    b.run()
    torch.cuda.synchronize()
    b.status()
    for i in range(len(n)):
        O = Oracle(n[i], l[i])
        rmpk, _ = O.setup(sa[i], None, se[i])
        ct = b.fetch(b.instance(i)[3], (l[i] + 1) * 3 * n[i]).reshape(l[i] + 1, 3, n[i])
        assert (ct == canon(O.encrypt(xs[i].astype(np.uint32), rmpk, s2[i], s3[i]))).all(), i
        assert int(cf.u32(out)[i]) % (64 * l[i] + 1) == int(xs[i] @ ys[i]) % (64 * l[i] + 1)
    b.close()
