"""The searches for the samplers' call starts that a run can be given -- the walk and pointer doubling by
cufe_sampler_call_search, the rule's own choice among them and the table -- against the oracle: few and many
calls, one refill per call, streams over several tiles of 4,096 refills, uneven streams in one run."""
import numpy as np
import pytest

from oracle.ffi import Oracle, canon
from tests.conftest import seeds

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402


@pytest.fixture
def search():
    def choose(mode):
        assert cf.lib().cufe_sampler_call_search(mode) == 0
    yield choose
    choose(0)


@pytest.mark.parametrize("sig,n,calls", [(0, 16, 1), (2, 16, 3000), (1, 64, 1023), (2, 64, 1024), (0, 512, 784), (2, 512, 1025),
                                         (2, 1024, 300), (1, 4096, 40), (2, 8192, 17)])
def test_every_search_equals_the_oracle(sig, n, calls, rng, oracle_built, search):
    c, O = cf.Context(n, 4), Oracle(n, 4)
    keys = seeds(rng, 3)
    want = np.stack([canon(O.gauss(sig, k, calls)[0]) for k in keys])
    for mode in (0, 1, 2):
        search(mode)
        assert (cf.u32(c.sample_cpu_map(sig, keys, calls)) == want).all(), mode
    c.sync()
    c.close()


@pytest.mark.parametrize("n,l", [([256, 512, 256, 1024], [900, 3, 1500, 64]), ([2048, 256, 256], [130, 1, 1400])])
def test_uneven_streams(n, l, rng, oracle_built, search):
    sa, se, s2, s3 = (seeds(rng, len(n)) for _ in range(4))
    xs = [rng.integers(0, 5, k).astype(np.uint32) for k in l]
    for mode in (0, 1, 2):
        search(mode)
        b = cf.Batch(n, l)
        b.setup(sa, None, se)
        b.bind(cf.to_dev(b.pack(xs).astype(np.uint32)), cf.to_dev(np.zeros(sum(l), np.int32)), cf.bytes_to_dev(s2),
               cf.bytes_to_dev(s3))
        b.run()
        torch.cuda.synchronize()
        b.status()
        for i in range(len(n)):
            O = Oracle(n[i], l[i])
            rmpk, _ = O.setup(sa[i], None, se[i])
            ct = b.fetch(b.instance(i)[3], (l[i] + 1) * 3 * n[i]).reshape(l[i] + 1, 3, n[i])
            assert (ct == canon(O.encrypt(xs[i], rmpk, s2[i], s3[i]))).all(), (mode, i)
        b.close()
