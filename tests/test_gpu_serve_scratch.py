"""A server tick filled to its scratch with long vectors on a small ring: the tables of call ends take more
there than the admission charges per request, and the tick has to run all the same."""
import numpy as np
import pytest

from oracle.ffi import Oracle, canon
from tests.conftest import seeds

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402


@pytest.mark.parametrize("n,ls,counts", [(1024, [1305, 40], [40, 0]), (1024, [1610, 40], [24, 0]), (1024, [1610, 200], [1, 60]),
                                         (512, [1610, 130], [20, 3])])
def test_full_ticks_of_long_vectors(n, ls, counts, rng, oracle_built):
    need = sum(k * (12 * n * (4 + l) + 44 * cf.lib().cufe_sampler_refills(2, l, n) + 480 + 8192) for l, k in zip(ls, counts))
    S = cf.Server([n, n], ls, arena_bytes=2 << 30, tick_bytes=(1 << 20) + need)
    sa, se = seeds(rng, 2), seeds(rng, 2)
    S.setup(sa, None, se)
    reqs = []
    for t in [0] * counts[0] + [1] * counts[1] + [1, 0]:  # a tick that is full, and one more
        x, s2, s3 = rng.integers(0, 5, ls[t]).astype(np.uint32), seeds(rng, 1)[0], seeds(rng, 1)[0]
        reqs.append((S.encrypt(t, x, s2, s3), t, x, s2, s3))
    S.drain()
    assert all(S.result(r[0])[0] == S.DONE for r in reqs) and S.stats()["ticks"] == 2
    for rid, t, x, s2, s3 in (reqs[0], reqs[-2], reqs[-1]):
        O = Oracle(n, ls[t])
        rmpk, _ = O.setup(sa[t], None, se[t])
        got = S.read(rid, (ls[t] + 1) * 3 * n).reshape(ls[t] + 1, 3, n)
        assert (got == canon(O.encrypt(x, rmpk, s2, s3))).all(), t
    S.close()
