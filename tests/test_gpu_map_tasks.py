"""The GPU-mapping sampler's two ways of sharing refills out over lanes: four lanes per task (few
polynomials in a call) and one (many).  The same polynomials drawn in one call and one at a time must be
the same, and equal the oracle's; 40 polynomials at n = 4096 draw about 60,000 refills, of which a few
need the slow path (three of the first ten uniform words rejected)."""
import numpy as np
import pytest

from oracle.ffi import Oracle, aes256_expand, canon
from tests.conftest import seeds

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402


@pytest.mark.parametrize("sig", [0, 1, 2])
@pytest.mark.parametrize("n,npolys", [(16, 3), (256, 33), (4096, 1), (4096, 40)])
def test_one_call_equals_single_polynomials(sig, n, npolys, rng, oracle_built):
    c = cf.Context(n, 4)
    key = seeds(rng)[0]
    poly0 = 3
    many = c.sample_gpu_map(sig, key, poly0, npolys)
    O = Oracle(n, 4)
    rk = aes256_expand(key)
    for i in range(npolys):
        one = c.sample_gpu_map(sig, key, poly0 + i, 1)
        assert torch.equal(one[0], many[i]), i
        if i % 7 == 0:
            assert (cf.u32(many[i]) == canon(O.gauss_modeB(rk, sig, poly0 + i))).all(), i
    c.sync()
    c.close()
