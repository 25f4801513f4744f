"""GPU-mapping encryption of one or two vectors with the ciphertexts written over the public key."""
import numpy as np
import pytest

from tests.conftest import seeds

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402


@pytest.mark.parametrize("n,l,batch", [(256, 9, 1), (256, 9, 2), (1024, 57, 2), (4096, 130, 2), (2048, 400, 2)])
def test_ciphertexts_over_the_public_key(n, l, batch, rng):
    c = cf.Context(n, l)
    mpk, _ = c.setup(*seeds(rng, 3))
    x = cf.to_dev(rng.integers(0, 5, (batch, l), dtype=np.uint32))
    s2 = seeds(rng, 1)
    want = c.encrypt_gpu_map(x, mpk, s2)
    for _ in range(20):
        ct = torch.zeros_like(want)
        ct[0].copy_(mpk)
        c.encrypt_gpu_map(x, ct[0], s2, ct=ct)
        assert torch.equal(ct, want)
    c.sync()
    c.close()
