"""Transforms and key material on buffers that start on a 16-byte but not a 32-byte boundary: the
kernels that hold 16 consecutive coefficients per thread read and write 256 bits at a time where the
address allows it and 128 where it does not.  Both must give the same residues, and so must the launches
for few and for many transforms."""
import numpy as np
import pytest

from tests.conftest import seeds

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402


def shifted(t):
    buf = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    assert buf.data_ptr() % 32 == 0
    v = buf[4:4 + t.numel()].view(t.shape)
    v.copy_(t)
    return v


@pytest.mark.parametrize("variant", [1, 2, 3, 6, 8, 9])
@pytest.mark.parametrize("n", [16, 64, 1024, 2048, 4096, 8192])
def test_transforms(n, variant, rng):
    ring = cf.Ring(n, 3)
    ring.set_variant(variant, variant)
    a = cf.to_dev(np.stack([rng.integers(0, q, (5, n), dtype=np.uint32) for q in ring.primes], axis=1))
    b = shifted(a)
    f, g = ring.forward(a.clone()), ring.forward(b)
    assert torch.equal(f, g)
    assert torch.equal(ring.inverse(g), a) and torch.equal(ring.inverse(f), a)
    ring.close()


@pytest.mark.parametrize("n,rows", [(1024, 394), (1024, 395), (4096, 98), (4096, 99), (8192, 1), (8192, 100),
                                    (1024, 1578), (1024, 1579), (4096, 394), (4096, 395), (8192, 196), (8192, 199)])
def test_one_launch_or_two(n, rows, rng):
    """few transforms go in one launch for all moduli, more in one per class of modulus: the same residues"""
    ring = cf.Ring(n, 3)
    a = cf.to_dev(np.stack([rng.integers(0, q, (rows, n), dtype=np.uint32) for q in ring.primes], axis=1))
    f = ring.forward(a.clone())
    for i in range(0, rows, 40):
        assert torch.equal(ring.forward(a[i:i + 40].clone()), f[i:i + 40])
        assert torch.equal(ring.inverse(f[i:i + 40].clone()), a[i:i + 40])
    assert torch.equal(ring.inverse(f), a)
    ring.close()


@pytest.mark.parametrize("n", [1024, 4096])
def test_scheme(n, rng):
    c = cf.Context(n, 3)
    sa, ss, se, s2, s3 = (seeds(rng, 1) for _ in range(5))
    mpk, msk = c.setup(sa, ss, se)
    mpk2, msk2 = c.setup(sa, ss, se, mpk=shifted(mpk), msk=shifted(msk))
    assert torch.equal(mpk, mpk2) and torch.equal(msk, msk2)
    x = cf.to_dev(rng.integers(0, 5, (1, 3), dtype=np.uint32))
    y = cf.to_dev(rng.integers(0, 17, (1, 3), dtype=np.uint32))
    ct = c.encrypt(x, mpk, s2, s3)
    ct2 = c.encrypt(x, mpk2, s2, s3, ct=shifted(ct))
    assert torch.equal(ct, ct2)
    sk = c.keygen(y, msk)
    assert torch.equal(c.decrypt(ct, y, sk), c.decrypt(ct2, y, shifted(sk)))
    c.close()
