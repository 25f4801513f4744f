"""Coefficient-0 decryption where the tensor cores cannot have it (rings below 64, or residues asked for): per pair or in
integer tiles, whichever the sizes make quicker, with the same residues and values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402


@pytest.mark.parametrize("n,l,nct,nkeys", [(16, 8, 40, 130), (32, 1, 1, 32), (64, 8, 40, 130), (2048, 124, 10, 33), (256, 30, 700, 32),
                                           (16, 300, 3, 50)])
def test_both_ways_give_the_same(n, l, nct, nkeys):
    rng = np.random.default_rng(n + nct)
    c = cf.Context(n, l)
    q = np.array(cf.Q, np.uint32)[None, :, None]
    ct = cf.to_dev(rng.integers(0, 2**31, (nct * (l + 1), 3, n), dtype=np.uint32) % q).reshape(nct, l + 1, 3, n)
    sky = cf.to_dev(rng.integers(0, 2**31, (nkeys, 3, n), dtype=np.uint32) % q)
    y = torch.from_numpy(rng.integers(-16, 17, (nkeys, l)).astype(np.int32)).to(c.dev)
    d0, d1 = (torch.empty((nct, nkeys, 3), dtype=torch.int32, device=c.dev) for _ in range(2))
    want = c.decrypt_coef0_form(0, ct, y, sky, y_signed=True, d0=d0)
    assert torch.equal(c.decrypt_coef0_form(2, ct, y, sky, y_signed=True), want)
    assert torch.equal(c.decrypt_coef0(ct, y, sky, y_signed=True, d0=d1), want) and torch.equal(d0, d1)
    assert torch.equal(c.decrypt_coef0(ct, y, sky, y_signed=True), want)
    c.sync()
    c.close()
