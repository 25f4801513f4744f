"""l-sums of a few rows, which have a kernel of their own, at the edges of its rule: 31 and 32 rows, two keys and
groups of four, small rings, several ciphertexts; weights of every size.  Against integer numpy."""
import numpy as np
import pytest

from tests.test_gpu_mac import RANGES, expect

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402


@pytest.mark.parametrize("lo,hi,signed", RANGES)
@pytest.mark.parametrize("n,l,keys", [(4096, 1, 2), (1024, 31, 5), (1024, 32, 5), (256, 8, 130), (16, 100, 40), (8192, 4, 3), (32, 128, 601)])
def test_keygen_sums(n, l, keys, lo, hi, signed):
    rng = np.random.default_rng(n + 7 * l + 31 * keys)
    y = rng.integers(lo, hi + 1, (keys, l), dtype=np.int64)
    y[0, 0], y[-1, -1] = lo, hi
    y = (y % 2**32).astype(np.uint32)
    v = rng.integers(0, 2**32, (l, 3, n), dtype=np.uint64).astype(np.uint32)
    v[0, :, :2] = 0xffffffff
    c = cf.Context(n, l)
    got = cf.u32(c.keygen(cf.to_dev(y), cf.to_dev(v), y_signed=signed))
    c.sync()
    some = np.unique(np.array([0, 1, keys // 2, keys - 2, keys - 1]).clip(0, keys - 1))
    assert (got[some] == expect(y[some], v, signed)).all()
    c.close()


@pytest.mark.parametrize("n,l,cts,keys", [(256, 5, 3, 6), (1024, 20, 9, 3), (64, 31, 40, 2)])
def test_decryption_of_several_ciphertexts(n, l, cts, keys):
    rng = np.random.default_rng(n)
    c = cf.Context(n, l)
    q = np.array(cf.Q, np.uint32)[None, None, :, None]
    ct = cf.to_dev(rng.integers(0, 2**31, (cts, l + 1, 3, n), dtype=np.uint32) % q)
    sky = cf.to_dev((rng.integers(0, 2**31, (keys, 1, 3, n), dtype=np.uint32) % q).reshape(keys, 3, n))
    y = torch.from_numpy(rng.integers(-16, 17, (keys, l)).astype(np.int32)).to(c.dev)
    many = c.decrypt(ct, y, sky, y_signed=True)
    for k in range(keys):
        for z in range(cts):  # one key and ciphertext: streamed
            one = c.decrypt(ct[z:z + 1].contiguous(), y[k:k + 1].contiguous(), sky[k:k + 1].contiguous(), y_signed=True)
            assert torch.equal(one[0, 0], many[z, k]), (z, k)
    c.sync()
    c.close()
