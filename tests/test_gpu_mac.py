"""The l-sums of key generation and decryption (cufe_b200/csrc/mac.cu) against integer numpy:
sum_i y[k][i] v[i][m][j] mod q_m, at the edges of its two kernels -- the streamed form (few keys,
long vectors, small rings) and the tensor-core form (tiles of 128 keys, 64 coefficients and 128
slots) -- and of the ranges of y that each takes a shorter route for (a signed byte, 2^15).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402

Q = np.array(cf.Q, np.uint64)


def expect(y, v, signed):
    """y [k][l] uint32 words, v [l][3][n] uint32 words -> [k][3][n]"""
    yr = (y.view(np.int32).astype(np.int64)[:, :, None] if signed else y.astype(np.int64)[:, :, None]) % Q.astype(np.int64)
    vr = v.astype(np.uint64) % Q[None, :, None]
    out = np.empty((len(y),) + v.shape[1:], np.uint32)
    for k in range(len(y)):
        prod = yr[k].astype(np.uint64)[:, :, None] * vr % Q[None, :, None]
        out[k] = prod.sum(0) % Q[:, None]
    return out


# (lowest, highest) y: a signed byte and one beyond, the unsigned byte range, 2^15, any word
RANGES = [(-128, 127, True), (-129, 128, True), (0, 127, False), (0, 128, False), (-32768, 32767, True),
          (-32769, 32768, True), (0, 65536, False), (0, 2**32 - 1, False), (-2**31, 2**31 - 1, True)]


@pytest.mark.parametrize("lo,hi,signed", RANGES)
@pytest.mark.parametrize("n,l,keys", [(16, 5, 9), (64, 127, 8), (64, 128, 129), (128, 129, 7), (32, 1025, 4),
                                      (64, 1280, 9), (64, 1281, 9), (256, 1, 257), (512, 40, 2), (64, 300, 1)])
def test_keygen_sums(n, l, keys, lo, hi, signed):
    rng = np.random.default_rng(n + 7 * l + 31 * keys)
    y = rng.integers(lo, hi + 1, (keys, l), dtype=np.int64)
    y[0, 0], y[-1, -1] = lo, hi  # one key at each end of the range
    v = rng.integers(0, 2**32, (l, 3, n), dtype=np.uint64).astype(np.uint32)
    v[0, :, :2], v[-1, :, :2] = 0xffffffff, [0, 0x7fffffff]
    y = (y % 2**32).astype(np.uint32)
    c = cf.Context(n, l)
    got = cf.u32(c.keygen(cf.to_dev(y), cf.to_dev(v), y_signed=signed))
    # the same buffers off their 16-byte alignment
    vo, so = torch.empty(v.size + 1, dtype=torch.int32, device=c.dev), torch.empty(keys * 3 * n + 1, dtype=torch.int32, device=c.dev)
    vo[1:].copy_(cf.to_dev(v).reshape(-1))
    c.keygen(cf.to_dev(y), vo[1:], y_signed=signed, sky=so[1:])
    c.sync()
    want = expect(y, v, signed)
    assert (got == want).all()
    assert (cf.u32(so[1:]).reshape(want.shape) == want).all()
    c.close()


@pytest.mark.parametrize("n,l", [(64, 20), (256, 131)])
def test_decrypt_many_keys_equals_one_at_a_time(n, l):
    rng = np.random.default_rng(n)
    c = cf.Context(n, l)
    q = Q.astype(np.uint32)[None, None, :, None]
    ct = cf.to_dev(rng.integers(0, 2**31, (3, l + 1, 3, n), dtype=np.uint32) % q)
    sky = cf.to_dev(rng.integers(0, 2**31, (11, 1, 3, n), dtype=np.uint32) % q).reshape(11, 3, n)
    y = torch.from_numpy(rng.integers(-16, 17, (11, l)).astype(np.int32)).to(c.dev)
    many = c.decrypt(ct, y, sky, y_signed=True)
    for k in range(11):
        for z in range(3):
            one = c.decrypt(ct[z:z + 1].contiguous(), y[k:k + 1].contiguous(), sky[k:k + 1].contiguous(), y_signed=True)
            assert torch.equal(one[0, 0], many[z, k]), (z, k)
    c.sync()
    c.close()
