"""The coefficient-0 decryption on the tensor cores (cufe_b200/csrc/coef0.cu) against the kernel of
one CTA per pair, at the edges of its tiles (128 ciphertexts, 64 keys, chunks of 64 slots, 8,192
slots in all) and with the largest residues, through the decoded values of every pair."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402


@pytest.mark.parametrize("n,l,nct,nkeys", [(64, 1, 1, 1), (64, 64, 128, 64), (64, 65, 129, 65), (128, 63, 3, 130),
                                           (1024, 40, 257, 5), (4096, 4096, 2, 3), (4096, 784, 130, 66), (8192, 1, 2, 2)])
def test_tensor_core_product_matches_per_pair(n, l, nct, nkeys):
    rng = np.random.default_rng(n + l + nct)
    c = cf.Context(n, l)
    q = torch.tensor(np.array(cf.Q, np.int64), device=c.dev)[None, :, None]

    def residues(*shape):
        u = torch.from_numpy(rng.integers(0, 2**31, 4096 + n, dtype=np.int64)).to(c.dev)
        i = torch.randint(0, u.numel(), shape, device=c.dev, generator=torch.Generator(c.dev).manual_seed(n))
        return (u[i] % q).to(torch.int32)

    ct = residues(nct, (l + 1), 3, n) if nct * l * n < 2**24 else residues(nct * (l + 1), 3, n).reshape(nct, l + 1, 3, n)
    sky = residues(nkeys, 3, n)
    ct[0, -1], sky[0] = (q[0] - 1).to(torch.int32), (q[0] - 1).to(torch.int32)  # largest sums of every diagonal
    sky[-1, :, 0] = 0  # b_0 = 0
    y = torch.from_numpy(rng.integers(-16, 17, (nkeys, l)).astype(np.int32)).to(c.dev)
    for signed in (True, False):
        ref = c.decrypt_coef0_form(0, ct, y, sky, y_signed=signed)
        got = c.decrypt_coef0_form(1, ct, y, sky, y_signed=signed)
        c.sync()
        assert torch.equal(ref, got), signed
    c.close()
