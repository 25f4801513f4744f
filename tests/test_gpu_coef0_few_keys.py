"""Coefficient-0 decryption with fewer than 32 keys leaves the context's workspace alone: it may overlap the
context's other calls on other streams, and be captured on a context whose workspace is still small.
Values are compared with the kernel of one CTA per pair."""
import numpy as np
import pytest

from tests.conftest import seeds

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402


def operands(c, nct, nkeys, rng):
    q = torch.tensor(np.array(cf.Q, np.int64), device=c.dev)[None, :, None]
    gen = torch.Generator(c.dev).manual_seed(nct + nkeys)

    def residues(rows):
        return torch.remainder(torch.randint(0, 2**31 - 1, (rows, 3, c.n), device=c.dev, generator=gen), q).to(torch.int32)

    ct = residues(nct * (c.l + 1)).reshape(nct, c.l + 1, 3, c.n)
    y = torch.from_numpy(rng.integers(-16, 17, (nkeys, c.l)).astype(np.int32)).to(c.dev)
    return ct, y, residues(nkeys)


@pytest.mark.parametrize("nct,nkeys", [(1024, 1), (64, 16), (70, 31)])
def test_overlaps_the_contexts_other_calls(nct, nkeys, rng):
    c = cf.Context(256, 40)
    ct, y, sky = operands(c, nct, nkeys, rng)
    want = c.decrypt_coef0_form(0, ct, y, sky, y_signed=True)
    mpk, _ = c.setup(*seeds(rng, 3))
    x = cf.to_dev(rng.integers(0, 5, (4, 40), dtype=np.uint32))
    s2, s3 = seeds(rng, 4), seeds(rng, 4)
    ct_want = c.encrypt(x, mpk, s2, s3)
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    outs, cts = [], []
    for _ in range(40):
        for st in streams[:2]:  # each other's scratch, and the encryptions' workspace
            with torch.cuda.stream(st):
                outs.append(c.decrypt_coef0(ct, y, sky, y_signed=True, stream=st))
        with torch.cuda.stream(streams[2]):
            cts.append(c.encrypt(x, mpk, s2, s3, stream=streams[2]))
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs)
    assert all(torch.equal(o, ct_want) for o in cts)
    c.sync()
    c.close()


@pytest.mark.parametrize("nct,nkeys", [(1030, 1), (80, 31)])
def test_captures_on_a_new_context(nct, nkeys, rng):
    c = cf.Context(1024, 20)
    ct, y, sky = operands(c, nct, nkeys, rng)
    want = c.decrypt_coef0_form(0, ct, y, sky, y_signed=True)
    out = torch.zeros_like(want)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        c.decrypt_coef0(ct, y, sky, y_signed=True, out=out)
    # a call that has to allocate, on another stream, while this thread captures
    st, other = torch.cuda.Stream(), torch.zeros_like(want)
    g2 = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g2):
        out.add_(0)
        c.decrypt_coef0(ct, y, sky, y_signed=True, out=other, stream=st)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want) and torch.equal(other, want)
    c.close()


def test_slices_of_the_scratch(rng):
    c = cf.Context(64, 1)
    ct, y, sky = operands(c, 200000, 2, rng)  # 307 MB of packed ciphertexts
    assert torch.equal(c.decrypt_coef0(ct, y, sky, y_signed=True), c.decrypt_coef0_form(0, ct, y, sky, y_signed=True))
    c.sync()
    c.close()
