"""Decryption into memory that overlaps its inputs: the ciphertexts, the weights, the function keys."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402


@pytest.mark.parametrize("n,l,nct,nkeys", [(256, 9, 1, 4), (1024, 40, 2, 3), (1024, 130, 1, 40), (64, 200, 5, 7), (4096, 33, 1, 2)])
def test_output_over_the_inputs(n, l, nct, nkeys, rng):
    c = cf.Context(n, l)
    poly, gen = 3 * n, torch.Generator(c.dev).manual_seed(n + l)
    sizes = {"dy": nct * nkeys * poly, "ct": nct * (l + 1) * poly, "sky": nkeys * poly, "y": nkeys * l}
    words = {k: torch.randint(0, 16000000, (v,), dtype=torch.int32, device=c.dev, generator=gen) for k, v in sizes.items()}
    words["y"] = torch.from_numpy(rng.integers(-16, 17, sizes["y"]).astype(np.int32)).to(c.dev)

    def call(ct, y, sky, dy, noalloc=False):
        f = c.decrypt_noalloc if noalloc else c.decrypt
        f(ct.view(nct, l + 1, 3, n), y.view(nkeys, l), sky.view(nkeys, 3, n), y_signed=True, dy=dy.view(nct, nkeys, 3, n))
        return dy.clone()

    want = call(words["ct"], words["y"], words["sky"], torch.empty(sizes["dy"], dtype=torch.int32, device=c.dev))
    forms = [False] + ([True] if nct == 1 and nkeys <= 4 else [])
    for name in ("ct", "y", "sky"):
        for shift in (0, 5 * n, -poly):  # the output's start against the input's
            for noalloc in forms:
                base = torch.zeros(2 * poly + sizes["dy"] + sizes[name] + 5 * n, dtype=torch.int32, device=c.dev)
                at = poly
                over = base[at:at + sizes[name]]
                over.copy_(words[name])
                use = dict(words, **{name: over})
                got = call(use["ct"], use["y"], use["sky"], base[at + shift:at + shift + sizes["dy"]], noalloc)
                assert torch.equal(got, want), (name, shift, noalloc)
    c.sync()
    c.close()
