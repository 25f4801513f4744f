"""Contexts of different lengths on different host threads: the many-key l-sums set nothing that another
context's launch depends on."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402


def test_keygen_of_different_lengths_in_several_threads(rng):
    n, keys, rounds = 64, 200, 2000
    jobs = []
    for l in (1280, 32, 700, 128, 1000, 300):
        c = cf.Context(n, l)
        y = torch.from_numpy(rng.integers(-16, 17, (keys, l)).astype(np.int32)).to(c.dev)
        msk = torch.randint(0, 16000000, (l, 3, n), dtype=torch.int32, device=c.dev)
        want = c.keygen(y, msk, y_signed=True)
        jobs.append((c, y, msk, want, torch.empty_like(want), torch.cuda.Stream()))
    torch.cuda.synchronize()
    errors = []

    def work(c, y, msk, want, out, st):
        try:
            for _ in range(rounds):
                c.keygen(y, msk, y_signed=True, sky=out, stream=st)
            st.synchronize()
            assert torch.equal(out, want)
        except Exception as e:  # reported by the test's thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for j in jobs:
        j[0].close()
