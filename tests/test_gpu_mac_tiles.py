"""Many-key l-sums in which every CTA walks over several coefficient tiles, back to back, so that its waits for
the tensor core take turns with its loads and stores.  Against integer numpy."""
import numpy as np
import pytest

from tests.test_gpu_mac import expect

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402


@pytest.mark.parametrize("n,l,keys", [(1024, 33, 600), (4096, 129, 260), (2048, 300, 300), (8192, 32, 130)])
def test_several_tiles_per_cta(n, l, keys):
    rng = np.random.default_rng(n + l + keys)
    y = rng.integers(-128, 128, (keys, l)).astype(np.int32).view(np.uint32)
    v = rng.integers(0, 2**32, (l, 3, n), dtype=np.uint64).astype(np.uint32)
    c = cf.Context(n, l)
    dy, dv = cf.to_dev(y), cf.to_dev(v)
    got = [c.keygen(dy, dv, y_signed=True) for _ in range(8)]
    c.sync()
    assert all(torch.equal(g, got[0]) for g in got)
    some = [0, 127, 128, keys - 1]
    assert (cf.u32(got[0])[some] == expect(y[some], v, True)).all()
    c.close()
