"""The table of call ends off its usual path: with windows that follow none or twice of the mean overshoot, the
overshoot leaves the copied part of a row, whose group of calls is made again, and after some hundred calls
the window, whose call ends are searched for.  Samples must equal the oracle's, to the calls that end in
the last tile of 4,096 refills; the same runs by the walk and by doubling too."""
import numpy as np
import pytest

from oracle.ffi import Oracle, canon
from tests.conftest import seeds

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402


@pytest.mark.parametrize("sig,n,calls", [(0, 1024, 400), (1, 1024, 785), (2, 1024, 1024), (2, 4096, 290), (0, 2048, 130), (2, 512, 144),
                                         (2, 1024, 13), (1, 512, 1)])
def test_every_form_equals_the_oracle(sig, n, calls, rng, oracle_built):
    c, O = cf.Context(n, 4), Oracle(n, 4)
    keys = seeds(rng, 2)
    want = np.stack([canon(O.gauss(sig, k, calls)[0]) for k in keys])
    for form in range(6):
        assert (cf.u32(c.sample_cpu_map_form(form, sig, keys, calls)) == want).all(), form
    c.sync()
    c.close()


def test_forms_that_the_sizes_do_not_allow(rng):
    c = cf.Context(256, 4)
    for form in (-1, 3, 4, 5, 6):  # windows of 192 entries or more and 192 between them
        with pytest.raises(cf.CufeError):
            c.sample_cpu_map_form(form, 2, seeds(rng, 1), 20)
    c.close()
