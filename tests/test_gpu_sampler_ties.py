"""The CPU-mapping sampler where the top halves of its 64-bit words decide nothing.

The candidate kernel compares the top 32 bits of the CDT and Bernoulli words and recomputes a
candidate from its full words only on a tie.  The keys below (found by search over small keys,
little-endian, in the first 60 refills of their streams) have such ties: Bernoulli ties of either
outcome per sigma, and CDT ties whose sample differs from the one the top half alone suggests.
Every sample must equal the oracle's.
"""
import numpy as np
import pytest

from oracle.ffi import Oracle, canon

pytestmark = pytest.mark.gpu

pytest.importorskip("torch")
import cufe_b200 as cf  # noqa: E402

BERNOULLI = {0: [11165, 14842, 22126, 67466, 73460], 1: [21034, 37189, 73802, 20016395, 20010833],
             2: [635, 18574, 33394, 41498, 60928]}
CDT = [31800472, 33698284, 34295304, 34501038, 40905373, 40103115, 50175422, 60334365, 64360347]


@pytest.mark.parametrize("sig", [0, 1, 2])
def test_tied_words_match_the_oracle(sig, oracle_built):
    n, calls = 512, 2  # at least 94 refills per call
    keys = np.zeros((len(BERNOULLI[sig]) + len(CDT), 32), np.uint8)
    for row, k in zip(keys, BERNOULLI[sig] + CDT):
        row[:8] = np.frombuffer(int(k).to_bytes(8, "little"), np.uint8)
    c = cf.Context(n, 4)
    got = cf.u32(c.sample_cpu_map(sig, keys, calls))
    c.sync()
    O = Oracle(n, 4)
    for i in range(len(keys)):
        ref, _ = O.gauss(sig, keys[i], calls)
        assert (got[i] == canon(ref)).all(), (sig, i)
    c.close()
