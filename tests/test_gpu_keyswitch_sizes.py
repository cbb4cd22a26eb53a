"""Identity key switching at the edges of its tiles and work split, bit-exact
against the oracle: 128-unit tiles taken in pairs, one key switch spread over all
SMs, accumulators cut between CTAs, and a result written over its own input."""
import numpy as np
import pytest

from cufhepp_b200 import client, engine, params as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [1, 7, 8, 9, 127, 128, 129, 255, 256, 257, 385]


@pytest.fixture(scope="module")
def setup(keys):
    sk, ek, _ = keys
    engine.initialize(ek)
    n = max(SIZES)
    rng = np.random.default_rng(81)
    x = rng.integers(0, 2**32, (n, P.TLWE1_WORDS), dtype=np.uint64).astype(np.uint32)
    # digits of every value, and the extreme words
    x[0] = 0
    x[1] = 0xFFFFFFFF
    x[2] = 0x7FFFFFFF
    x[3] = 0x80000000
    yield x, O.iks_batch(x, None, 1, 0, 0, ek.ksk)
    engine.cleanup()


@pytest.mark.parametrize("n", SIZES)
def test_sizes(setup, n):
    x, want = setup
    d = engine.to_device(x[:n])
    out = engine.DeviceBuffer(n * P.TLWE0_WORDS * 4)
    for _ in range(2):  # the rows are cleared on every call
        engine.identity_keyswitch(d, n, out)
    assert np.array_equal(engine.from_device(out, (n, P.TLWE0_WORDS)), want[:n])


def test_result_over_its_input(setup):
    x, want = setup
    n = 257
    d = engine.to_device(x[:n])
    engine.identity_keyswitch(d, n, d)
    assert np.array_equal(engine.from_device(d, (n, P.TLWE0_WORDS)), want[:n])
