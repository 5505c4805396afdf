"""P and K of every size reach the device and come back whole: below, at and just beyond the size from
which they go through pinned chunks, with a last chunk of one element and fewer chunks than slots."""
import numpy as np
import pytest

from libgint_b200.capi import LibGint

MIN = (8 << 20) // 8         # doubles from which copies are staged
CHUNK = (1 << 20) // 8       # doubles per chunk


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, MIN - 1, MIN, MIN + 1, MIN + CHUNK - 1, 23 * CHUNK + 1])
def test_K_round_trip(engine_so, n):
    g = LibGint()
    g.init()
    rng = np.random.default_rng(n)
    for rep in range(2):     # the second time the chunks hold the first array's end
        K = rng.standard_normal(n)
        g.set_P(np.zeros(n))
        assert not g.get_K(n).any()
        g.set_K(K)
        assert np.array_equal(g.get_K(n), K)
        assert g.last_error()[0] == 0, g.last_error()
    g.close()
