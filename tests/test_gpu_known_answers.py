"""Known answers of the clip band and of the k-of-32 as the kernels compute them, against the
oracle: every band (inverted ones too), and values up to the bit planes' largest drive."""
import numpy as np
import pytest

import axon_b200 as ax
import oracle_lib as O

pytestmark = pytest.mark.gpu


def test_every_clip_band():
    """All 16 values of a counter, in every lane, for all 256 pairs of bounds."""
    values = np.arange(16, dtype=np.uint32)
    planes = [np.where((values >> i) & 1, 0xFFFFFFFF, 0).astype(np.uint32) for i in range(4)]
    mask = np.zeros(16, dtype=np.uint32)
    for lo in range(16):
        for hi in range(16):
            got = [p.copy() for p in planes]
            ax.bstest(2, lo, hi, got, mask)
            for e, g in zip(O.bstest(2, lo, hi, [p.copy() for p in planes], mask), got):
                assert np.array_equal(e, g), (lo, hi)


@pytest.mark.parametrize("top", [2, 30, 600, 1 << 14])
def test_k_of_32_on_planes(top):
    rng = np.random.default_rng(top)
    v = rng.integers(0, top, (34 * 40, 32)).astype(np.uint32)
    v[::7] = top - 1  # all equal
    k = np.repeat(np.arange(34, dtype=np.uint32), 40)
    assert np.array_equal(ax.kwtatest(v, k), O.kwtatest(v, k))
