"""The radix sort at the edges of its tile shapes, bit for bit against a stable numpy argsort: 256
threads x 2 to 4 pairs (128 tiles at most) up to 131,072 pairs, then 512 and 1024 threads x 5 to 8 (one
tile per SM, 152 of them), then 512 x 6."""
import numpy as np
import pytest

from forcegpu._lib import radix_sort

pytestmark = pytest.mark.gpu

STEP = 256 * 128            # one more pair per thread in the small tiles
SMS = 152


@pytest.mark.parametrize("n", [511, 512, 513, 2 * STEP, 2 * STEP + 1, 3 * STEP + 1, 4 * STEP, 4 * STEP + 1, 200_003,
                               SMS * 512 * 5, SMS * 512 * 5 + 1, SMS * 512 * 6 + 1,
                               SMS * 512 * 7 + 1, SMS * 512 * 8, SMS * 512 * 8 + 1, SMS * 1024 * 5 + 1,
                               SMS * 1024 * 8, SMS * 1024 * 8 + 1])
@pytest.mark.parametrize("lo_bit", [40, 61])
def test_every_shape_is_the_stable_sort(n, lo_bit):
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 63, n, dtype=np.int64).astype(np.uint64) << np.uint64(1)
    ko, vo = radix_sort(keys, np.arange(n, dtype=np.uint32), lo_bit=lo_bit)
    order = np.argsort(keys >> np.uint64(lo_bit), kind="stable")
    np.testing.assert_array_equal(vo, order.astype(np.uint32))
    np.testing.assert_array_equal(ko, keys[order])
