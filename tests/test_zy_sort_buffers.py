"""fl_radix_sort_noalloc with its output apart from its input (the first pass reads the input itself),
in place, and with only one of the two arrays in place, for even and odd numbers of digit passes, at
the edges of its tiles: numpy's stable sort, and an input apart is left as it was."""
import numpy as np
import pytest

from forcegpu._lib import radix_sort_noalloc

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("keys_in_place,vals_in_place", [(False, False), (True, True), (True, False), (False, True)])
@pytest.mark.parametrize("lo_bit", [0, 8, 37, 56])
@pytest.mark.parametrize("n", [1, 511, 513, 65_537, 131_073, 262_143])
def test_sort_for_every_placing_of_the_buffers(n, lo_bit, keys_in_place, vals_in_place):
    rng = np.random.default_rng(n + lo_bit)
    keys = rng.integers(0, 300, n, dtype=np.uint64) << np.uint64(55) | rng.integers(0, 2 ** 40, n, dtype=np.uint64)
    vals = rng.permutation(n).astype(np.uint32)
    k = torch.from_numpy(keys.view(np.int64).copy()).cuda()
    v = torch.from_numpy(vals.view(np.int32).copy()).cuda()
    ko = k if keys_in_place else torch.empty_like(k)
    vo = v if vals_in_place else torch.empty_like(v)
    torch.cuda.synchronize()
    radix_sort_noalloc(k.data_ptr(), v.data_ptr(), n, lo_bit, ko.data_ptr(), vo.data_ptr(), 0)
    order = np.argsort(keys >> np.uint64(lo_bit), kind="stable")
    np.testing.assert_array_equal(ko.cpu().numpy().view(np.uint64), keys[order])
    np.testing.assert_array_equal(vo.cpu().numpy().view(np.uint32), vals[order])
    if not keys_in_place:
        np.testing.assert_array_equal(k.cpu().numpy().view(np.uint64), keys)
    if not vals_in_place:
        np.testing.assert_array_equal(v.cpu().numpy().view(np.uint32), vals)
