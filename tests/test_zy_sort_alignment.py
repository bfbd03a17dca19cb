"""fl_radix_sort_noalloc with buffers that start between two elements: such an input, apart from its
output, is sorted as any other, and such an output is refused before anything runs."""
import numpy as np
import pytest

from forcegpu._lib import FL_E_ARG, FlError, radix_sort_noalloc


@pytest.mark.gpu
@pytest.mark.parametrize("koff,voff", [(0, 0), (4, 0), (0, 2), (1, 3)])
@pytest.mark.parametrize("lo_bit", [0, 56])
@pytest.mark.parametrize("n", [1, 1000, 70_000])
def test_an_input_may_start_at_any_byte(n, lo_bit, koff, voff):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + koff)
    keys = rng.integers(0, 300, n, dtype=np.uint64) << np.uint64(55) | rng.integers(0, 2 ** 40, n, dtype=np.uint64)
    vals = rng.permutation(n).astype(np.uint32)

    def place(a, off):  # the bytes of `a` on the GPU, `off` bytes after an aligned address
        return torch.from_numpy(np.concatenate([np.zeros(off, np.uint8), a.view(np.uint8)])).cuda()

    k, v = place(keys, koff), place(vals, voff)
    ko = torch.empty(n, dtype=torch.int64, device="cuda")
    vo = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    radix_sort_noalloc(k.data_ptr() + koff, v.data_ptr() + voff, n, lo_bit, ko.data_ptr(), vo.data_ptr(), 0)
    order = np.argsort(keys >> np.uint64(lo_bit), kind="stable")
    np.testing.assert_array_equal(ko.cpu().numpy().view(np.uint64), keys[order])
    np.testing.assert_array_equal(vo.cpu().numpy().view(np.uint32), vals[order])
    np.testing.assert_array_equal(k.cpu().numpy()[koff:], keys.view(np.uint8))  # the input is left as it was
    np.testing.assert_array_equal(v.cpu().numpy()[voff:], vals.view(np.uint8))


@pytest.mark.parametrize("koff,voff", [(4, 0), (0, 2)])
def test_an_output_between_two_elements_is_refused(koff, voff):
    at = 1 << 20  # addresses that the call must not touch
    with pytest.raises(FlError) as e:
        radix_sort_noalloc(at, 2 * at, 100, 0, 3 * at + koff, 4 * at + voff, 0)
    assert e.value.code == FL_E_ARG and "aligned" in str(e.value)
