"""The radix sort on both sides of the line between its tile sizes, over one to four passes."""
import numpy as np
import pytest

from libcl_gb300 import RadixSort

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [786431, 786432, 786433, 2097153])
@pytest.mark.parametrize("bits", [(0, 32), (0, 24), (8, 20), (4, 8)])
def test_tile_sizes(cuda, n, bits):
    import torch
    keys = np.random.default_rng(n).integers(0, 1 << 32, n, dtype=np.uint32)
    keys[::3] = keys[0]  # a digit far longer than a tile's share
    k = torch.from_numpy(keys.view(np.int32)).cuda()
    v = torch.arange(n, dtype=torch.int32, device="cuda")
    s = RadixSort()
    s.compute(k, v, *bits)
    digit = (keys >> np.uint32(bits[0])) & np.uint32((1 << (bits[1] - bits[0])) - 1)
    order = np.argsort(digit, kind="stable")
    assert np.array_equal(v.cpu().numpy(), order)
    assert np.array_equal(k.cpu().numpy().view(np.uint32), keys[order])
