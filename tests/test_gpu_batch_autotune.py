"""The batch autotuner leaves the sort's digit and tile alone where the step it keeps uses neither."""
import pytest

from libcl_gb300 import BUF_FORCE, BUF_POSITION, BUF_VELOCITY, OPT_RADIX_BITS, OPT_SORT_TILE, Batch3D
from libcl_gb300.scenes import batched_ensemble

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,tile", [(6, 8), (6, 16), (7, 8), (7, 16), (8, 8), (8, 16)])
def test_digit_and_tile_stay_with_the_counting_sort(cuda, bits, tile):
    import torch
    b = batched_ensemble(n_scenes=12, seed=3, n_min=1000, n_max=20000)
    bt = Batch3D()
    bt.set_scenes(b.shared, b.descs)
    bt.buffer(BUF_POSITION).copy_(torch.from_numpy(b.pos))
    bt.buffer(BUF_VELOCITY).zero_()
    bt.buffer(BUF_FORCE).zero_()
    bt.set_option(OPT_RADIX_BITS, bits)
    bt.set_option(OPT_SORT_TILE, tile)
    bt.autotune()
    cfg = bt.config()
    if not cfg["persistent"]:
        assert (cfg["radix_bits"], cfg["sort_tile_items"]) == (bits, tile)
    bt.compute()
    assert bt.sync_status() == 0
