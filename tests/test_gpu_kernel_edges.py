"""Edge sizes of the kernels' batches, rings and tiles: every result equals the
CPU oracle's byte for byte."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 3, 8])
def test_xxh3_around_the_chain_batches(gpu_lib, offset):
    """Lengths around one, two and three batches of the block chain (48 blocks
    of 1 KiB after the first) and every count of trailing stripes."""
    import torch
    import openzl_gb300 as oz

    blocks = [0, 1, 2, 47, 48, 49, 50, 96, 97, 98, 145, 146, 513, 700]
    lengths = [b * 1024 + r for b in blocks for r in (1, 63, 64, 65, 700, 960, 961, 1023, 1024)]
    rng = np.random.default_rng(48)
    data = rng.integers(0, 256, max(lengths) + 16).astype(np.uint8)
    dev = torch.from_numpy(data).cuda()
    for n in lengths:
        want = oracle.lib().ozo_xxh3_64(data[offset:].ctypes.data, n)
        assert oz.xxh3_64_device(dev.data_ptr() + offset, n) == want, n
