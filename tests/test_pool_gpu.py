"""The device memory pool keeps up to 4 GiB (and up to 1 GiB of rounding) beyond what the program holds, follows it up and
down, and gives the rest back to the driver at the next synchronise."""
import pytest
import torch

from tensorax_b200 import _lib

pytestmark = pytest.mark.gpu

GIB = 1 << 30


def test_freed_blocks_beyond_the_reserve_go_back_to_the_driver():
    lib = _lib.load()

    def free():
        _lib.check(lib.tx_sdpa_finish(None))
        return torch.cuda.mem_get_info()[0]

    _lib.check(lib.tx_cuda_pool_trim())
    start = free()
    blocks = [lib.tx_cuda_malloc(GIB) for _ in range(14)]
    assert all(blocks) and free() <= start - 14 * GIB
    for p in blocks[2:]:
        _lib.check(lib.tx_cuda_free(p))
    assert start - 7.25 * GIB <= free() <= start - 2 * GIB        # two held, at most five kept
    again = [lib.tx_cuda_malloc(GIB) for _ in range(8)]           # and up again
    assert all(again) and free() <= start - 10 * GIB
    for p in blocks[:2] + again:
        _lib.check(lib.tx_cuda_free(p))
    assert free() >= start - 5.25 * GIB
    _lib.check(lib.tx_cuda_pool_trim())
    assert free() >= start - 0.25 * GIB
