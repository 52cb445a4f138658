"""The height of the expert products' tiles: by the pairs an expert gets, and on tcgen05 by the products' size."""
import pytest

from vllm_cpp_b200.csrc import ops


@pytest.mark.parametrize("n,top,experts,size,plain,tensor", [
    (8, 4, 32, 4096 * 2048, 16, 16),              # a pair an expert
    (127, 4, 32, 4096 * 2048, 16, 16), (128, 4, 32, 4096 * 2048, 16, 128),
    (511, 4, 32, 4096 * 2048, 16, 128), (512, 4, 32, 4096 * 2048, 64, 128), (2048, 4, 32, 4096 * 2048, 64, 128),
    (64, 2, 8, 2048 * 1024, 16, 16), (192, 2, 8, 2048 * 1024, 16, 128),
    (800, 1, 4, 1024 * 512, 64, 128), (512, 1, 4, 1024 * 512, 64, 16),
    (300, 2, 3, 64 * 96, 64, 16), (300, 2, 3, None, 64, 128)])
def test_heights(n, top, experts, size, plain, tensor):
    assert ops.moe_tile_rows(n, top, experts) == plain
    assert ops.moe_tile_rows(n, top, experts, True, size) == tensor
    assert ops.moe_max_tiles(n, top, experts, tensor) >= -(-n * top // tensor)
