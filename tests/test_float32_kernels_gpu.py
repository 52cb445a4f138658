"""The 32-bit path's product at the edges of its tiles and of the rules that pick a kernel, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from vllm_cpp_b200.csrc import ops
    return ops


def _rand(gen, *shape):
    return torch.randn(*shape, device="cuda", generator=gen)


# (N, K): one column, a column beyond a tile, few and many columns; one k, a k beyond a copy's 32, sums of 1, 2, 4 and 8 slices, a last
# slice that is short, K that 16-byte copies do not cover
SHAPES = [(1, 1), (129, 33), (127, 511), (257, 516), (65, 2050), (130, 2052), (16385, 36), (16384, 640), (300, 4100)]


@pytest.mark.parametrize("n,k", SHAPES)
def test_product_rows_do_not_depend_on_the_call(ops, n, k):
    """Every M of the dispatch: within the bound of a float chain (each of the K roundings is at most 2^-24 of the sum of
    magnitudes so far) and, row by row, the same bits whatever M."""
    gen = torch.Generator(device="cuda").manual_seed(n + k)
    a, w = _rand(gen, 300, k), _rand(gen, n, k)
    want = a.double() @ w.double().T
    bound = (k + 8) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    whole = torch.empty(300, n, device="cuda")
    ops.gemm_f32(a, w, whole)
    assert bool(((whole.double() - want).abs() <= bound).all())
    for m in (1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 127, 129):
        out = torch.full((m, n), 7.0, device="cuda")
        ops.gemm_f32(a[:m], w, out)
        assert torch.equal(out, whole[:m]), m


@pytest.mark.parametrize("m", [3, 12, 40, 200])
def test_product_of_strided_and_misaligned_rows(ops, m):
    gen = torch.Generator(device="cuda").manual_seed(m)
    big_a, big_w = _rand(gen, m, 1031), _rand(gen, 133, 1031)
    a, w = big_a[:, 3:3 + 1024], big_w[:, 1:1 + 1024]                    # rows of 16-byte pieces at addresses that are not
    out = torch.zeros(m, 140, device="cuda")
    ops.gemm_f32(a, w, out[:, 5:5 + 133])
    want = torch.empty(m, 133, device="cuda")
    ops.gemm_f32(a.contiguous(), w.contiguous(), want)
    assert torch.equal(out[:, 5:138], want) and not out[:, :5].any() and not out[:, 138:].any()
