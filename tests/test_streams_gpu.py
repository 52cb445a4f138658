"""Streams rejoined and normed with a row in registers: rows of part of a CTA's threads, of one, two and four pieces a thread, and those the
general kernels keep (rows that 16-byte pieces do not cover, three streams), against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("S", [1, 2, 3, 4])
@pytest.mark.parametrize("hidden", [4, 130, 132, 1024, 4096, 4100, 8196, 16384])
def test_join_and_norm(S, hidden, dtype):
    from vllm_cpp_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(S * hidden)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    n = 5
    x, y, mix, out_coef, coef, w, b = rnd(S, n, hidden), rnd(n, hidden).to(dtype), rnd(S, S), rnd(S), rnd(S), rnd(hidden), rnd(hidden)
    want = torch.einsum("st,snd->tnd", mix.double(), x.double()) + out_coef.double()[:, None, None] * y.double()

    def normed(streams, bias):
        u = torch.einsum("s,snd->nd", coef.double(), streams)
        d = u - u.mean(-1, keepdim=True)
        return d / (d.square().mean(-1, keepdim=True) + 1e-6).sqrt() * w.double() + (b.double() if bias else 0.0)
    # sums of a few products and of a row's squares in float32, and the stored type's rounding
    tol = 3e-5 if dtype == torch.float32 else 2.0 ** -8
    for bias in (True, False):
        got, out = x.clone(), torch.full((n, hidden), 9.0, dtype=dtype, device="cuda")
        ops.stream_join(got, y, mix, out_coef, 1e-6, coef, w, b if bias else None, out)
        assert bool(((got.double() - want).abs() <= 1e-5 * (1 + want.abs())).all())
        ref = normed(want, bias)
        assert bool(((out.double() - ref).abs() <= tol * (4 + ref.abs())).all())
    got = x.clone()
    ops.stream_join(got, y, mix, out_coef)
    assert bool(((got.double() - want).abs() <= 1e-5 * (1 + want.abs())).all())
    rows = torch.tensor([4, 0, 2], dtype=torch.int32, device="cuda")
    out = torch.empty(3, hidden, dtype=dtype, device="cuda")
    ops.stream_norm(x, coef, w, b, out, 1e-6, row_index=rows, out_scale=0.5)
    ref = 0.5 * normed(x.double(), True)[rows.long()]
    assert bool(((out.double() - ref).abs() <= tol * (4 + ref.abs())).all())
