"""The experts' products on tcgen05 (tiles of 128 rows) at the edges of their tiles, against 64 bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _lists(ops, ids, n_experts):
    n, top = ids.shape
    tiles = ops.moe_max_tiles(n, top, n_experts, 128)
    z = lambda k: torch.full((k,), -1, dtype=torch.int32, device="cuda")  # noqa: E731
    lists = dict(sorted_token=z(n * top), pos=z(n * top), tile_expert=z(tiles), tile_row0=z(tiles), tile_rows=z(tiles), meta=z(4))
    ops.moe_sort(ids, n_experts, 128, *lists.values())
    return lists, tiles


# tokens on (experts, choices): one row; a tile to the row and one beyond; experts without rows and with several tiles, an identity expert.
# (N, K): below a tile and beyond one, whole tiles, K of less than a slice, of a slice and 8, of more slices than stages
@pytest.mark.parametrize("n,experts,top", [(1, 3, 1), (128, 1, 1), (129, 2, 2), (300, 7, 3)])
@pytest.mark.parametrize("N,K", [(8, 8), (136, 72), (256, 64), (520, 264)])
@pytest.mark.parametrize("mode", ["gated", "gelu", "plain"])
def test_products(n, experts, top, N, K, mode):
    from vllm_cpp_b200.csrc import ops
    rng = np.random.default_rng(n + N)
    gen = torch.Generator(device="cuda").manual_seed(n * N + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    chosen = np.stack([rng.permutation(experts + 1)[:top] if experts > 1 else np.zeros(top, int) for _ in range(n)])    # `experts`: an identity
    if n == 300:
        chosen[:, 0] = np.where(chosen[:, 1:].min(1) > 0, 0, chosen[:, 0])       # expert 0 gets several tiles
    ids = torch.from_numpy(chosen.astype(np.int32)).cuda()
    lists, tiles = _lists(ops, ids, experts)
    args = (lists["sorted_token"], lists["tile_expert"], lists["tile_row0"], lists["tile_rows"], lists["meta"], tiles, 128)
    pos = lists["pos"].view(n, top)
    rows = int((pos >= 0).sum())
    pairs = n * top
    token_of = torch.zeros(pairs, dtype=torch.long, device="cuda")
    expert_of = torch.zeros(pairs, dtype=torch.long, device="cuda")
    t, c = (pos >= 0).nonzero(as_tuple=True)
    token_of[pos[t, c].long()], expert_of[pos[t, c].long()] = t, ids[t, c].long()
    out = torch.full((pairs, N), 7.0, dtype=torch.float32 if mode == "plain" else torch.bfloat16, device="cuda")
    w = (rnd(experts, 2 * N if mode == "gated" else N, K) * K ** -0.5).bfloat16()
    if mode == "plain":
        a = rnd(pairs, K).bfloat16()
        ops.moe_expert_gemm(a, w, out, *args, gated=False)
        x = a.double()
    else:
        a = rnd(n, K + 8).bfloat16()[:, :K]                                       # rows of a wider buffer
        scale = torch.rand(pairs, device="cuda") + 0.5 if mode == "gelu" else None
        ops.moe_expert_gemm(a, w, out, *args, gated=mode == "gated", gelu=mode == "gelu", limit=1.5, alpha=1.702, up_shift=1.0, row_scale=scale)
        x = a.double()[token_of]
    ops.check_status()
    got = out.double()
    assert bool((got[rows:] == 7.0).all())                                        # pairs without a row
    for e in range(experts):
        at = ((expert_of == e) & (torch.arange(pairs, device="cuda") < rows)).nonzero()[:, 0]
        z = x[at] @ w[e].double().T
        mag = x[at].abs() @ w[e].double().abs().T
        tol = 2.0 ** -20 * mag                                                    # float sums of at most 264 products
        if mode == "gated":
            g, u = z[:, :N].clamp(max=1.5), z[:, N:].clamp(-1.5, 1.5)
            want = g * torch.sigmoid(1.702 * g) * (u + 1.0)
            tol = 4 * (tol[:, :N] + tol[:, N:]) + 2.0 ** -8 * want.abs() + 1e-6
        elif mode == "gelu":
            want = torch.nn.functional.gelu(z * scale[at].double()[:, None])
            tol = 4 * tol + 2.0 ** -8 * want.abs() + 1e-6
        else:
            want = z
        assert bool(((got[at] - want).abs() <= tol).all()), (mode, e)


@pytest.mark.parametrize("step,first", [(64, 0), (72, 8), (66, 0), (72, 1)])
def test_rows_that_16_byte_copies_do_not_fit(step, first):
    """Tokens' rows anywhere: those at other than 16-byte boundaries take the products that read single elements."""
    from vllm_cpp_b200.csrc import ops
    from vllm_cpp_b200.parts.base import Workspace
    from vllm_cpp_b200.parts.moe import RoutedExperts
    gen = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    n, width, ff, experts, top = 300, 64, 72, 4, 2
    part = RoutedExperts(width, ff, experts, 0, top, 1.5, torch.bfloat16, "cuda", correction=False)
    params = {"router": rnd(experts, width)}
    for e in range(experts):
        params.update({f"e{e}.gate": (rnd(ff, width) / 8).bfloat16(), f"e{e}.up": (rnd(ff, width) / 8).bfloat16(), f"e{e}.down": (rnd(width, ff) / 8).bfloat16()})
    part.load_params(params)
    x = torch.empty(n * step + first, dtype=torch.bfloat16, device="cuda")[first:].view(n, step)[:, :width].copy_(rnd(n, width))
    assert ops.moe_tensor_tiles(x, width, ff) == (step != 66 and first != 1)
    out, z = torch.empty(n, width, dtype=torch.bfloat16, device="cuda"), x.double() @ params["router"].double().T
    part.forward(x, out, None, Workspace("cuda"))
    ops.check_status()
    p = torch.softmax(z, 1)
    best, ids = p.topk(top, dim=1)
    want = torch.zeros(n, width, dtype=torch.float64, device="cuda")
    for e in range(experts):
        g, u = (x.double() @ params[f"e{e}.{m}"].double().T for m in ("gate", "up"))
        g, u = g.clamp(max=1.5), u.clamp(-1.5, 1.5)
        act = (g * torch.sigmoid(1.702 * g) * (u + 1.0)).bfloat16().double()
        want += (act @ params[f"e{e}.down"].double().T) * (best * (ids == e)).sum(1, keepdim=True)
    clear = (p.topk(top + 1, dim=1).values.diff(dim=1)[:, -1].abs() > 1e-4)
    # the activation's rounding, which falls the other way near ties, and the result's
    assert bool(((out.double() - want).abs()[clear] <= 2.0 ** -7 * want.abs().max()).all())
