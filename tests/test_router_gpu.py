"""Router logits of few tokens (a warp per output and one or two tokens), of many (five outputs a warp) and of rows that 4-element pieces do not cover, and the
choices' rows joined four elements at a time and one at a time; against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,width,outs", [(1, 4, 3), (8, 1028, 33), (9, 2052, 16), (64, 4096, 40), (65, 4096, 16), (65, 1028, 17), (71, 132, 41), (200, 260, 130), (700, 516, 33), (160, 516, 130),
                                          (3, 1030, 9), (70, 1030, 9)])
def test_logits_and_choice(n, width, outs, dtype):
    from vllm_cpp_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(n + width)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    top = min(4, outs)
    h = rnd(n, width + 4).to(dtype)[:, :width]
    w = rnd(outs, width) / width ** 0.5
    ids, weights = torch.empty(n, top, dtype=torch.int32, device="cuda"), torch.empty(n, top, device="cuda")
    logits = torch.full((n, outs), 9.0, device="cuda")
    ops.moe_router(h, w, None, ids, weights, logits, score="sigmoid")
    want = h.double() @ w.double().T
    # float32 sums of `width` products of size 1 / sqrt(width), in at most 32 + 8 + width / 256 steps
    assert bool(((logits.double() - want).abs() <= 1e-5).all())
    assert torch.equal(ids.long(), logits.topk(top, dim=1).indices)
    assert bool(((weights.double() - torch.sigmoid(logits.double()).gather(1, ids.long())).abs() <= 1e-6).all())


# one kernel or another by the number of logits: 1 and 8 tokens a warp each, then two tokens a warp, then many
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("outs,width", [(3, 4), (16, 132), (33, 1028), (64, 4096), (130, 260), (17, 1030)])
def test_logits_do_not_depend_on_the_step(outs, width, dtype):
    """A token's logits are the same bits in whichever step it stands, so a near tie is decided alike."""
    from vllm_cpp_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(outs)
    h, w = torch.randn(700, width, device="cuda", generator=gen).to(dtype), torch.randn(outs, width, device="cuda", generator=gen)

    def logits(rows):
        n, z = rows.shape[0], torch.empty(rows.shape[0], outs, device="cuda")
        ops.moe_router(rows, w, None, torch.empty(n, 1, dtype=torch.int32, device="cuda"), torch.empty(n, 1, device="cuda"), z, score="sigmoid")
        return z
    whole = logits(h)
    for n in (1, 8, 64, 65, 76, 150, 301):
        assert torch.equal(logits(h[:n]), whole[:n]), n
    odd = torch.empty(5, width + 1, dtype=dtype, device="cuda")[:, :width]      # rows that pieces do not cover: the third kernel
    if width % 4 == 0:
        assert torch.equal(logits(odd.copy_(h[:5])), whole[:5])


@pytest.mark.parametrize("n,width", [(3, 1028), (8, 4), (5, 3076), (65, 1028), (3, 1030)])
def test_logits_of_infinite_activations(n, width):
    """An infinite activation gives infinite logits, of its weight's sign; other tokens' logits do not see it."""
    from vllm_cpp_b200.csrc import ops
    outs = 12
    gen = torch.Generator(device="cuda").manual_seed(width)
    h, w = torch.randn(n, width, device="cuda", generator=gen), torch.randn(outs, width, device="cuda", generator=gen)
    h[0, 1], h[2, width - 2] = float("inf"), -float("inf")
    ids, weights, logits = torch.empty(n, 2, dtype=torch.int32, device="cuda"), torch.empty(n, 2, device="cuda"), torch.empty(n, outs, device="cuda")
    ops.moe_router(h, w, None, ids, weights, logits, score="sigmoid")
    assert torch.equal(logits[0], torch.sign(w[:, 1]) * float("inf")) and torch.equal(logits[2], -torch.sign(w[:, width - 2]) * float("inf"))
    rest = [t for t in range(n) if t not in (0, 2)]
    assert bool(((logits[rest].double() - h[rest].double() @ w.double().T).abs() <= 1e-5 * width ** 0.5).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,width,top", [(1, 4, 1), (5, 1028, 3), (7, 1024, 4), (9, 132, 5), (3, 4096, 9), (6, 130, 3), (40, 64, 8), (33, 128, 9), (5, 124, 2)])
def test_combine(n, width, top, dtype):
    from vllm_cpp_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(n + width)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    y, h, add, weights = rnd(n * top, width), rnd(n, width + 4).to(dtype)[:, :width], rnd(n, width).to(dtype), rnd(n, top)
    pos = torch.randperm(n * top, device="cuda", generator=gen).to(torch.int32).view(n, top)
    pos[rnd(n, top) > 1.0] = -1
    rows = torch.where((pos >= 0)[..., None], y.double()[pos.clamp(min=0).long()], h.double()[:, None, :])
    for w, more in ((weights, add), (None, None), (weights, None)):
        out = torch.full((n, width), 9.0, dtype=dtype, device="cuda")
        ops.moe_combine(y, h, pos, w, out, more)
        want = (rows * (w.double()[..., None] if w is not None else 1.0)).sum(1) + (more.double() if more is not None else 0.0)
        # top + 1 float32 additions of numbers up to 5, and the stored type's rounding
        assert bool(((out.double() - want).abs() <= 1e-5 * (1 + want.abs()) + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0.0)).all())


@pytest.mark.parametrize("score", ["softmax", "sigmoid"])
@pytest.mark.parametrize("groups,keep", [(1, 1), (4, 2)])
def test_choice_where_scores_are_no_numbers(score, groups, keep):
    """Rows whose logits are infinite or no numbers, and corrections of -infinity: every choice is another output, the lowest ones among those without a
    score, and a row's neighbours are not touched."""
    from vllm_cpp_b200.csrc import ops
    n, width, outs, top = 9, 64, 40, 6
    gen = torch.Generator(device="cuda").manual_seed(groups)
    h, w = torch.randn(n, width, device="cuda", generator=gen), torch.randn(outs, width, device="cuda", generator=gen)
    plain = h.clone()
    h[1], h[3, 5], h[5, 7], h[7, 0] = float("nan"), float("nan"), float("inf"), -float("inf")
    never = torch.zeros(outs, device="cuda")
    never[4:] = -float("inf")                                             # four outputs are left for six choices
    for correction in (None, never):
        got = []
        for rows in (h, plain):
            ids, weights = torch.full((n, top), -7, dtype=torch.int32, device="cuda"), torch.empty(n, top, device="cuda")
            ops.moe_router(rows, w, correction, ids, weights, torch.empty(n, outs, device="cuda"), score=score, groups=groups, keep_groups=keep, group_top=2)
            assert int(ids.min()) >= 0 and int(ids.max()) < outs
            assert all(len(set(r)) == top for r in ids.tolist())
            got.append((ids, weights))
        clean = [0, 2, 4, 6, 8]
        assert torch.equal(got[0][0][clean], got[1][0][clean]) and torch.equal(got[0][1][clean], got[1][1][clean])
        if groups == 1:
            assert got[0][0][1].tolist() == list(range(top))              # nothing has a score
        if correction is not None and groups == 1:
            assert all(set(range(4)) <= set(r) for r in got[1][0].tolist())
