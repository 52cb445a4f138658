"""The walk of the gated delta rule with four, two and one column a thread (many, some and few heads of requests), key channels that lanes do not
fill and value channels that a CTA does not, unequal portions; and the gates' tiles of 64 tokens by 64 channels at their edges; against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# requests, heads, qk heads: with 148 SMs 4 * (tokens / 21) * heads * (value channels / columns a CTA) is from 1,480 on for four columns, from 1,184 on for two, else
# one, as for keys of up to 32 channels; two as well for keys beyond 256, and (the last) for a prompt beside many single tokens
@pytest.mark.parametrize("reqs,H,G,dk,dv", [(33, 16, 8, 30, 40), (33, 16, 16, 128, 70), (33, 12, 4, 130, 36), (12, 16, 4, 30, 40), (40, 10, 5, 64, 32), (12, 8, 8, 64, 70),
                                            (3, 6, 3, 128, 40), (2, 4, 1, 36, 20), (2, 3, 3, 300, 70), (120, 8, 8, 300, 40), (-7, 8, 4, 40, 36)])
def test_gated_delta_walk(reqs, H, G, dk, dv):
    from vllm_cpp_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(reqs + dk)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    lens = [1 + (7 * r) % 19 if reqs > 0 else 1 for r in range(abs(reqs))]
    reqs = len(lens)
    lens[0] = 21
    n = sum(lens)
    start = [0]
    for x in lens:
        start.append(start[-1] + x)
    q, k, v = rnd(n, G * dk), rnd(n, G * dk), rnd(n, H * dv)
    beta, dec, a_log, dt = rnd(n, H), rnd(n, H * dk), 0.1 * rnd(H), rnd(H * dk)
    slots = torch.randperm(reqs + 2, device="cuda", generator=gen)[:reqs].to(torch.int32)
    state = rnd(reqs + 2, H, dk, dv)
    S0 = state.double()
    out = torch.full((n, H * dv), 9.0, device="cuda")
    ops.gated_delta_scan(q, k, v, beta, dec, a_log, dt, state, out, torch.tensor(start, dtype=torch.int32, device="cuda"), slots, reqs, num_heads=H,
                         num_qk_heads=G, q_scale=dk ** -0.5, unit_eps=1e-6, max_q_len=max(lens))
    unit = lambda x: x / (x.square().sum(-1, keepdim=True) + 1e-6).sqrt()  # noqa: E731
    heads = lambda x: unit(x.double().view(n, G, dk)).repeat_interleave(H // G, dim=1)  # noqa: E731
    qd, kd, vd = heads(q) * dk ** -0.5, heads(k), v.double().view(n, H, dv)
    g = torch.exp(-torch.exp(a_log.double())[:, None] * torch.nn.functional.softplus(dec.double() + dt.double()).view(n, H, dk))
    b = torch.sigmoid(beta.double())
    want, S = torch.zeros(n, H, dv, dtype=torch.float64, device="cuda"), S0[slots.long()].clone()
    for t in range(max(lens)):
        live = torch.tensor([r for r in range(reqs) if t < lens[r]], device="cuda")
        at = torch.tensor([start[r] + t for r in range(reqs) if t < lens[r]], device="cuda")
        s = g[at][..., None] * S[live]
        u = b[at][..., None] * (vd[at] - torch.einsum("rhkv,rhk->rhv", s, kd[at]))
        s = s + kd[at][..., None] * u[..., None, :]
        S[live] = s
        want[at] = torch.einsum("rhkv,rhk->rhv", s, qd[at])
    # float32 sums of dk products per token, carried over at most 21 tokens of a contracting state
    assert bool(((out.double().view_as(want) - want).abs() <= 2e-5 * want.abs().max()).all())
    assert bool(((state.double()[slots.long()] - S).abs() <= 2e-5 * S.abs().max()).all())
    rest = [i for i in range(reqs + 2) if i not in slots.tolist()]
    assert bool((state.double()[rest] == S0[rest]).all())


# of 148 SMs: one column a thread alone, two or four beside others; 8, 16 and 32 lanes a column, and keys whose last lanes are padding
@pytest.mark.parametrize("H,G,dk,dv", [(8, 4, 64, 40), (8, 4, 50, 24), (16, 8, 128, 64), (8, 8, 130, 36), (6, 3, 300, 64), (8, 4, 30, 40)])
def test_walk_does_not_depend_on_the_step(H, G, dk, dv):
    """A request's outputs and state are the same bits alone and beside 1, 3, 11 and 80 others."""
    from vllm_cpp_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(dk)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    lens = [23] + [17, 9, 23, 8, 12] * 16
    n = sum(lens)
    q, k, v = rnd(n, G * dk), rnd(n, G * dk), rnd(n, H * dv)
    beta, dec, a_log, dt, first = rnd(n, H), rnd(n, H * dk), 0.1 * rnd(H), rnd(H * dk), rnd(len(lens), H, dk, dv)
    seen = None
    for reqs in (1, 2, 4, 12, len(lens)):
        m = sum(lens[:reqs])
        start = torch.tensor([sum(lens[:r]) for r in range(reqs + 1)], dtype=torch.int32, device="cuda")
        state, out = first[:reqs].clone(), torch.full((m, H * dv), 9.0, device="cuda")
        ops.gated_delta_scan(q[:m], k[:m], v[:m], beta[:m], dec[:m], a_log, dt, state, out, start, torch.arange(reqs, dtype=torch.int32, device="cuda"),
                             reqs, num_heads=H, num_qk_heads=G, q_scale=dk ** -0.5, unit_eps=1e-6, max_q_len=23)
        got = (out[:23].clone(), state[0].clone())
        assert seen is None or (torch.equal(seen[0], got[0]) and torch.equal(seen[1], got[1])), reqs
        seen = seen or got


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,B,bs", [(33, 3, 8), (64, 2, 64), (65, 2, 72), (130, 1, 136), (100, 3, 20), (70, 2, 33)])
def test_gates(dtype, n, B, bs):
    from vllm_cpp_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(n + bs)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    W = B * bs
    wide = rnd(n, W + 4)
    u, wa, wi, ba, bi, lam = wide[:, :W], (rnd(B, bs, bs) / bs ** 0.5).to(dtype), (rnd(B, bs, bs) / bs ** 0.5).to(dtype), rnd(W), rnd(W), rnd(W)
    decay, drive = torch.full((n, W), 9.0, device="cuda"), torch.full((n, W), 9.0, device="cuda")
    ops.gate_blocks(u, wa, wi, ba, bi, lam, decay, drive, 8.0)
    ub = u.double().reshape(n, B, bs)
    r, i = (torch.sigmoid(torch.einsum("nbk,bok->nbo", ub, w.double()).reshape(n, W) + bias.double()) for w, bias in ((wa, ba), (wi, bi)))
    d = torch.exp(-8.0 * r * torch.nn.functional.softplus(lam.double()))
    f = torch.sqrt(1 - d * d) * i * u.double()
    # float32 sums of bs products enter an exponent of at most 8 softplus(lam); sqrt(1 - d^2) loses 2^-24 / (2 sqrt(1 - d^2)) near d = 1
    assert bool(((decay.double() - d).abs() <= 3e-5).all())
    assert bool(((drive.double() - f).abs() <= 3e-5 * (1 + f.abs()) + 1e-6 * u.double().abs() / torch.sqrt(1 - d * d)).all())
