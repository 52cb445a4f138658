"""The 32-bit path's product and attention at the edges of their tiles and of the rules that pick a kernel, against 64 bits."""
import numpy as np
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


def _attention_case(seed, lens, news, nh, nkv, d, page, planes, dtype):
    """Requests that hold ``lens`` tokens of which the last ``news`` ask; pages in a shuffled order."""
    from vllm_cpp_b200.cache.manager import cdiv
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    width = max(cdiv(n, page) for n in lens)
    pages = sum(cdiv(n, page) for n in lens) + 1
    order = rng.permutation(pages).tolist()
    bt = np.full((len(lens), width), -1, dtype=np.int32)
    rows = {}
    cache = torch.zeros(pages, planes, nkv, page * d, dtype=dtype, device="cuda")
    esize = 2 if dtype == torch.bfloat16 else 4

    def place(slot):
        e = np.arange(d)
        if (d * esize) % 128:
            return slot * d + e
        per_plane, per_chunk = 128 // esize, 16 // esize
        plane, w = e // per_plane, e % per_plane
        return plane * page * per_plane + slot * per_plane + ((w // per_chunk) ^ (slot & 7)) * per_chunk + w % per_chunk

    for r, n in enumerate(lens):
        rows[r] = _rand(gen, n, planes, nkv, d).to(dtype)
        for b in range(cdiv(n, page)):
            bt[r, b] = order.pop()
        for j in range(n):
            cache[int(bt[r, j // page])][:, :, torch.from_numpy(place(j % page)).cuda()] = rows[r][j]
    pos = np.concatenate([np.arange(n - k, n) for n, k in zip(lens, news)]).astype(np.int32)
    req = np.concatenate([np.full(k, r) for r, k in enumerate(news)]).astype(np.int32)
    q = _rand(gen, len(pos), nh, d).to(dtype)
    return q, cache, rows, pos, req, bt


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,d,page,planes,window,sink", [
    (2, 2, 4, 16, 2, 0, False), (6, 3, 16, 16, 2, 0, False), (7, 1, 32, 16, 2, 5, False), (18, 2, 36, 32, 2, 0, True), (16, 2, 64, 16, 1, 0, True),
    (3, 3, 80, 48, 2, 70, False), (28, 4, 128, 16, 2, 0, False), (9, 1, 132, 16, 2, 0, True), (10, 2, 256, 16, 1, 33, False),
    (12, 4, 84, 16, 2, 0, True), (8, 2, 96, 16, 2, 0, False), (6, 3, 68, 16, 1, 40, True), (5, 5, 96, 16, 2, 0, False), (4, 1, 72, 32, 2, 0, False)])
def test_attention_rows(ops, dtype, nh, nkv, d, page, planes, window, sink):
    """Groups of one, two and more heads than a warp takes, rows of part of a warp's lanes and of two pieces a lane, keys shared among
    several warps (few tokens) and not (many), windows, sinks, one plane."""
    for lens, news in (([1, 130, 37], [1, 1, 1]), ([150, 61], [150, 40]), ([700], [700])):
        if lens == [700] and (d > 64 or dtype == torch.bfloat16):
            continue
        q, cache, rows, pos, req, bt = _attention_case(nh + d, lens, news, nh, nkv, d, page, planes, dtype)
        s = torch.randn(nh, device="cuda") if sink else None
        out = torch.empty(len(pos), nh * d, dtype=dtype, device="cuda")
        dev = lambda x: torch.from_numpy(x).cuda()  # noqa: E731
        ops.attention_simt(q.view(len(pos), -1), cache, out, dev(pos), dev(req), dev(bt), num_heads=nh, num_kv_heads=nkv, head_dim=d,
                           page_size=page, window=window, scale=d ** -0.5, planes=planes, sink=s)
        want = torch.empty(len(pos), nh, d, dtype=torch.float64, device="cuda")
        size = torch.empty(len(pos), nh, 1, dtype=torch.float64, device="cuda")
        for r in range(len(lens)):
            at = torch.from_numpy(np.nonzero(req == r)[0]).cuda()
            p, j = torch.from_numpy(pos[req == r]).cuda()[:, None], torch.arange(lens[r], device="cuda")[None, :]
            seen = (j <= p) & ((j > p - window) if window else (j >= 0))
            for h in range(nh):
                k, v = rows[r][:, 0, h // (nh // nkv)].double(), rows[r][:, -1, h // (nh // nkv)].double()
                x = (q[at, h].double() @ k.T * d ** -0.5).masked_fill(~seen, -np.inf)
                if sink:
                    x = torch.cat([x, s[h].double().expand(len(at), 1)], 1)
                w = torch.softmax(x, -1)[:, : lens[r]]
                want[at, h] = w @ v
                size[at, h] = w @ v.abs().amax(-1, keepdim=True)
        # float: scores of size 10 carry about 10 * 2^-22 into the weights; the stored result is rounded once more in bfloat16
        tol = 2e-5 if dtype == torch.float32 else 2e-5 + 2.0 ** -8
        assert bool(((out.view(len(pos), nh, d).double() - want).abs() <= tol * size.clamp(min=1.0)).all())
    ops.check_status()


@pytest.mark.parametrize("nh,nkv,d,window", [(4, 4, 32, 0), (14, 2, 128, 0), (8, 1, 256, 90), (3, 3, 80, 0), (8, 2, 96, 0)])
def test_attention_rows_do_not_depend_on_the_call(ops, nh, nkv, d, window):
    """A token alone (a warp per part of its keys) and among many (two and four warps, and one, walk the parts) has the same bits, with keys of one
    part, of a few and of eight."""
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    q, cache, rows, pos, req, bt = _attention_case(nh, [1, 63, 64, 65, 200, 530], [1] * 6, nh, nkv, d, 16, 2, torch.float32)

    def run(times):
        at = np.tile(np.arange(6), times)
        out = torch.empty(len(at), nh * d, device="cuda")
        ops.attention_simt(q.view(6, -1)[dev(at)].contiguous(), cache, out, dev(pos[at]), dev(req[at]), dev(bt), num_heads=nh, num_kv_heads=nkv, head_dim=d,
                           page_size=16, window=window, scale=d ** -0.5)
        return out.view(times, 6, -1)
    alone = run(1)
    for times in (20, 40, 90, 150, 400):
        assert torch.equal(run(times), alone.expand(times, -1, -1))
    ops.check_status()
