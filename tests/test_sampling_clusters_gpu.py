"""Sampling by clusters of CTAs: rows on both sides of the sizes at which a row gets one, four or eight CTAs, with ties, flat rows,
infinities, and rows that 16-byte reads do not fit, against 64 bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

VOCABS = [5, 16383, 16384, 65535, 65536, 100003]


def _rows(vocab, seed):
    rng = np.random.default_rng(seed)
    x = (2 * rng.standard_normal((8, vocab + 3))).astype(np.float32)
    x[1] = 1.5                                                          # all equal: the order is the ids'
    x[2] = np.round(x[2] * 2) / 2                                       # many ties
    x[3, :vocab] = -np.inf
    x[3, [0, vocab // 2, vocab - 1]] = [0.0, 1.0, 1.0]                  # three ids, the last of every run among them
    x[4] *= 0.001
    x[5, vocab - 1] = 30.0
    x[6] *= 6
    return x


def _order(x, temp):
    """ids by falling weight, the lower id first among equals, and their weights in float64 (those of the float32 weights)."""
    v = x if temp == 1.0 else (x * (np.float32(1.0) / np.float32(temp))).astype(np.float32)
    e = np.exp((v - v.max()).astype(np.float64)).astype(np.float32)
    ids = np.lexsort((np.arange(len(e)), -e))
    return ids, e[ids].astype(np.float64)


@pytest.mark.parametrize("vocab", VOCABS)
def test_filtered_rows(vocab):
    """The kept set is what sorting would keep, and the draw the id whose interval of the kept ids' running sum holds u.  The
    weights are float32 numbers of either side's exponential (relative error 2^-22), so the bounds may lie that far apart."""
    from vllm_cpp_b200.csrc import ops
    buf = torch.from_numpy(_rows(vocab, vocab)).cuda()
    logits, x = buf[:, :vocab], _rows(vocab, vocab)[:, :vocab]
    temps = np.array([1.0, 1.0, 0.7, 1.0, 1.3, 0.9, 0.8, 1.0], dtype=np.float32)
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    out = torch.empty(8, dtype=torch.int32, device="cuda")
    for k, p, u in [(-1, 0.9, 0.3), (1, 1.0, 0.99), (50, 1.0, 0.7), (3, 0.4, 0.0), (700, 0.95, 0.9999999), (-1, 0.05, 0.5), (vocab - 1, 0.999, 0.2)]:
        ks, ps = np.full(8, max(k, -1) or -1, dtype=np.int32), np.full(8, p, dtype=np.float32)
        us = np.full(8, u, dtype=np.float32)
        got = []
        for _ in range(2):
            out.fill_(-7)
            ops.sample_filtered(logits, dev(temps), dev(us), dev(ps), dev(ks), out)
            got.append(out.cpu().numpy().copy())
        assert (got[0] == got[1]).all()
        for r in range(8):
            ids, w = _order(x[r], float(temps[r]))
            n = min(vocab, int(ks[r])) if ks[r] > 0 else vocab
            c = np.cumsum(w[:n])
            if p < 1.0:
                n = min(n, int(np.searchsorted(c, float(np.float32(p)) * c[-1], side="left")) + 1)
            at = int(np.where(ids == got[0][r])[0][0])
            # ids whose weights differ by a few units in the last place may stand in another order under the other exponential
            near = np.count_nonzero((np.abs(w - w[at]) <= 2.0 ** -21 * w[at]) & (x[r][ids] != x[r][ids[at]]))
            slack = 2.0 ** -20 * c[-1] + near * w[at]
            below = c[min(at, len(c)) - 1] if at else 0.0
            kept = c[n - 1]
            assert at < n + near or (p < 1.0 and c[min(at, len(c)) - 1] <= float(np.float32(p)) * c[-1] + slack), (vocab, k, p, u, r)
            assert below - slack <= float(np.float32(u)) * kept <= (c[at] if at < len(c) else c[-1]) + slack, (vocab, k, p, u, r, at, n)


@pytest.mark.parametrize("vocab", VOCABS)
def test_whole_rows(vocab):
    from vllm_cpp_b200.csrc import ops
    x = _rows(vocab, vocab)[:, :vocab]
    logits = torch.from_numpy(_rows(vocab, vocab)).cuda()[:, :vocab]
    out = torch.empty(8, dtype=torch.int32, device="cuda")
    dev = lambda a: torch.from_numpy(np.asarray(a, dtype=np.float32)).cuda()  # noqa: E731
    ops.sample(logits, dev(np.zeros(8)), dev(np.zeros(8)), out)
    assert out.cpu().numpy().tolist() == [int(np.argmax(r)) for r in x]
    for u in (0.0, 0.123, 0.5, 0.875, 0.99999994):
        out.fill_(-7)
        ops.sample(logits, dev(np.ones(8)), dev(np.full(8, u)), out)
        for r, g in enumerate(out.cpu().numpy()):
            e = np.exp(x[r].astype(np.float64) - x[r].max())
            c = np.cumsum(e)
            # sums of up to 8 x 16 slabs of float32 sums
            assert 0 <= g < vocab and (c[g - 1] if g else 0.0) - 2e-5 * c[-1] <= u * c[-1] <= c[g] + 2e-5 * c[-1], (vocab, u, r, g)
            assert e[g] > 0


# slabs with ids: 3 and 15 of a short row's 32, 14, 15 and all of a run's 16
@pytest.mark.parametrize("vocab", [384, 1800, 100352, 152064, 65536])
def test_every_draw_has_an_id(vocab):
    """The largest uniform number that 24 bits give: the draw lies within the last place of the row's sum, in whichever order that was added up."""
    from vllm_cpp_b200.csrc import ops
    rows = 512
    gen = torch.Generator(device="cuda").manual_seed(vocab)
    ones, u = torch.ones(rows, device="cuda"), torch.full((rows,), 1.0 - 2.0 ** -24, device="cuda")
    for _ in range(4):
        logits = torch.randn(rows, vocab, device="cuda", generator=gen)
        out = torch.full((rows,), -7, dtype=torch.int32, device="cuda")
        ops.sample(logits, ones, u, out)
        assert int(out.min()) >= 0 and int(out.max()) < vocab
        # what lies behind the id drawn is at most the roundings of the sums (as in test_whole_rows)
        e = torch.softmax(logits.double(), dim=1)
        behind = 1.0 - e.cumsum(1).gather(1, out.long()[:, None])
        assert bool((behind <= 2e-5).all())


@pytest.mark.parametrize("vocab", [5000, 20000, 70001])
@pytest.mark.parametrize("listed", [1, 4095, 4096, 4097])
def test_ids_at_the_lists_end(vocab, listed):
    """`listed` ids of one weight stand in the bin that top-k and top-p fall into: the list takes 4,096, one more goes to the search by digits.  Equal
    weights stand in the order of their ids, so the draw is known: of the k kept ones, or of those that weigh p times all (the others e^-60 of these)."""
    from vllm_cpp_b200.csrc import ops
    rng = np.random.default_rng(vocab + listed)
    x = np.full((3, vocab), -50.0, dtype=np.float32)
    for r in x:
        r[rng.permutation(vocab)[:listed]] = 1.3
    dev = lambda a, t: torch.from_numpy(np.asarray(a, dtype=t)).cuda()  # noqa: E731
    k = min(10, listed)
    for u in (0.0, 0.55, 1.0 - 2.0 ** -24):
        out = torch.full((3,), -7, dtype=torch.int32, device="cuda")
        ops.sample_filtered(dev(x, np.float32), dev([0.7, 0.7, 0.85], np.float32), dev([u] * 3, np.float32), dev([1.0, 0.5, 0.5], np.float32),
                            dev([k, -1, k], np.int32), out)
        kept = (k, (listed + 1) // 2, (k + 1) // 2)
        assert out.tolist() == [int(np.flatnonzero(r > 0)[min(int(u * n), n - 1)]) for r, n in zip(x, kept)], (u, kept)


@pytest.mark.parametrize("vocab", [300, 5000, 20000, 152064])
def test_rows_that_are_no_numbers(vocab):
    """Infinities and what is no number: a row gives an id of the vocabulary; the one +infinity is taken, -infinity and what is no number are not where
    another id has weight."""
    from vllm_cpp_b200.csrc import ops
    x = np.random.default_rng(vocab).standard_normal((7, vocab)).astype(np.float32)
    x[0] = np.nan
    x[1] = -np.inf
    x[2, vocab // 3] = np.inf
    x[3, 1::2] = np.nan
    x[4, ::2] = -np.inf
    x[5] = np.finfo(np.float32).min
    x[6, [1, vocab - 2]] = np.inf
    dev = lambda a, t: torch.from_numpy(np.asarray(a, dtype=t)).cuda()  # noqa: E731
    logits, u = dev(x, np.float32), dev([0.37] * 7, np.float32)
    for temp in (1.0, 0.6):
        for p, k in ((0.9, -1), (1.0, 40), (0.8, 7), (1.0 - 2.0 ** -24, vocab - 1)):
            out = torch.full((7,), -7, dtype=torch.int32, device="cuda")
            ops.sample_all(logits, dev([temp] * 7, np.float32), u, dev([p] * 7, np.float32), dev([k] * 7, np.int32), out)
            got = out.tolist()
            assert all(0 <= g < vocab for g in got), (temp, p, k, got)
            assert got[2] == vocab // 3 and got[3] % 2 == 0 and got[4] % 2 == 1 and got[6] in (1, vocab - 2), (temp, p, k, got)
        ops.sample(logits, dev([temp] * 7, np.float32), u, out.fill_(-7))
        assert all(0 <= g < vocab for g in out.tolist())
        ops.sample(logits, dev([0.0] * 7, np.float32), u, out.fill_(-7))
        assert all(0 <= g < vocab for g in out.tolist()) and out.tolist()[2] == vocab // 3 and out.tolist()[6] == 1


@pytest.mark.parametrize("vocab", [9001, 20000, 70001, 152064])
def test_rows_do_not_depend_on_the_batch(vocab):
    """How many CTAs share a row depends on the batch, its draw does not: 1 to 300 rows, which take eight CTAs to one."""
    from vllm_cpp_b200.csrc import ops
    gen = torch.Generator(device="cuda").manual_seed(vocab)
    logits = 2 * torch.randn(300, vocab, device="cuda", generator=gen)
    logits[5::7] *= 0.01                                                # flat rows: the search by digits
    u = torch.rand(300, device="cuda", generator=gen)
    temp, p, k = torch.full((300,), 0.8, device="cuda"), torch.ones(300, device="cuda"), torch.full((300,), -1, dtype=torch.int32, device="cuda")
    temp[::5] = 0.0
    p[1::3], k[2::4] = 0.9, 40
    whole = None
    for n in (300, 140, 70, 60, 40, 25, 20, 9, 1):
        drawn, mixed = torch.full((n,), -7, dtype=torch.int32, device="cuda"), torch.full((n,), -7, dtype=torch.int32, device="cuda")
        ops.sample(logits[:n], temp[:n], u[:n], drawn)
        ops.sample_all(logits[:n], temp[:n], u[:n], p[:n], k[:n], mixed)
        whole = whole or (drawn, mixed)
        assert torch.equal(drawn, whole[0][:n]) and torch.equal(mixed, whole[1][:n]), n
        assert bool(((mixed >= 0) & (mixed < vocab)).all())


@pytest.mark.parametrize("vocab", [997, 70001])
def test_all_rows_in_one_launch(vocab):
    """Greedy, plain and filtered rows side by side: what the two launches leave."""
    from vllm_cpp_b200.csrc import ops
    logits = torch.from_numpy(_rows(vocab, 3)).cuda()[:, :vocab]
    dev = lambda a, t: torch.from_numpy(np.asarray(a, dtype=t)).cuda()  # noqa: E731
    temp, u = dev([0, 1, 0.7, 1, 0.9, 0, 1.2, 0.5], np.float32), dev([0.5, 0.25, 0.9, 0.1, 0.6, 0.3, 0.7, 0.999], np.float32)
    p, k = dev([1, 0.9, 1, 1, 0.5, 0.5, 1, 0.99], np.float32), dev([-1, -1, 40, -1, 7, 3, -1, 5000], np.int32)
    one, two = torch.full((8,), -7, dtype=torch.int32, device="cuda"), torch.full((8,), -7, dtype=torch.int32, device="cuda")
    ops.sample_all(logits, temp, u, p, k, one)
    ops.sample(logits, temp, u, two)
    ops.sample_filtered(logits, temp, u, p, k, two)
    assert torch.equal(one, two) and bool((one >= 0).all())
