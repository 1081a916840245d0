"""The sampling kernel where its work is cut differently: one to eight CTAs per row, slices that end in
the middle of a thread's tokens, rows too long for shared memory, rows that put more tokens into the
threshold's interval than the candidate list holds, and rows with infinite logits."""
import numpy as np
import pytest
import torch

DEV = "cuda:0"


def expect(x, tau):
    """(p, s, threshold) in 64 bits."""
    x = x.astype(np.float64)
    e = np.exp(x - x.max())
    p = e / e.sum()
    with np.errstate(divide="ignore", invalid="ignore"):
        nl = -np.log(p)
        s = np.abs(nl - np.nansum(nl * p))
    order = np.argsort(s, kind="stable")
    cum = np.cumsum(p[order])
    at = int(np.searchsorted(cum, tau))
    return p, s, (s[order][at] if at < len(s) else np.inf)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,n,scale,tau,temp", [
    (1, 1, 1.0, 0.5, 1.0), (3, 31, 2.0, 0.9, 1.0), (2, 511, 1.0, 0.3, 0.7), (1, 513, 4.0, 0.95, 1.0),
    (1, 4095, 2.0, 0.8, 1.0), (1, 4096, 2.0, 0.8, 1.3), (5, 8191, 3.0, 0.6, 1.0), (40, 16385, 2.0, 0.9, 1.0),   # 1 to 8 CTAs
    (1, 50277, 2.0, 0.8, 1.0), (30, 50277, 2.0, 0.98, 0.5), (75, 50277, 5.0, 0.2, 1.0), (300, 25600, 1.0, 0.5, 1.0),
    (150, 25601, 1.0, 0.5, 1.0), (1, 65536, 3.0, 0.99, 1.0),
    (2, 50277, 0.02, 0.5, 1.0), (150, 50277, 0.05, 0.9, 1.0),      # nearly flat: more candidates than the list holds
    (1, 204800, 2.0, 0.8, 1.0), (2, 204801, 2.0, 0.8, 1.0),        # the longest rows held in shared memory, and beyond
])
def test_kept_tokens_and_draws_match_64_bit_arithmetic(rows, n, scale, tau, temp):
    from rwkvstic_b200 import ops
    rng = np.random.default_rng(rows * 1000003 + n)
    x = (rng.standard_normal((rows, n)) * scale).astype(np.float32)
    u = rng.random(rows).astype(np.float32)
    tok, probs = ops.sample_typical(torch.from_numpy(x).to(DEV), temp, tau, u=torch.from_numpy(u).to(DEV), return_probs=True)
    plain = ops.sample_typical(torch.from_numpy(x).to(DEV), temp, tau, u=torch.from_numpy(u).to(DEV))
    assert torch.equal(tok, plain)
    tok, probs = tok.cpu().numpy(), probs.cpu().numpy()
    for r in sorted({*range(min(rows, 6)), *range(0, rows, 37), *range(max(0, rows - 4), rows)}):      # every wave of clusters
        p, s, t = expect(x[r], tau)
        # fp32 s = |(log Z - (l - max)) - entropy|: five roundings, each of a value of at most
        # max - l + log Z (+ 1 for the fp64 sums of fp32 terms behind log Z and the entropy)
        xd = x[r].astype(np.float64)
        eps = 5 * 2.0 ** -24 * ((xd.max() - xd) + np.log(np.exp(xd - xd.max()).sum()) + 1.0)
        kept = probs[r] > 0
        assert not kept[s > t + eps].any(), f"row {r}"
        assert kept[(s < t - eps) & (p > 1e-30)].all(), f"row {r}"
        want = p ** (1.0 / temp)
        assert np.allclose(probs[r][kept], want[kept], rtol=2e-5, atol=0)
        w = probs[r].astype(np.float64)
        cum = np.cumsum(w)
        target = float(u[r]) * cum[-1]
        k = int(tok[r])
        assert w[k] > 0 and cum[k] - w[k] - 1e-9 * cum[-1] <= target <= cum[k] + 1e-9 * cum[-1], f"row {r}"


@pytest.mark.gpu
def test_infinite_and_equal_logits():
    from rwkvstic_b200 import ops
    x = torch.full((4, 50277), float("-inf"))
    x[0, 31337] = 1.0                              # one possible token
    x[1, 7], x[1, 50276] = 0.0, 0.0                # two equal ones
    x[2] = 3.0                                     # all equal: every token is the threshold's
    x[3, 1000:1100] = torch.linspace(-1, 1, 100)
    u = torch.tensor([0.9, 0.9, 0.5, 0.0])
    tok, probs = ops.sample_typical(x.to(DEV), 1.0, 0.9, u=u.to(DEV), return_probs=True)
    tok, kept = tok.tolist(), (probs > 0).cpu()
    assert tok[0] == 31337 and tok[1] == 50276 and abs(tok[2] - 25138) <= 1 and 1000 <= tok[3] < 1100
    assert kept.sum(1).tolist()[:3] == [1, 2, 50277] and not kept[3, :1000].any() and not kept[3, 1100:].any()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2048, 4096, 16384, 65536])
def test_small_terms_of_the_softmax_sum_are_not_lost(n):
    """One token in four at the maximum, the others e^-17.5 of it: together they are 7.5e-8 of Z, more than fp32
    resolves, but each is less than half a unit of the last place of a 1.  The probability of the likely tokens is
    1 / Z, so it shows whether Z kept them."""
    from rwkvstic_b200 import ops
    x = torch.full((1, n), -17.5)
    x[0].view(-1, 512)[::4] = 0.0
    z = np.exp(x[0].double().numpy()).sum()
    tok, probs = ops.sample_typical(x.to(DEV), 1.0, 0.9, u=torch.tensor([0.5], device=DEV), return_probs=True)
    assert float(probs.max()) == np.float32(1.0 / z)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [24576, 50277, 31])
def test_a_row_gives_the_same_alone_and_beside_others(n):
    """A call of few rows gives a row more CTAs than a call of many; its probabilities and its draw are the same bits.
    The last row has one token in four at the maximum and the rest e^-17.5 of it: sums that depend on how the row is
    cut show there."""
    from rwkvstic_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(n)
    x = torch.randn(300, n, generator=g, device=DEV) * 2.0
    x[-1] = torch.where(torch.arange(n, device=DEV) // 512 % 4 == 0, 0.0, -17.5)
    u = torch.rand(300, generator=g, device=DEV)
    for temp, tau in [(1.0, 0.8), (0.7, 0.95)]:
        tok, probs = ops.sample_typical(x, temp, tau, u=u, return_probs=True)
        for rows in (1, 7, 30, 75):                  # eight, four, two CTAs a row at 50277 tokens
            for first in (0, 111, 300 - rows):
                at = slice(first, first + rows)
                t, p = ops.sample_typical(x[at].contiguous(), temp, tau, u=u[at].contiguous(), return_probs=True)
                assert torch.equal(p, probs[at]) and torch.equal(t, tok[at])
