"""Cluster sampler at its edges: vocabulary sizes around the slice and cluster limits, unaligned rows, cuts that fall into
long ties, top-k above and below the gathered list, degenerate rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(logits, temperature, top_k, top_p, min_p, u, got):
    """The drawn token's interval of the float64 CDF holds the target, up to the error of f32 sums of V terms."""
    V = logits.shape[1]
    # a probability is off by a few ulp, a sum of V of them (partial sums of at most V / 512 + 512 in a row) by less than this
    eps = 2.0 ** -23 * (V / 512 + 512)
    for r, tok in enumerate(got.tolist()):
        T = float(temperature[r])
        if T <= 0:
            assert tok == int(logits[r].argmax()), r
            continue
        x = logits[r].double() / T
        k = int(top_k[r])
        if 0 < k < V:
            # the scaled logits are f32 in the kernel: neighbours of the cut may tie there
            cut = torch.topk(x, k).values[-1]
            x = torch.where(x < cut - 4e-7 * cut.abs(), torch.full_like(x, -float("inf")), x)
        p = torch.softmax(x, 0)
        keep = torch.ones_like(p, dtype=torch.bool)
        unsure = 0.0               # mass that lies so near the nucleus cut that f32 sums do not settle its side
        tp = float(top_p[r])
        if 0 < tp < 1:
            sp = torch.sort(p, descending=True).values
            cum = torch.cumsum(sp, 0)
            lo = sp[min(int(torch.searchsorted(cum, tp + eps)), V - 1)] * (1 - 1e-5)
            hi = sp[min(int(torch.searchsorted(cum, max(tp - eps, 0.0))), V - 1)]
            assert float(p[tok]) >= float(lo), (r, "outside the nucleus")
            keep = p >= hi * (1 - 1e-5)
            unsure = float(p[(p >= lo) & ~keep].sum())
        if float(min_p[r]) > 0:
            assert float(p[tok]) >= float(min_p[r]) * float(p.max()) * (1 - 1e-5), r
            keep &= p >= float(min_p[r]) * p.max()
        q = torch.where(keep, p, torch.zeros_like(p))
        cdf = torch.cumsum(q, 0) / q.sum()
        edge = eps + unsure / float(q.sum()) + 1e-5
        lo, hi = float(cdf[tok - 1]) if tok else 0.0, float(cdf[tok])
        assert lo - edge <= float(u[r]) <= hi + edge, (r, tok, lo, hi, float(u[r]))


@pytest.mark.parametrize("V,ld", [(1, 1), (2, 2), (33, 35), (1023, 1023), (19456, 19456), (19457, 19460), (40001, 40001),
                                  (155648, 155648), (155649, 155649), (360449, 360449)])
def test_sampler_sizes(V, ld):
    from plow_b200.ops import sampler
    g = torch.Generator(device="cuda").manual_seed(V)
    rows = 14
    logits = (torch.randn(rows, ld, device="cuda", generator=g) * 2.5)[:, :V]
    temperature = torch.tensor([0.0, 1.0, 0.7, 1.3, 1.0, 1.0, 0.5, 1.0, 2.0, 1.0, 1.0, 0.9, 1.0, 0.6], device="cuda")
    top_k = torch.tensor([0, 0, 50, 0, 1, 0, 2048, 2049, 0, max(1, V - 1), 5, 40, V, 0], dtype=torch.int32, device="cuda")
    top_p = torch.tensor([1.0, 1.0, 1.0, 0.9, 1.0, 0.5, 0.8, 0.95, 0.9999, 0.1, 1.0, 0.7, 0.0, 0.99], device="cuda")
    min_p = torch.tensor([0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.05, 0.0, 0.2, 0.01, 0.0, 0.0], device="cuda")
    for _ in range(3):
        u = torch.rand(rows, device="cuda", generator=g)
        got = sampler.sample(logits, temperature, top_k, top_p, min_p, u=u)
        assert int(got.min()) >= 0 and int(got.max()) < V
        _check(logits, temperature, top_k, top_p, min_p, u, got)


# CTAs per row 8 to 1, all resident at once or not; greedy rows then are one CTA's
@pytest.mark.parametrize("rows,V,ld", [(37, 16384, 16384), (64, 9001, 9003), (74, 8192, 8192), (200, 4095, 4096), (310, 20003, 20005), (40, 150001, 150001)])
def test_sampler_many_rows(rows, V, ld):
    from plow_b200.ops import sampler
    g = torch.Generator(device="cuda").manual_seed(V)
    logits = (torch.randn(rows, ld, device="cuda", generator=g) * 2)[:, :V]
    logits[:, V // 3] = logits[:, V - 1]                     # ties: the lowest index
    r = torch.arange(rows, device="cuda")
    top = torch.arange(0, rows, 4, device="cuda")
    logits[top, V - 1] = logits[top, V // 3] = 30.0
    temperature = torch.where(r % 2 == 0, 0.0, 0.8)
    top_k = torch.where(r % 3 == 0, 40, 0).int()
    top_p = torch.where(r % 5 == 0, 0.9, 1.0)
    u = torch.rand(rows, device="cuda", generator=g)
    got = sampler.sample(logits, temperature, top_k, top_p, torch.zeros(rows, device="cuda"), u=u)
    assert (got[top].long() == V // 3).all()
    _check(logits, temperature, top_k, top_p, torch.zeros(rows), u, got)


@pytest.mark.parametrize("V", [3, 700, 9000, 60000, 361000])
def test_sampler_nonfinite_rows(V):
    """A NaN or +inf among the scaled logits leaves no probabilities: no token, whatever the filters.  Greedy rows order by value."""
    from plow_b200.ops import sampler
    g = torch.Generator(device="cuda").manual_seed(V)
    rows = torch.randn(7, V, device="cuda", generator=g)
    for r, (at, v) in enumerate([(0, "nan"), (V // 2, "nan"), (V - 1, "-nan"), (V - 1, "inf"), (1, "-inf"), (0, "nan"), (2, "inf")]):
        rows[r, at] = float(v)
    temp = torch.tensor([1.0, 0.7, 1.0, 1.0, 1.0, 0.0, 0.0], device="cuda")
    for k, p, m in ((0, 1.0, 0.0), (1, 1.0, 0.0), (50, 0.9, 0.1), (3000, 1.0, 0.0), (0, 0.5, 0.0)):
        kk = torch.full((7,), k, dtype=torch.int32, device="cuda")
        got = sampler.sample(rows, temp, kk, torch.full_like(temp, p), torch.full_like(temp, m), u=torch.full_like(temp, 0.4)).tolist()
        assert got[:4] == [-1] * 4, (k, p)
        assert 0 <= got[4] < V and got[4] != 1
        assert got[5] == 0 and got[6] == 2


@pytest.mark.parametrize("V", [500, 9000, 60000])
def test_sampler_ties_and_degenerate_rows(V):
    """All logits equal, two values, one live token, masked rows: every element at a cut value is kept."""
    from plow_b200.ops import sampler
    inf = float("inf")
    rows = torch.full((6, V), 0.25, device="cuda")
    rows[1, V // 2:] = -0.75                       # two values
    rows[2] = -inf                                 # one live token
    rows[2, V - 1] = 1.0
    rows[3] = -inf                                 # nothing to draw: no token
    rows[4, ::2] = -inf                            # half masked
    rows[5, 3] = 80.0                              # everything else underflows
    u = torch.full((6,), 0.5, device="cuda")
    one = torch.ones(6, device="cuda")
    for k, p in ((0, 1.0), (7, 1.0), (V // 4, 0.4), (0, 0.3)):
        got = sampler.sample(rows, one, torch.full((6,), k, dtype=torch.int32, device="cuda"), one * p, one * 0, u=u).tolist()
        tol = 1 + V // 1000
        assert abs(got[0] - V // 2) <= tol                      # ties are kept: the cut removes nothing
        if k or p < 1:
            assert abs(got[1] - V // 4) <= tol                  # the lower value falls out of either filter
        assert got[2] == V - 1 and got[3] == -1 and got[5] == 3
        assert got[4] % 2 == 1 and abs(got[4] - V // 2) <= tol
