"""Two-tile flash kernel against the fp32 statement of the op: chunk and tile edges, several sequences in one call, rows that
are skipped, odd page counts, a second tile that is empty or partly filled, sliding windows, head ratios."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(q, kc, vc, pt, seq, pos, window):
    rows, nq, hd = q.shape
    nkv = kc.shape[2]
    out = torch.zeros(rows, nq * hd, dtype=torch.float32, device=q.device)
    for s in torch.unique(seq).tolist():
        sel = ((seq == s) & (pos >= 0)).nonzero()[:, 0]
        if not sel.numel():
            continue
        n = int(pos[sel].max()) + 1
        t = torch.arange(n, device=q.device)
        pages = pt[s][(t // 64)].long()
        k = kc[pages, t % 64].float().repeat_interleave(nq // nkv, 1)
        v = vc[pages, t % 64].float().repeat_interleave(nq // nkv, 1)
        sc = torch.einsum("rhd,nhd->hrn", q[sel].float(), k) / math.sqrt(hd)
        p = pos[sel].long()[:, None]
        hide = t[None] > p
        if window:
            hide |= t[None] <= p - window
        sc = sc.masked_fill(hide[None], float("-inf"))
        out[sel] = torch.einsum("hrn,nhd->rhd", sc.softmax(-1), v).reshape(len(sel), -1)
    return out


# (new rows, cached prefix) per sequence, idle rows before each
@pytest.mark.parametrize("runs,idle,nq,nkv,window", [
    ([(257, 0)], 0, 32, 8, 0), ([(300, 0), (1, 700), (65, 63)], 0, 32, 8, 0), ([(129, 1), (127, 64), (64, 128)], 3, 8, 8, 0),
    ([(1, 0), (2, 62), (31, 96), (33, 5), (256, 191)], 1, 16, 2, 0), ([(500, 77)], 0, 8, 1, 100), ([(330, 1000)], 0, 32, 8, 64),
    ([(1, 40 + 13 * i) for i in range(260)], 0, 32, 8, 0), ([(400, 3)], 0, 4, 4, 129),
    # more one-tile items than SMs: chunks of two tiles, cut from each run's own first row
    ([(650, 77)], 0, 32, 8, 100), ([(1300, 0)], 0, 16, 2, 0), ([(2500, 30), (31, 0)], 2, 8, 8, 0), ([(33, 100 + i) for i in range(21)], 1, 32, 8, 0),
    ([(15, 3 * i) for i in range(70)], 0, 32, 8, 0), ([(64, 0), (65, 10), (63, 90), (128, 1), (129, 0), (1, 700), (2, 5), (190, 40)], 1, 32, 8, 0)])
def test_prefill_attention(runs, idle, nq, nkv, window):
    from plow_b200.ops import gqa, native
    hd, dev = 128, "cuda"
    g = torch.Generator(device=dev).manual_seed(len(runs) * 7 + window)
    per = max((n + p + 63) // 64 for n, p in runs)
    n_pages = len(runs) * per + 1
    kc = torch.randn(n_pages, 64, nkv, hd, device=dev, generator=g).bfloat16()
    vc = torch.randn(n_pages, 64, nkv, hd, device=dev, generator=g).bfloat16()
    pt = torch.randperm(n_pages - 1, device=dev, generator=g).int()[: len(runs) * per].view(len(runs), per).contiguous() + 1
    seq, pos = [], []
    for i, (n, p) in enumerate(runs):
        seq += [i] * (idle + n)
        pos += [-1] * idle + list(range(p, p + n))
    rows = len(seq)
    seq = torch.tensor(seq, dtype=torch.int32, device=dev)
    pos = torch.tensor(pos, dtype=torch.int32, device=dev)
    q = (torch.randn(rows, nq, hd, device=dev, generator=g) * 1.5).bfloat16()
    ws = gqa.AttnWorkspace(rows, nq, nkv, hd, per * 64, dev, max_splits=1)
    out = torch.full((rows, nq * hd), 7.0, device=dev).bfloat16()
    gqa.attention(q, kc, vc, pt, seq, pos, ws, window=window, out=out)
    torch.cuda.synchronize()
    native.check_status()
    want = _ref(q, kc, vc, pt, seq, pos, window)
    live = pos >= 0
    # bf16 probabilities and result: 2^-9 each against values that average out to less than one
    rel = (out[live].float() - want[live]).norm() / want[live].norm()
    assert rel < 5e-3, rel
    assert (out[live].float() - want[live]).abs().max() < 4e-2
    assert (out[~live] == 7.0).all()


def test_prefill_attention_default_workspace():
    """The workspace's own split count at the served head ratio: whole and partly filled second tiles, more items than SMs."""
    from plow_b200.ops import gqa, native
    runs, nq, nkv, hd, dev = [(700, 0), (1, 900), (33, 64), (520, 300), (20, 5), (2, 1000), (150, 0)], 32, 8, 128, "cuda"
    g = torch.Generator(device=dev).manual_seed(9)
    per = max((n + p + 63) // 64 for n, p in runs)
    kc = torch.randn(len(runs) * per, 64, nkv, hd, device=dev, generator=g).bfloat16()
    vc = torch.randn(len(runs) * per, 64, nkv, hd, device=dev, generator=g).bfloat16()
    pt = torch.randperm(len(runs) * per, device=dev, generator=g).int().view(len(runs), per).contiguous()
    seq = torch.cat([torch.full((n,), i, dtype=torch.int32) for i, (n, _) in enumerate(runs)]).to(dev)
    pos = torch.cat([torch.arange(p, p + n, dtype=torch.int32) for n, p in runs]).to(dev)
    q = torch.randn(len(pos), nq, hd, device=dev, generator=g).bfloat16()
    ws = gqa.AttnWorkspace(len(pos), nq, nkv, hd, per * 64, dev)
    assert ws.max_splits == 1                 # this many rows fill the chip unsplit: the two-tile kernel
    out = gqa.attention(q, kc, vc, pt, seq, pos, ws)
    torch.cuda.synchronize()
    native.check_status()
    want = _ref(q, kc, vc, pt, seq, pos, 0)
    assert (out.float() - want).norm() / want.norm() < 5e-3


def test_prefill_attention_negative_scale():
    """A negative softmax scale attends to the smallest scores."""
    from plow_b200.ops import gqa
    nq, nkv, hd, rows, dev = 8, 2, 128, 300, "cuda"
    kc = torch.randn(6, 64, nkv, hd, device=dev).bfloat16()
    vc = torch.randn(6, 64, nkv, hd, device=dev).bfloat16()
    pt = torch.arange(1, 6, dtype=torch.int32, device=dev).view(1, 5)
    seq = torch.zeros(rows, dtype=torch.int32, device=dev)
    pos = torch.arange(rows, dtype=torch.int32, device=dev)
    q = torch.randn(rows, nq, hd, device=dev).bfloat16()
    ws = gqa.AttnWorkspace(rows, nq, nkv, hd, 320, dev, max_splits=1)
    a = gqa.attention(q, kc, vc, pt, seq, pos, ws, scale=-0.07)
    b = gqa.attention(-q, kc, vc, pt, seq, pos, ws, scale=0.07)
    assert torch.equal(a, b)


def _nonfinite_case():
    rows, nq, nkv, hd, dev = 300, 8, 2, 128, "cuda"
    g = torch.Generator(device=dev).manual_seed(5)
    kc = torch.randn(6, 64, nkv, hd, device=dev, generator=g).bfloat16()
    vc = torch.randn(6, 64, nkv, hd, device=dev, generator=g).bfloat16()
    pt = torch.tensor([[3, 1, 5, 2, 4]], dtype=torch.int32, device=dev)
    seq = torch.zeros(rows, dtype=torch.int32, device=dev)
    pos = torch.arange(rows, dtype=torch.int32, device=dev)
    q = torch.randn(rows, nq, hd, device=dev, generator=g).bfloat16()
    return q, kc, vc, pt, seq, pos


# the exponentials of a tile take two ways, chosen by the key's place in its group of sixteen
@pytest.mark.parametrize("t", list(range(32, 48)) + [0, 63, 64, 127, 129, 299])
@pytest.mark.parametrize("value", ["nan", "inf"])
def test_prefill_nonfinite_scores_reach_the_rows_that_see_them(t, value):
    """A NaN or infinite score makes NaN of every row that attends to its key and of no other."""
    from plow_b200.ops import gqa
    q, kc, vc, pt, seq, pos = _nonfinite_case()
    kc[pt[0, t // 64].long(), t % 64, :, 0] = float(value)
    q[:, :, 0] = q[:, :, 0].abs() + 0.5                       # the infinite product is positive
    ws = gqa.AttnWorkspace(len(pos), 8, 2, 128, 320, "cuda", max_splits=1)
    out = gqa.attention(q, kc, vc, pt, seq, pos, ws)
    assert out[t:].isnan().all()
    assert out[:t].isfinite().all()


def test_prefill_hidden_cells_weigh_nothing():
    """Cells behind the rows' end and before their windows hold the largest finite values."""
    from plow_b200.ops import gqa
    q, kc, vc, pt, seq, pos = _nonfinite_case()
    rows, window = len(pos), 40
    pos = pos + 15
    want = _ref(q, kc, vc, pt, seq, pos, window)
    flat = vc[pt[0].long()].view(320, 2, 128)
    t = torch.arange(320, device="cuda")
    flat[(t > int(pos[-1])) | (t <= int(pos[0]) - window)] = 3.3e38
    vc[pt[0].long()] = flat.view(5, 64, 2, 128)
    ws = gqa.AttnWorkspace(rows, 8, 2, 128, 320, "cuda", max_splits=1)
    out = gqa.attention(q, kc, vc, pt, seq, pos, ws, window=window)
    assert (out.float() - want).norm() / want.norm() < 5e-3


@pytest.mark.parametrize("rows,nq,nkv,pair_mode,norm,kv8,pad", [
    (3, 32, 8, 0, False, False, 0), (70, 32, 8, 1, True, False, 4), (300, 8, 1, 0, True, True, 0), (5, 4, 4, 1, False, True, 0),
    (9, 16, 2, 0, False, False, 2)])
def test_rope_kv_layouts(rows, nq, nkv, pair_mode, norm, kv8, pad):
    """Vector and general writer (rows padded off the 8-byte grid) against the rotation in float32; idle rows untouched."""
    from plow_b200.ops import gqa
    hd, dev = 128, "cuda"
    g = torch.Generator(device=dev).manual_seed(rows)
    W = (nq + 2 * nkv) * hd
    qkv = torch.randn(rows, W + pad, device=dev, generator=g).bfloat16()[:, pad // 2:pad // 2 + W]
    tab = torch.randn(400, hd, device=dev, generator=g)
    pos = torch.randint(0, 400, (rows,), dtype=torch.int32, device=dev, generator=g)
    pos[rows // 2] = -1
    seq = torch.arange(rows, dtype=torch.int32, device=dev)
    pt = torch.randperm(rows * 7, device=dev, generator=g).int().view(rows, 7).contiguous()
    qn, kn = [(torch.rand(hd, device=dev, generator=g) + 0.5).bfloat16() if norm else None for _ in range(2)]
    kc = torch.zeros(rows * 7, 64, nkv, hd, dtype=torch.uint8 if kv8 else torch.bfloat16, device=dev)
    vc = torch.zeros_like(kc)
    ks = torch.zeros(rows * 7, 64, 2 * nkv, device=dev) if kv8 else None
    q = torch.full((rows, nq, hd), 7.0, device=dev).bfloat16()
    gqa.rope_kv(qkv, kc, vc, tab, pos, seq, pt, nq, nkv, hd, pair_mode=pair_mode, qn=qn, kn=kn, eps=1e-6, q_out=q, kv_scale=ks)
    torch.cuda.synchronize()
    live = (pos >= 0).nonzero()[:, 0]
    x = qkv[live].float().view(-1, nq + 2 * nkv, hd)

    def rot(t, gamma):
        if gamma is not None:
            t = (t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + 1e-6) * gamma.float()).bfloat16().float()
        c, s = tab[pos[live].long(), :64][:, None], tab[pos[live].long(), 64:][:, None]
        a, b = (t[..., 0::2], t[..., 1::2]) if pair_mode else (t[..., :64], t[..., 64:])
        u, w = a * c - b * s, b * c + a * s
        return torch.stack([u, w], -1).flatten(-2) if pair_mode else torch.cat([u, w], -1)
    page = pt[seq[live].long(), (pos[live] // 64).long()].long()
    at = (pos[live] % 64).long()
    want_k, want_v = rot(x[:, nq:nq + nkv], kn), x[:, nq + nkv:]

    def cells(c, o):
        c = c[page, at]
        return c.view(torch.float8_e4m3fn).float() * ks[page, at][:, o:o + nkv, None] if kv8 else c.float()
    # one bf16 rounding (of the norm too, which the rotation mixes between two values); cells of the e4m3 cache one rounding of a
    # 448-scaled row
    cell = 2.0 ** -4 if kv8 else 2.0 ** -7
    for got, want, tol in ((q[live].float(), rot(x[:, :nq], qn), 2.0 ** -7), (cells(kc, 0), want_k, cell), (cells(vc, nkv), want_v, cell)):
        assert ((got - want).abs() <= tol * want.abs().amax(-1, keepdim=True)).all()
    assert (q[pos < 0] == 7.0).all()


@pytest.mark.parametrize("T,heads,pair_mode", [(1, 128, 1), (37, 128, 1), (5, 12, 1), (9, 16, 0)])
def test_mla_q_rope_layouts(T, heads, pair_mode):
    from plow_b200.ops import mla
    dev = "cuda"
    q = torch.randn(T, heads * 192, device=dev).bfloat16()
    tab = torch.randn(200, 64, device=dev)
    pos = torch.randint(0, 200, (T,), dtype=torch.int32, device=dev)
    if T > 1:
        pos[0] = -1
    src = q.clone()
    mla.q_rope(q, tab, pos, heads, 128, 64, pair_mode)
    a = src.view(T, heads, 192).float()
    c, s = tab[pos.clamp_min(0).long(), :32][:, None], tab[pos.clamp_min(0).long(), 32:][:, None]
    x, y = (a[..., 128::2], a[..., 129::2]) if pair_mode else (a[..., 128:160], a[..., 160:])
    u, w = x * c - y * s, y * c + x * s
    want = a.clone()
    want[..., 128:] = torch.stack([u, w], -1).flatten(-2) if pair_mode else torch.cat([u, w], -1)
    want[pos < 0] = a[pos < 0]
    got = q.view(T, heads, 192).float()
    assert torch.equal(got[..., :128], a[..., :128])
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all()
