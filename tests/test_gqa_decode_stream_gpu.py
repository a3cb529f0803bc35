"""Streaming decode form of the grouped-query attention: sequences from one token up, pages cut between CTAs anywhere, idle
rows, head ratios, sliding windows, both cache types; calls that are no decode step keep the tile form."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(lens, nq, nkv, kv8, seed, idle=()):
    from plow_b200.ops import gqa
    hd, dev = 128, "cuda"
    g = torch.Generator(device=dev).manual_seed(seed)
    rows, per = len(lens), (max(lens) + 63) // 64
    n_pages = rows * per + 1
    kc = (torch.randn(n_pages, 64, nkv, hd, device=dev, generator=g) * 2).bfloat16()
    vc = torch.randn(n_pages, 64, nkv, hd, device=dev, generator=g).bfloat16()
    pt = torch.randperm(n_pages, device=dev, generator=g).int()[: rows * per].view(rows, per).contiguous()
    pos = torch.tensor(lens, dtype=torch.int32, device=dev) - 1
    for r in idle:
        pos[r] = -1
    seq = torch.randperm(rows, device=dev, generator=g).int()
    q = torch.randn(rows, nq, hd, device=dev, generator=g).bfloat16()
    if not kv8:
        return q, kc, vc, pt, seq, pos, None, kc, vc
    k8, ks = gqa.quant_cache(kc)
    v8, vs = gqa.quant_cache(vc)
    return q, k8, v8, pt, seq, pos, torch.cat([ks, vs], -1).contiguous(), k8.float() * ks[..., None], v8.float() * vs[..., None]


@pytest.mark.parametrize("kv8", [False, True])
@pytest.mark.parametrize("lens,nq,nkv,window,idle", [
    ([1], 32, 8, 0, ()), ([1, 2, 63, 64, 65, 127, 128, 129], 8, 8, 0, (3,)), ([5000], 32, 8, 0, ()), ([4000, 1, 1, 17], 8, 1, 0, (0, 2)),
    ([100 + 37 * i for i in range(64)], 32, 8, 0, (0, 31, 63)), ([3000, 700, 70], 16, 4, 200, ()), ([513] * 256, 4, 2, 0, ()),
    ([1200, 800], 8, 4, 64, ()), ([40, 40, 40], 32, 8, 0, (0, 1, 2)),
    # whole sequences per CTA up to their longest, and one page or one row too many; a fold of more partials than one batch
    ([768] * 18, 32, 8, 0, (5,)), ([768] * 19, 32, 8, 0, ()), ([768, 769], 32, 8, 0, ()), ([9000], 8, 1, 0, ())])
def test_decode_stream(lens, nq, nkv, window, idle, kv8):
    from plow_b200.ops import gqa, native
    q, kc, vc, pt, seq, pos, ks, kd, vd = _case(lens, nq, nkv, kv8, len(lens) + sum(lens) % 97, idle)
    rows = len(lens)
    ws = gqa.AttnWorkspace(rows, nq, nkv, 128, max(lens), "cuda")
    assert ws.dec is not None
    ref = gqa.reference(q, kd, vd, pt, seq, pos, window=window)
    for _ in range(2):                         # the arrival counts are set up anew by every call
        out = torch.full((rows, nq * 128), 7.0, device="cuda").bfloat16()
        gqa.attention(q, kc, vc, pt, seq, pos, ws, window=window, out=out, kv_scale=ks)
        torch.cuda.synchronize()
        native.check_status()
        live = pos >= 0
        if live.any():
            rel = (out[live].float() - ref[live]).norm() / ref[live].norm()
            assert rel < 6e-3, rel             # bf16 probabilities and result
        assert (out[~live] == 7.0).all()


def test_decode_workspace_serves_fewer_rows_and_other_calls():
    """One workspace: a decode step of fewer rows than it was made for, then a chunk of one sequence, then a step again."""
    from plow_b200.ops import gqa, native
    nq, nkv = 32, 8
    q, kc, vc, pt, seq, pos, _, _, _ = _case([300 + 11 * i for i in range(40)], nq, nkv, False, 3)
    ws = gqa.AttnWorkspace(48, nq, nkv, 128, 1024, "cuda")
    for _ in range(2):
        out = gqa.attention(q[:9], kc, vc, pt, seq[:9], pos[:9], ws)
        ref = gqa.reference(q[:9], kc, vc, pt, seq[:9], pos[:9])
        assert (out.float() - ref).norm() / ref.norm() < 6e-3
        cs, cp = torch.full((40,), 5, dtype=torch.int32, device="cuda"), torch.arange(250, 290, dtype=torch.int32, device="cuda")
        out = gqa.attention(q, kc, vc, pt, cs, cp, ws)
        ref = gqa.reference(q, kc, vc, pt, cs, cp)
        assert (out.float() - ref).norm() / ref.norm() < 6e-3
    native.check_status()


@pytest.mark.parametrize("form", ["stream", "tile"])
@pytest.mark.parametrize("lens,nq,nkv,window", [([1, 63, 64, 65, 130, 700], 32, 8, 0), ([900, 77, 3000, 40], 8, 4, 70), ([5, 1500], 16, 2, 33)])
def test_unused_e4m3_cells_may_hold_anything(lens, nq, nkv, window, form):
    """Cells that no row attends to (behind a sequence's end, before its window) are NaN codes with NaN and infinite scales."""
    from plow_b200.ops import gqa, native
    q, kc, vc, pt, seq, pos, ks, kd, vd = _case(lens, nq, nkv, True, sum(lens))
    if form == "tile":                                        # two tokens of a sequence in a row: no decode step
        n = torch.tensor([0 if v == 1 else 1 for v in lens], device="cuda").bool()
        seq, pos = seq.repeat_interleave(2), torch.stack([torch.where(n, pos - 1, -1), pos], 1).view(-1).int().contiguous()
        q = q.repeat_interleave(2, 0).contiguous()
    rows = len(pos)
    ref = gqa.reference(q, kd, vd, pt, seq, pos, window=window)
    used = torch.zeros(kc.shape[0], 64, dtype=torch.bool, device="cuda")
    for r in range(rows):
        hi = int(pos[r])
        t = torch.arange(max(0, hi - window + 1) if window else 0, hi + 1, device="cuda")
        used[pt[int(seq[r])][t // 64].long(), t % 64] = True
    kc, vc, ks = kc.view(torch.uint8).clone(), vc.view(torch.uint8).clone(), ks.clone()
    kc[~used] = 0x7F
    vc[~used] = 0xFF
    bad = torch.full_like(ks, float("nan"))
    bad[:, 1::2] = float("inf")
    ks = torch.where(used[..., None], ks, bad)
    ws = gqa.AttnWorkspace(rows, nq, nkv, 128, max(lens), "cuda")
    out = gqa.attention(q, kc, vc, pt, seq, pos, ws, window=window, kv_scale=ks)
    torch.cuda.synchronize()
    native.check_status()
    live = pos >= 0
    assert (out[live].float() - ref[live]).norm() / ref[live].norm() < 6e-3


@pytest.mark.parametrize("form", ["stream", "tile"])
@pytest.mark.parametrize("zero", ["some", "pages", "all"])
def test_zero_value_scales(zero, form):
    """A value scale of zero is a value of zero: the token keeps its share of the softmax."""
    from plow_b200.ops import gqa, native
    lens, nq, nkv = [70, 500, 1300], 8, 2
    q, kc, vc, pt, seq, pos, ks, kd, vd = _case(lens, nq, nkv, True, 11)
    if form == "tile":
        seq, pos, q = seq.repeat_interleave(2), torch.stack([pos - 1, pos], 1).view(-1).contiguous(), q.repeat_interleave(2, 0).contiguous()
    t = torch.arange(64, device="cuda")
    hide = {"some": (t % 3 == 0)[None].repeat(kc.shape[0], 1), "pages": (torch.arange(kc.shape[0], device="cuda") % 2 == 0)[:, None].repeat(1, 64),
            "all": torch.ones(kc.shape[0], 64, dtype=torch.bool, device="cuda")}[zero]
    ks = ks.clone()
    ks[..., nkv:][hide] = 0.0
    vd = torch.where(hide[..., None, None], torch.zeros_like(vd), vd)
    ref = gqa.reference(q, kd, vd, pt, seq, pos)
    ws = gqa.AttnWorkspace(len(pos), nq, nkv, 128, max(lens), "cuda")
    out = gqa.attention(q, kc, vc, pt, seq, pos, ws, kv_scale=ks).float()
    torch.cuda.synchronize()
    native.check_status()
    assert (out - ref).norm() <= 6e-3 * ref.norm()            # "all": exactly zero


@pytest.mark.parametrize("kv8", [False, True])
def test_repeats_bit_for_bit(kv8):
    """Every SM at work on many pages: the ring, the scales and the fold give the same bits each time."""
    from plow_b200.ops import gqa, native
    lens = torch.randint(512, 4353, (64,), generator=torch.Generator().manual_seed(4)).tolist()
    q, kc, vc, pt, seq, pos, ks, _, _ = _case(lens, 32, 8, kv8, 21)
    ws = gqa.AttnWorkspace(64, 32, 8, 128, 4352, "cuda")
    first = gqa.attention(q, kc, vc, pt, seq, pos, ws, kv_scale=ks)
    bad = torch.zeros((), dtype=torch.int64, device="cuda")
    for _ in range(300):
        bad += (gqa.attention(q, kc, vc, pt, seq, pos, ws, kv_scale=ks) != first).any()
    torch.cuda.synchronize()
    native.check_status()
    assert int(bad) == 0
