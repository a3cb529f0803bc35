"""Work list of the latent decode and the merge + W_uv kernel at their edges: one row, rows around the merge warps' batches and the
128-row tile, rows without tokens, one split and the most that the kernel merges, lists beyond the length-ordered size."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _splits(n, tps, max_splits):
    tiles = (n + 63) // 64
    ns = max(1, min(max_splits, -(-tiles // tps)))
    per = max(1, -(-tiles // ns))
    return tiles, per, max(1, -(-tiles // per))


@pytest.mark.parametrize("T", [1, 33, 256, 257, 1500])
def test_items_cover_every_page_once(T):
    from plow_b200.ops import mla
    g = torch.Generator().manual_seed(T)
    lens = torch.randint(0, 4097, (T,), generator=g).tolist()
    lens[T // 2] = 0 if T > 1 else 4096
    ws = mla.DecodeWorkspace(T, 4096, tiles_per_split=4, heads=1, latent=8)
    ws.claims.fill_(5)
    mla.build_items(torch.tensor(lens, dtype=torch.int32, device="cuda"), T, ws)
    want = []
    for r, n in enumerate(lens):
        tiles, per, ns = _splits(n, 4, ws.max_splits)
        if tiles:
            want.append((per, r, [(r, h, s, s * per, min(per, tiles - s * per), 0, 0, 0) for s in range(ns) for h in (0, 1)]))
    if T <= 256:
        want.sort(key=lambda x: (-x[0], x[1]))               # longest first
    flat = [i for w in want for i in w[2]]
    assert int(ws.n_items) == len(flat) and not ws.claims.any()
    assert [tuple(i) for i in ws.items.view(-1, 8)[:len(flat)].tolist()] == flat


@pytest.mark.parametrize("T,max_ctx", [(1, 64), (7, 32768), (8, 4096), (9, 32768), (63, 8192), (64, 32768), (65, 8192), (128, 8192), (129, 8192), (200, 2048)])
def test_fold_rows(T, max_ctx):
    from plow_b200.ops import mla, native
    H, dev = 8, "cuda"
    g = torch.Generator(device=dev).manual_seed(T)
    ws = mla.DecodeWorkspace(T, max_ctx, heads=H)
    lens = torch.randint(1, max_ctx + 1, (T,), generator=g, device=dev, dtype=torch.int32)
    lens[0] = max_ctx
    ws.opart.copy_(torch.randn(ws.opart.shape, device=dev, generator=g))
    ws.lse.copy_(torch.randn(ws.lse.shape, device=dev, generator=g) * 3)
    wuv = (torch.randn(H * 128, 512, device=dev, generator=g) * 0.1).bfloat16()
    ns = [_splits(n, 32, ws.max_splits)[2] for n in lens.tolist()]
    live = (torch.arange(ws.max_splits, device=dev)[None] < torch.tensor(ns, device=dev)[:, None])[..., None]
    p = torch.softmax(torch.where(live, ws.lse * 0.6931471805599453, torch.full_like(ws.lse, -float("inf"))), 1)      # [T, splits, H]
    ws.opart[~live[..., 0]] = float("nan")                   # what lies past a row's splits is not read
    merged = torch.where(live[..., None], p[..., None].double() * torch.nan_to_num(ws.opart.double()), 0.0).sum(1)
    ref = torch.einsum("thc,hvc->thv", merged, wuv.view(H, 128, 512).double()).reshape(T, -1)
    ao = torch.full((T + 1, H * 128), 7.0, device=dev).bfloat16()
    aq, saq = mla.fold(ws, lens, wuv, T, H, ao[:T], want_fp8=True)
    torch.cuda.synchronize()
    native.check_status()
    # the merged operand and the result are each rounded to bf16 once (2^-9 relative)
    rel = ((ao[:T].double() - ref).norm(dim=1) / ref.norm(dim=1)).max()
    assert rel < 2 ** -8, rel
    assert (ao[T] == 7.0).all()
    back = aq.double().view(T, H, 128) * saq.t()[..., None].double()
    # e4m3: half of 2^-3 relative at most, per element of magnitude above the smallest normal
    assert ((back.view(T, -1) - ao[:T].double()).norm(dim=1) / ao[:T].double().norm(dim=1)).max() < 2 ** -4
