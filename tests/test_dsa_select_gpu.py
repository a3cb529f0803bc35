"""Index scores and exact top-k at their edges: row lengths around the tile, the CTA's run of tiles, the cluster's slices and the
selection size; rows of ties; rows too long for shared memory."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _order(scores, top_k):
    """Positions of the top_k by (score desc, lowest index), over the bit order of the floats (-0 is below +0)."""
    b = scores.view(torch.int32).long()
    key = torch.where(b < 0, -(b & 0x7FFFFFFF) - 1, b)
    return torch.sort(torch.sort(key, descending=True, stable=True).indices[:top_k]).values


@pytest.mark.parametrize("lens,top_k,kind", [
    ([1, 0, 63, 64, 65, 127, 128, 129], 64, "rand"),
    ([1023, 1024, 1025, 1152, 2047, 2048, 2049, 2176], 2048, "rand"),
    ([4097, 8191, 16384, 10241, 500], 2048, "rand"),
    ([16384, 1, 1000, 8191, 2305, 512] * 2, 2048, "rand"),           # four tiles a CTA (above: two; below: eight)
    ([5000] * 150 + [7, 4999], 512, "rand"),
    ([9000] * 300, 100, "rand"),
    ([6000, 2049, 12345], 2048, "few"),
    ([6000, 2048, 12345], 2048, "zero"),
    ([40000, 39999], 1, "rand"),
    ([360001, 333], 2048, "rand"),
    ([360001], 2048, "few"),
])
def test_dsa_select_edges(lens, top_k, kind):
    from plow_b200.ops import dsa, native
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(len(lens) + top_k)
    rows, max_len = len(lens), max(lens)
    mp = (max_len + 63) // 64
    n_pages = mp + 3                                       # the rows share one shuffled pool of pages
    cache = torch.randn(n_pages, 64, 128, device=dev, generator=g)
    if kind == "few":
        cache[:] = torch.randn(1, 4, 128, device=dev, generator=g).repeat(1, 16, 1)
    cache = cache.to(torch.float8_e4m3fn)
    cs = torch.ones(n_pages, 64, device=dev) if kind != "rand" else torch.rand(n_pages, 64, device=dev, generator=g) + 0.5
    pt = torch.stack([torch.randperm(n_pages, device=dev, generator=g)[:mp] for _ in range(rows)]).int()
    q = torch.randn(rows, 64 * 128, device=dev, generator=g).bfloat16()
    w = torch.randn(rows, 64, device=dev, generator=g) * (kind != "zero")
    tab = torch.cat([torch.ones(max_len, 32, device=dev), torch.zeros(max_len, 32, device=dev)], 1)
    pos = torch.tensor(lens, dtype=torch.int32, device=dev) - 1
    seq = torch.arange(rows, dtype=torch.int32, device=dev).flip(0)
    ws = dsa.SelectWorkspace(rows, max_len, dev)
    ws.scores.fill_(float("inf"))                          # what lies past a row is never taken
    sel = dsa.select(q, w, cache, cs, tab, pos, seq, pt, top_k, ws, 64)
    torch.cuda.synchronize()
    native.check_status()
    for r, n in enumerate(lens):
        got = ws.scores[r, :n]
        assert torch.isinf(ws.scores[r, n:]).all()
        if r < 8 and n:
            # over the e4m3 heads and weights that the preparation kernel wrote, which has its own test
            q8, wq = ws.q8[r].double(), ws.wq[r].double()
            parts = cache[pt[seq[r]].long()].view(-1, 128)[:n].split(65536)
            want = torch.cat([torch.relu(part.double() @ q8.T) @ wq for part in parts])
            mag = torch.cat([(part.double().abs() @ q8.abs().T) @ wq.abs() for part in parts])
            kscale = cs[pt[seq[r]].long()].view(-1)[:n].double()
            # exact products; 128 f32 adds, 64 f32 fused multiply-adds and one multiply, each within 2^-23 of the magnitudes
            bound = mag * kscale * (128 + 64 + 1) * 2 ** -23
            assert ((got.double() - want * kscale).abs() <= bound).all(), r
        want = torch.full((top_k,), -1, dtype=torch.long, device=dev)
        if n <= top_k:
            want[:n] = torch.arange(n, device=dev)
        else:
            want[:] = _order(got, top_k)
        assert torch.equal(sel[r].long(), want), r
