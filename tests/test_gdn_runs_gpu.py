"""Gated delta rule over mixed runs: run lengths around the two-token step, the stage and the row block, sequences that
start and that continue, idle rows between them, head ratios, rows whose start is not aligned for vector loads."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(lens, starts, hk, hv, idle, pad, seed):
    """rows of the runs in turn, `idle` inactive rows before each; qkvz rows `pad` elements wider than needed"""
    d, conv, dev = 128, 4, "cuda"
    g = torch.Generator(device=dev).manual_seed(seed)
    C = (2 * hk + hv) * d
    rows = sum(lens) + idle * len(lens)
    qkvz = torch.randn(rows, C + hv * d + pad, device=dev, generator=g).bfloat16()
    qkvz = qkvz[:, pad:]
    ba = torch.randn(rows, 2 * hv, device=dev, generator=g).bfloat16()
    conv_w = torch.randn(C, conv, device=dev, generator=g) * 0.5
    a_log = torch.randn(hv, device=dev, generator=g) * 0.5
    dt_bias = torch.randn(hv, device=dev, generator=g) * 0.5
    conv_state = torch.randn(len(lens), C, conv - 1, device=dev, generator=g)
    ssm_state = torch.randn(len(lens), hv, d, d, device=dev, generator=g) * 0.1
    pos, seq, spans = [], [], []
    for i, (n, p) in enumerate(zip(lens, starts)):
        pos += [-1] * idle
        seq += [i] * idle
        spans.append((len(pos), n))
        pos += range(p, p + n)
        seq += [i] * n
    t = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    return qkvz, ba, conv_w, a_log, dt_bias, conv_state, ssm_state, t(pos), t(seq), spans


@pytest.mark.parametrize("lens,starts,hk,hv,idle,pad", [
    ([1], [0], 2, 4, 0, 0), ([1, 1, 1], [0, 5, 9], 16, 32, 1, 0), ([2, 3, 4], [0, 7, 0], 2, 2, 0, 0),
    ([7, 8, 9, 1, 2], [0, 11, 0, 3, 1], 2, 4, 2, 1), ([15, 16, 17, 18], [4, 0, 1, 2], 1, 4, 0, 3),
    ([100, 1, 301], [0, 64, 1000], 2, 4, 1, 2), ([70, 5, 4, 3, 66], [0, 1, 0, 9, 2], 2, 4, 1, 0), ([25, 24, 23, 1, 1, 1, 200], [0, 1, 2, 3, 4, 5, 6], 2, 4, 0, 4),
    # 128 items a run: more than blocks (the second halves take some), more than halves (a half takes several, short runs skipped between)
    ([41, 50], [3, 0], 16, 32, 0, 0), ([3, 40, 1, 2, 27, 4, 9], [0, 5, 9, 0, 2, 7, 1], 16, 32, 1, 0), ([1] * 40, list(range(40)), 16, 32, 0, 0)])
def test_gdn_runs(lens, starts, hk, hv, idle, pad):
    from plow_b200.ops import gdn
    qkvz, ba, conv_w, a_log, dt_bias, cs, ss, pos, seq, spans = _case(lens, starts, hk, hv, idle, pad, sum(lens))
    cs0, ss0 = cs.clone(), ss.clone()
    out = torch.full((qkvz.shape[0], hv * 128), 7.0, device="cuda").bfloat16()
    gdn.gdn(qkvz, ba, conv_w, a_log, dt_bias, cs, ss, pos, seq, hk, hv, out=out)
    torch.cuda.synchronize()
    for i, (r0, n) in enumerate(spans):
        fresh = starts[i] == 0
        o, h, S = gdn.reference(qkvz[r0:r0 + n], ba[r0:r0 + n], conv_w, a_log, dt_bias, hk, hv,
                                conv_hist=None if fresh else cs0[i], S=None if fresh else ss0[i])
        # the output is rounded to bf16 (2^-9 of itself); sums of 128 f32 terms in another order are far below that
        assert ((out[r0:r0 + n].float() - o).abs() <= 2.0 ** -8 * o.abs() + 2e-5 * o.abs().max()).all(), i
        # f32 state: a few ulp a token, contracted by the decay
        assert (ss[i] - S).norm() <= 5e-6 * S.norm(), i
        assert torch.equal(cs[i], h), i
    assert (out[pos < 0] == 7.0).all()


@pytest.mark.parametrize("hd,pad,ofs", [(128, 0, 256), (128, 1, 256), (128, 0, 258), (64, 0, 128)])
def test_gated_norm_layouts(hd, pad, ofs):
    from plow_b200.ops import gdn
    rows, heads = 37, 3
    o = torch.randn(rows, heads * hd, device="cuda").bfloat16()
    z = torch.randn(rows, ofs + heads * hd + 4 + pad, device="cuda").bfloat16()
    gamma = torch.rand(hd, device="cuda") + 0.5
    got = gdn.gated_norm(o, z, ofs, gamma, heads, hd, 1e-6).float().view(rows, heads, hd)
    x = o.double().view(rows, heads, hd)
    zz = z[:, ofs:ofs + heads * hd].double().view(rows, heads, hd)
    want = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6) * gamma.double() * torch.nn.functional.silu(zz)
    # one rounding to bf16
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all()
