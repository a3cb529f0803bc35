"""The launch counter of the bench agrees with the kernel nodes of the captured calls."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _kernel_nodes(fn):
    fn()                                                      # one-time set-up happens outside the capture
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        fn()
    rt = C.CDLL("libcudart.so.12")
    graph, n = C.c_void_p(g.raw_cuda_graph()), C.c_size_t(0)
    assert rt.cudaGraphGetNodes(graph, None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert rt.cudaGraphGetNodes(graph, nodes, C.byref(n)) == 0
    kinds = []
    for node in nodes:
        t = C.c_int(-1)
        assert rt.cudaGraphNodeGetType(C.c_void_p(node), C.byref(t)) == 0
        kinds.append(t.value)
    return kinds.count(0)                                     # cudaGraphNodeTypeKernel


def _counted(fn):
    from plow_b200.ops import native
    n0 = native.LAUNCHES["n"]
    fn()
    return native.LAUNCHES["n"] - n0


@pytest.mark.parametrize("rows,splits", [(4, 1), (4, 5), (400, 1), (400, 3)])
def test_attention(rows, splits):
    from plow_b200.ops import gqa
    kc = torch.randn(10, 64, 2, 128, device="cuda").bfloat16()
    pt = torch.arange(10, dtype=torch.int32, device="cuda").view(1, 10)
    seq, pos = torch.zeros(rows, dtype=torch.int32, device="cuda"), torch.arange(rows, dtype=torch.int32, device="cuda")
    q = torch.randn(rows, 8, 128, device="cuda").bfloat16()
    ws = gqa.AttnWorkspace(rows, 8, 2, 128, 640, "cuda", max_splits=splits)
    out = torch.empty(rows, 1024, dtype=torch.bfloat16, device="cuda")

    def run():
        gqa.attention(q, kc, kc, pt, seq, pos, ws, out=out)
    assert _counted(run) == _kernel_nodes(run)


@pytest.mark.parametrize("rows", [1, 64, 65])
def test_gdn(rows):
    from plow_b200.ops import gdn
    C_ = 4 * 128
    x, ba = torch.randn(rows, C_ + 256, device="cuda").bfloat16(), torch.randn(rows, 4, device="cuda").bfloat16()
    w, a, dt = torch.randn(C_, 4, device="cuda"), torch.zeros(2, device="cuda"), torch.zeros(2, device="cuda")
    cs, ss = torch.zeros(1, C_, 3, device="cuda"), torch.zeros(1, 2, 128, 128, device="cuda")
    pos, seq = torch.arange(rows, dtype=torch.int32, device="cuda"), torch.zeros(rows, dtype=torch.int32, device="cuda")

    def run():
        gdn.gdn(x, ba, w, a, dt, cs, ss, pos, seq, 1, 2)
    assert _counted(run) == _kernel_nodes(run)


@pytest.mark.parametrize("build,merge", [(True, True), (False, True), (False, False)])
def test_latent_decode(build, merge):
    from plow_b200.ops import mla
    T = 2
    ws = mla.DecodeWorkspace(T, 256)
    kvlen = torch.full((T,), 100, dtype=torch.int32, device="cuda")
    mla.build_items(kvlen, T, ws)
    q8, sq = torch.zeros(128, T, 576, dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn), torch.ones(128, T, device="cuda")
    kv = torch.zeros(4, 64, 576, dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn)
    scale, smax = torch.ones(4, 64, device="cuda"), torch.ones(4, 4, device="cuda")
    pt = torch.arange(4, dtype=torch.int32, device="cuda").view(T, 2)
    slot = torch.arange(T, dtype=torch.int32, device="cuda")
    claim = iter(range(16))                                   # a list serves one launch per work counter

    def run():
        mla.decode(q8, sq, kv, scale, smax, pt, slot, kvlen, ws, 0.1, merge=merge, build_items=build, claim_slot=next(claim))
    assert _counted(run) == _kernel_nodes(run)
