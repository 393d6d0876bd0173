"""Calls of every route recorded into a CUDA graph: launches carry an attribute that lets them overlap the one before, clusters
are a launch attribute, and a call may be two launches.  A replay must give the bits of the calls made one by one."""
import pytest
import torch

from helpers import BLOCK, FEW_ROWS, ONE_TILE, fmha_plan

pytestmark = pytest.mark.gpu

# (B, H, Sq, Skv, causal) and the plan it must have
CALLS = [((1, 2, 300, 300, True), (BLOCK, 0, 0, 0)), ((2, 3, 5, 700, True), (FEW_ROWS, 4, 0, 0)),
         ((300, 1, 128, 128, True), (ONE_TILE, 1, 0, 0)), ((1, 4, 256, 2048, False), (ONE_TILE, 8, 0, 0)),
         ((12, 1, 3074, 2600, False), (BLOCK, 0, 2, 8))]


@pytest.mark.parametrize("static", [False, True])
def test_a_graph_of_all_routes_equals_the_calls_one_by_one(lib, cuda, static):
    D = 128
    g = torch.Generator().manual_seed(3)
    draw = lambda *s: torch.randn(*s, generator=g).half().cuda()      # noqa: E731
    ins = [(draw(B, Sq, H, D), draw(B, Skv, H, D), draw(B, Skv, H, D)) for (B, H, Sq, Skv, _), _ in CALLS]
    a, b = draw(256, 2056), draw(128, 2056)
    outs = [torch.zeros_like(q) for q, _, _ in ins] + [torch.zeros(128, 256, dtype=torch.float16, device="cuda"),
                                                      torch.zeros(128 * 256, dtype=torch.float32, device="cuda")]
    for (B, H, Sq, Skv, causal), plan in CALLS:
        assert fmha_plan(lib, 0, B, H, Sq, Skv, D, causal) == plan

    def calls():
        s = torch.cuda.current_stream().cuda_stream
        for (q, k, v), o, ((B, H, Sq, Skv, causal), _) in zip(ins, outs, CALLS):
            args = lib.fmha_args(q, k, v, o, dtype=0, batch=B, heads=H, seqlen_q=Sq, seqlen_kv=Skv, head_dim=D,
                                 softmax_scale=D ** -0.5, causal=causal)
            assert (lib.fmha_forward_static_raw if static else lib.fmha_forward_raw)(args, s) == 0
        lib.gemm(a, b, outs[-2], dtype=0, m=256, n=128, k=2056, stream=s)
        lib.convert(outs[-2], 0, outs[-1], 3, outs[-1].numel(), scale=2.0, stream=s)

    calls()
    lib.check_device()
    want = [o.clone() for o in outs]
    for o in outs:
        o.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls()
    assert all(bool((o == 0).all()) for o in outs)
    for _ in range(2):
        for o in outs:
            o.zero_()
        graph.replay()
        lib.check_device()
        assert all(torch.equal(o, w) for o, w in zip(outs, want))
