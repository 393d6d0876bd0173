"""Launches overlap their set-up with the launch before them in the stream (programmatic dependent launch).  A chain in
which every call reads what the call before it wrote, and overwrites what the call before that one read, must give the
same bits as the same chain with the device drained between the calls."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,S", [(64, 96), (128, 300), (256, 129)])
@pytest.mark.parametrize("side_stream", [False, True])
def test_chained_calls_equal_the_chain_with_waits(lib, cuda, D, S, side_stream):
    H, rounds = 2, 6
    g = torch.Generator().manual_seed(S)
    x0 = torch.randn(1, S, H, D, generator=g).half().cuda()
    w = (torch.randn(H * D, H * D, generator=g) / (H * D) ** 0.5).half().cuda()
    stream = torch.cuda.Stream() if side_stream else torch.cuda.current_stream()
    torch.cuda.synchronize()

    def chain(wait):
        x, y, f = x0.clone(), torch.zeros_like(x0), torch.zeros(x0.numel(), dtype=torch.float32, device="cuda")
        lse = torch.zeros(1, H, S, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        sp = stream.cuda_stream
        for _ in range(rounds):
            lib.fmha_forward(x, x, x, y, dtype=0, batch=1, heads=H, seqlen_q=S, seqlen_kv=S, head_dim=D,
                             softmax_scale=D ** -0.5, causal=True, lse=lse, stream=sp)
            if wait:
                torch.cuda.synchronize()
            lib.gemm(y, w, x, dtype=0, m=S // 8 * 8, n=H * D, k=H * D, c_row_major=True, stream=sp)    # x = y W^T
            if wait:
                torch.cuda.synchronize()
            lib.convert(x, 0, f, 3, x.numel(), scale=3.0, stream=sp)
            if wait:
                torch.cuda.synchronize()
            lib.convert(f, 3, x, 0, x.numel(), scale=0.5, stream=sp)
            if wait:
                torch.cuda.synchronize()
        lib.check_device()
        return x, y, f, lse

    for a, b in zip(chain(False), chain(True)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype,D", [(0, 64), (2, 64), (1, 128)])
def test_kernels_with_tensor_memory_follow_each_other_on_an_sm(lib, cuda, dtype, D):
    """Launches of half an SM (one-tile attention), of a whole one (256-row attention, d = 256) and of CTA pairs (GEMM), each on
    its way while the one before it runs: the results are those of the launches with waits between them."""
    g = torch.Generator().manual_seed(D)
    cast = {0: torch.float16, 1: torch.bfloat16, 2: torch.float8_e4m3fn}
    at = {}
    for name, (B, S, hd) in {"one tile": (300, 128, D), "block": (2, 400, D), "d256": (2, 300, 256)}.items():
        q, k, v = (torch.randn(B, S, 1, hd, generator=g).to(cast[dtype]).cuda() for _ in range(3))
        at[name] = (B, S, hd, q, k, v)
    a, b = (torch.randn(r, 512, generator=g).half().cuda() for r in (768, 1024))

    def chain(wait):
        outs = []
        for i in range(4):
            for name, (B, S, hd, q, k, v) in at.items():
                o = torch.zeros(B, S, 1, hd, dtype=torch.float16, device="cuda")
                lib.fmha_forward(q, k, v, o, dtype=dtype, batch=B, heads=1, seqlen_q=S, seqlen_kv=S, head_dim=hd,
                                 softmax_scale=hd ** -0.5, causal=bool(i & 1))
                outs.append(o)
                if wait:
                    torch.cuda.synchronize()
                c = torch.zeros(1024, 768, dtype=torch.float16, device="cuda")
                lib.gemm(a, b, c, dtype=0, m=768, n=1024, k=512)
                outs.append(c)
                if wait:
                    torch.cuda.synchronize()
        lib.check_device()
        return outs

    for x, y in zip(chain(False), chain(True)):
        assert torch.equal(x, y)
