"""GEMM shapes with too few 256 x 256 tiles for the SMs: narrower tiles, the reduction split over a cluster, operands
exchanged.  The sizes are the smallest found for each of the plans (ragged in every dimension, last k-blocks that are mostly
zero fill, columns no pair has to finish, batches); the truth is the CPU oracle, and for fp32 the fp64 product of the operands
cut to tf32.  Tolerance: half a unit of the output type (test_gemm_gpu.py) plus fp32 summation order, which for K products of
size up to 1 stays below K * 2^-24 * sqrt(K) / 2."""
import numpy as np
import pytest
import torch

from helpers import gemm_plan
from test_gemm_gpu import run

pytestmark = pytest.mark.gpu

# (M, N, K, L, row-major): tile width / split / operands exchanged, in bf16
SHAPES = [(8, 8, 8, 1, False),            # 64
          (8, 1544, 72, 3, True),         # 64, exchanged
          (8, 1544, 1032, 1, True),       # 64 / 2
          (8, 2056, 1032, 3, True),       # 64 / 2, exchanged
          (8, 8, 1032, 1, False),         # 64 / 3: column units without an owner
          (8, 1544, 1032, 3, True),       # 64 / 3, exchanged
          (8, 8, 2056, 1, False),         # 64 / 4
          (8, 2056, 1032, 1, True),       # 64 / 2
          (8, 776, 1032, 3, True),        # 64 / 4, exchanged
          (72, 3080, 4104, 3, True),      # 128, exchanged
          (72, 1544, 1032, 3, True),      # 128 / 3, exchanged
          (16, 1544, 72, 3, True),        # 128
          (720, 9456, 64, 1, True),       # 128, three waves
          (136, 776, 2056, 3, False),     # 128 / 2
          (72, 2056, 2056, 3, True),      # 128 / 2, exchanged
          (72, 776, 1032, 3, True),       # 128 / 3
          (72, 520, 4104, 3, True),       # 128 / 4
          (1032, 72, 2056, 3, False),     # 128 / 4, exchanged
          (264, 776, 2056, 3, True),      # 256 / 2
          (264, 2056, 2056, 1, True),     # 256 / 3
          (1032, 520, 4104, 1, False)]    # 256 / 4
# tile width, pairs that share a tile's reduction, operands exchanged
PLANS = [(64, 1, 0), (64, 1, 1), (64, 2, 0), (64, 2, 1), (64, 3, 0), (64, 3, 1), (64, 4, 0), (64, 2, 0), (64, 4, 1),
         (128, 1, 1), (128, 3, 1), (128, 1, 0), (128, 1, 0), (128, 2, 0), (128, 2, 1), (128, 3, 0), (128, 4, 0), (128, 4, 1),
         (256, 2, 0), (256, 3, 0), (256, 4, 0)]


def test_the_shapes_reach_the_plans(lib, cuda):
    assert [gemm_plan(lib, *s, dtype=1) for s in SHAPES] == PLANS
    assert gemm_plan(lib, 8192, 8192, 8192, 1, False, dtype=0) == (256, 1, 0)
    assert gemm_plan(lib, 2048, 768, 4096, 1, False, dtype=0) == (128, 1, 0)
    # a short reduction does not pay for further waves of narrow tiles
    for M, N, K, L, dtype in ((256, 18944, 8, 1, 1), (256, 18944, 64, 1, 1), (776, 3992, 136, 1, 1), (256, 30000, 8, 1, 3),
                              (464, 2040, 520, 4, 3), (1024, 1024, 264, 8, 3)):
        assert gemm_plan(lib, M, N, K, L, True, dtype) == (256, 1, 0), (M, N, K, L, dtype)


@pytest.mark.parametrize("M,N,K,L,row_major", SHAPES)
def test_narrow_and_split_plans_match_the_oracle(lib, oracle, cuda, M, N, K, L, row_major):
    run(lib, oracle, M, N, K, dtype=0, row_major=row_major, L=L, seed=K)
    run(lib, oracle, M, N, K, dtype=1, row_major=row_major, L=L, alpha=0.5, beta=2.0, seed=K + 1)
    run(lib, oracle, M, N, K, dtype=0, row_major=not row_major, L=L, alpha=-1.0, beta=0.5, seed=K + 2)


@pytest.mark.parametrize("M,N,K,L,row_major", SHAPES)
def test_narrow_and_split_plans_in_tf32_with_a_separate_source(lib, cuda, M, N, K, L, row_major):
    g = torch.Generator().manual_seed(M + N)
    a, b = (torch.rand(L, r, K, generator=g) * 2 - 1 for r in (M, N))
    shape = (L, M, N) if row_major else (L, N, M)
    src = torch.rand(*shape, generator=g)
    d = torch.full((L * M * N + 64,), -3.0, device="cuda")
    lib.gemm(a.cuda(), b.cuda(), d, dtype=3, m=M, n=N, k=K, l=L, alpha=0.5, beta=-2.0, c_row_major=row_major, c_src=src.cuda())
    lib.check_device()
    cut = lambda x: x.view(torch.int32).bitwise_and(-8192).view(torch.float32).double().numpy()    # noqa: E731
    ref = 0.5 * np.einsum("lmk,lnk->lmn" if row_major else "lmk,lnk->lnm", cut(a), cut(b), optimize=True) - 2.0 * src.double().numpy()
    err = np.abs(d[:L * M * N].view(*shape).cpu().numpy() - ref).max()
    assert err <= K * 2.0 ** -24 * K ** 0.5 / 2 + 2.0 ** -22, err
    assert bool((d[L * M * N:] == -3.0).all())


def test_threads_on_streams_of_their_own_get_the_plans_and_results_of_one(lib, cuda):
    import threading
    g = torch.Generator().manual_seed(2)
    calls = []
    for i, (M, N, K, L, row_major) in enumerate(SHAPES[:12]):
        a, b = (torch.randn(L, r, K, generator=g).bfloat16().cuda() for r in (M, N))
        c, d = (torch.zeros(L, M, N, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        calls.append((a, b, c, d, dict(dtype=1, m=M, n=N, k=K, l=L, c_row_major=row_major)))
    torch.cuda.synchronize()
    plans, errors = {}, []

    def work(i):
        try:
            torch.cuda.set_device(0)
            a, b, c, _, kw = calls[i]
            plans[i] = gemm_plan(lib, *SHAPES[i], dtype=1)
            stream = torch.cuda.Stream()
            for _ in range(3):
                lib.gemm(a, b, c, **kw, stream=stream.cuda_stream)
            stream.synchronize()
        except Exception as e:      # noqa: BLE001 - reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    lib.check_device()
    assert [plans[i] for i in range(len(calls))] == PLANS[:len(calls)]
    for a, b, c, d, kw in calls:
        lib.gemm(a, b, d, **kw)
        lib.check_device()
        assert torch.equal(c, d)
