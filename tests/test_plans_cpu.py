"""The rules that choose a kernel by size (cfk_fmha_plan), which need no GPU: where their lines lie, and that a plan is one the
kernels can run, over sizes, types, masks and head counts."""
import random

import pytest

import cfk_b200
from helpers import BLOCK, FEW_ROWS, ONE_TILE, fmha_plan


@pytest.mark.parametrize("dtype,B,H,Sq,Skv,D,causal,plan", [
    (0, 4, 16, 4096, 4096, 128, False, (BLOCK, 0, 0, 0)),
    (1, 2, 32, 8192, 8192, 128, True, (BLOCK, 0, 0, 0)),
    (0, 4, 8, 4096, 4096, 256, False, (BLOCK, 0, 0, 0)),
    (1, 4, 32, 1, 6001, 128, True, (FEW_ROWS, 2, 0, 0)),
    (1, 2, 1, 1, 65536, 128, True, (FEW_ROWS, 8, 0, 0)),
    (0, 1, 1, 32, 4096, 128, False, (FEW_ROWS, 8, 0, 0)),
    (0, 1, 1, 128, 1024, 128, False, (FEW_ROWS, 8, 0, 0)),
    (0, 1, 8, 129, 4096, 128, False, (ONE_TILE, 8, 0, 0)),       # more than 128 rows
    (0, 1, 8, 128, 1023, 128, False, (ONE_TILE, 4, 0, 0)),       # more than 32 rows, fewer than 1024 keys
    (0, 1, 19, 128, 1024, 128, False, (ONE_TILE, 4, 0, 0)),      # more than 32 rows, groups of 16 beyond the SMs
    (0, 1, 37, 16, 1024, 256, False, (FEW_ROWS, 4, 0, 0)),       # d = 256: four CTAs or more per group
    (0, 1, 38, 16, 1024, 256, False, (BLOCK, 0, 0, 0)),
    (0, 1, 37, 16, 1023, 256, False, (BLOCK, 0, 0, 0)),
    (0, 2, 111, 32, 4096, 128, False, (FEW_ROWS, 1, 0, 0)),      # two groups per head: one wave of 444 ..
    (0, 1, 223, 32, 4096, 128, False, (BLOCK, 0, 0, 0)),         # .. two, as the 256-row kernel has ..
    (1, 4, 74, 17, 4096, 128, True, (BLOCK, 0, 0, 0)),
    (1, 4, 74, 17, 800, 128, True, (FEW_ROWS, 1, 0, 0)),         # (two-term P)
    (0, 4, 74, 16, 4096, 128, True, (FEW_ROWS, 1, 0, 0)),        # (one group per head)
    (2, 4, 74, 32, 4096, 128, False, (FEW_ROWS, 1, 0, 0)),       # (e4m3 V)
    (0, 1, 297, 32, 4096, 128, False, (FEW_ROWS, 1, 0, 0)),      # .. two against three
    (0, 1, 8, 300, 896, 128, False, (BLOCK, 0, 0, 0)),           # split keys from 8 key tiles on, that is 897 keys
    (0, 1, 8, 300, 897, 128, False, (ONE_TILE, 4, 0, 0)),
    (0, 1, 12, 3080, 3080, 128, False, (BLOCK, 0, 8, 8)),        # a remainder of 8 rows
    (0, 1, 12, 3080, 3080, 128, True, (BLOCK, 0, 0, 0)),
    (0, 1, 12, 3104, 3104, 128, False, (BLOCK, 0, 32, 8)),
    (0, 1, 12, 3105, 3105, 128, False, (BLOCK, 0, 0, 0)),
])
def test_where_the_lines_lie(lib, dtype, B, H, Sq, Skv, D, causal, plan):
    assert fmha_plan(lib, dtype, B, H, Sq, Skv, D, causal) == plan


def test_every_plan_can_be_run(lib):
    """Few rows: 128 at most.  Key parts: 1, 2, 4 or 8 CTAs of one cluster.  A remainder: of unmasked calls, what is left behind
    whole blocks, 32 rows at most.  The choice does not depend on addresses, strides, scales or the statistics asked for."""
    rng = random.Random(11)
    log = lambda lo, hi: int(round(lo * (hi / lo) ** rng.random()))      # noqa: E731
    seen = set()
    for _ in range(4000):
        dtype, D = rng.choice([0, 1, 2]), rng.choice([64, 128, 256])
        Skv = log(1, 70000)
        Sq = min(Skv, log(1, 9000)) if rng.random() < 0.8 else log(1, 9000)
        if rng.random() < 0.3:
            Sq = 128 * log(1, 32) + rng.randint(1, 32)
        B, H, causal = log(1, 64), log(1, 64), rng.random() < 0.4 and Sq <= Skv
        hybrid = dtype == 2 and D != 256 and rng.random() < 0.3
        kernel, splits, rows, tail_splits = plan = fmha_plan(lib, dtype, B, H, Sq, Skv, D, causal, v_fp16=hybrid)
        seen.add((kernel, min(splits, 2), rows > 0))
        assert kernel in (BLOCK, FEW_ROWS, ONE_TILE) and (kernel != ONE_TILE or D != 256)
        assert splits in ((0,) if kernel == BLOCK else (1, 2, 4, 8))
        if kernel == FEW_ROWS:
            assert Sq <= 128 and rows == 0
        if rows:
            assert not causal and D != 256 and rows <= 32 and splits < 2 and tail_splits in (1, 2, 4, 8)
            assert rows == Sq % (256 if kernel == BLOCK else 128) and Sq > rows
        else:
            assert tail_splits == 0
        assert plan == lib.fmha_plan(lib.fmha_args(
            0x10010, 0x20, 0x30, 0x40, dtype=dtype, batch=B, heads=H, seqlen_q=Sq, seqlen_kv=Skv, head_dim=D, softmax_scale=3.0,
            causal=causal, v_fp16=hybrid, out_dtype=1, lse=0x50, q_stride=(1 << 30, 1 << 20, 1 << 10)))
    assert seen == {(BLOCK, 0, False), (BLOCK, 0, True), (FEW_ROWS, 1, False), (FEW_ROWS, 2, False), (ONE_TILE, 1, False),
                    (ONE_TILE, 1, True), (ONE_TILE, 2, False)}


def test_knobs_and_the_score_dump_keep_their_kernel(lib):
    call = (0, 1, 8, 256, 2048, 128, False)
    assert fmha_plan(lib, *call) == (ONE_TILE, 8, 0, 0)
    assert fmha_plan(lib, *call, s_dump=0x60) == (BLOCK, 0, 0, 0)
    for which, value, kernel in ((cfk_b200.TUNE_FMHA_SCHED, 0, 0), (cfk_b200.TUNE_FMHA_SCHED, 1, 0),
                                 (cfk_b200.TUNE_FMHA_KERNEL, 1, 1), (cfk_b200.TUNE_FMHA_KERNEL, 2, 2)):
        lib.set_tunable(which, value)
        try:
            assert fmha_plan(lib, *call) == (kernel, 0, 0, 0)
        finally:
            lib.set_tunable(which, -1)


def test_plans_refuse_what_the_calls_refuse(lib):
    for kw, code in ((dict(Sq=200, Skv=100, causal=True), 2), (dict(D=96), 2), (dict(B=0), 1), (dict(dtype=3), 1)):
        base = dict(dtype=0, B=1, H=1, Sq=8, Skv=8, D=64, causal=False)
        base.update(kw)
        with pytest.raises(cfk_b200.CfkError) as e:
            fmha_plan(lib, **base)
        assert e.value.code == code
    assert lib.lib.cfk_fmha_plan(None, None) == 1 and lib.lib.cfk_gemm_plan(None, None) == 1
