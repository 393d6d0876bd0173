"""Few query rows against a long cache run in a kernel that splits the keys over the CTAs of a cluster.  Sizes are the
edges of its tiles (16 rows, 64 or 128 keys, a quarter of that per warp), of the split (one tile more or less than a CTA's
share, CTAs without a visible key) and of the rule that sends a call to it.  Tolerances are those of test_fmha_gpu.py."""
import math

import numpy as np
import pytest
import torch

from helpers import BLOCK, FEW_ROWS, fmha_plan, make_qkv, run_fmha
from test_fmha_gpu import check

pytestmark = pytest.mark.gpu

# (B, H, Sq, Skv): 1 to 8 CTAs per group of rows, whole and ragged tiles
SHAPES = [(1, 1, 1, 1), (2, 3, 1, 63), (1, 2, 3, 64), (1, 2, 16, 65), (2, 1, 17, 128), (1, 3, 9, 129), (1, 2, 32, 33),
          (3, 5, 1, 777), (1, 1, 7, 4099), (160, 1, 2, 300), (1, 1, 33, 1024), (1, 2, 100, 1500), (75, 2, 16, 200)]


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("dtype", [0, 1, 2])
@pytest.mark.parametrize("causal", [False, True])
def test_few_rows_match_the_oracle(lib, cuda, oracle, D, dtype, causal):
    for i, (B, H, Sq, Skv) in enumerate(SHAPES):
        # d = 256: from 1024 keys on
        assert fmha_plan(lib, dtype, B, H, Sq, Skv, D, causal)[0] == (FEW_ROWS if D != 256 or Skv >= 1024 else BLOCK)
        low, f32, scales = make_qkv(dtype, B, Sq, Skv, H, D, seed=500 + i)
        got, stats = run_fmha(lib, low, scales, dtype, causal)
        check(oracle, got, stats, f32, 1.0 / math.sqrt(D), causal, dtype)


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("Sq,Skv", [(30, 1040), (100, 1100)])
def test_bf16_rows_keep_the_two_term_p_of_their_whole_block(lib, cuda, oracle, D, Sq, Skv):
    """The first row sees fewer than 1024 keys, so P is a sum of two bf16 terms for every row of the call, as in the kernels with
    blocks of 256 (d = 256: 128) rows, also where a group of 16 rows begins above 1024.  The rounding of O to fp16 is then
    what is left, 2^-12 at most and about 2.0e-4 in the mean of squares; one bf16 term of P gives 1.5e-3."""
    assert fmha_plan(lib, 1, 1, 2, Sq, Skv, D, True)[0] == FEW_ROWS
    low, f32, scales = make_qkv(1, 1, Sq, Skv, 2, D, seed=Sq)
    got, _ = run_fmha(lib, low, scales, 1, True)
    want = oracle.attention(f32[0], f32[1], f32[2], 1.0 / math.sqrt(D), True)["o"]
    for row in range(0, Sq, 16):
        d, w = (got - want)[:, row:row + 16], want[:, row:row + 16]
        assert np.sqrt((d ** 2).sum() / (w ** 2).sum()) < 5e-4, row


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("causal", [False, True])
def test_few_rows_of_e4m3_keep_p_in_fp16(lib, cuda, oracle, D, causal):
    """With P in fp16 what is left are two roundings to 11 bits, of P and of O: 2^-10 together (P in e4m3: 2.6e-2)."""
    low, f32, scales = make_qkv(2, 2, 9, 1100, 2, D, seed=D)
    assert fmha_plan(lib, 2, 2, 2, 9, 1100, D, causal)[0] == FEW_ROWS
    got, _ = run_fmha(lib, low, scales, 2, causal)
    want = oracle.attention(f32[0], f32[1], f32[2], 1.0 / math.sqrt(D), causal)["o"]
    assert np.sqrt(((got - want) ** 2).sum() / (want ** 2).sum()) < 2.0 ** -10


@pytest.mark.parametrize("D", [64, 128])
def test_few_rows_hybrid_and_a_head_range_of_a_wider_tensor(lib, cuda, oracle, D):
    """e4m3 Q and K with fp16 V (the hybrid mode), heads 1 and 2 of five: strides of the whole tensor, and the other heads
    of O and everything behind the last row stay as they were."""
    B, H, HT, Sq, Skv = 2, 2, 5, 5, 700
    (q, k, _), (qf, kf, _), (qs, ks, _) = make_qkv(2, B, Sq, Skv, HT, D, seed=77)
    v = torch.randn(B, Skv, HT, D, generator=torch.Generator().manual_seed(78)).half()
    qd, kd, vd = q.cuda(), k.cuda(), v.cuda()
    o = torch.full((B, Sq, HT, D), -7.0, dtype=torch.float16, device="cuda")
    lse = torch.zeros(B, H, Sq, device="cuda")
    at = [t.data_ptr() + D * t.element_size() for t in (qd, kd, vd, o)]
    sq, skv = (Sq * HT * D, HT * D, D), (Skv * HT * D, HT * D, D)
    lib.fmha_forward(*at, dtype=2, batch=B, heads=H, seqlen_q=Sq, seqlen_kv=Skv, head_dim=D, softmax_scale=D ** -0.5,
                     causal=True, lse=lse, q_descale=qs, k_descale=ks, v_fp16=True, q_stride=sq, k_stride=skv,
                     v_stride=skv, o_stride=sq)
    lib.check_device()
    cut = lambda x: np.ascontiguousarray(x[:, :, 1:3])    # noqa: E731
    check(oracle, cut(o.float().cpu().numpy()), {}, (cut(qf), cut(kf), cut(v.float().numpy())), D ** -0.5, True, 0)
    rest = o.clone()
    rest[:, :, 1:3] = -7.0
    assert bool((rest == -7.0).all())


def test_few_rows_keep_large_steps_of_the_maximum(lib, cuda, oracle):
    """The running maximum moves by far more than the 2^8 it may lag, late and in one warp's keys only; a key whose scores
    are so low that its probability is zero changes nothing."""
    low, _, scales = make_qkv(0, 1, 2, 900, 1, 128, seed=9)
    q, k, v = low
    k[0, 850] = q[0, 0, 0:1] * 3
    k[0, 10] = -q[0, 0, 0:1] * 50
    f32 = [x.float().numpy() for x in (q, k, v)]
    got, stats = run_fmha(lib, (q, k, v), scales, 0, False)
    check(oracle, got, stats, f32, 1.0 / math.sqrt(128), False, 0)
