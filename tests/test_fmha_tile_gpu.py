"""Calls with too few 256-row blocks for the SMs run in a kernel with one 128-row tile per CTA.  With whole keys it does the
same arithmetic in the same order as the 256-row kernel (an explicit schedule selects that one), so the bits are equal; with
the keys split over a cluster it is compared with the oracle.  Sizes: edges of the 128-row and 128-key tiles, parts without a
visible key, ragged ends.  Tolerances are those of test_fmha_gpu.py."""
import math

import numpy as np
import pytest
import torch

from helpers import BLOCK, ONE_TILE, fmha_plan, make_qkv, run_fmha
from test_fmha_gpu import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,D", [(0, 64), (0, 128), (1, 64), (1, 128), (2, 64), (2, 128)])
@pytest.mark.parametrize("B,H,Sq,Skv", [(150, 2, 128, 128), (60, 5, 161, 257), (20, 15, 300, 300), (25, 4, 640, 640),
                                        (75, 4, 33, 385), (60, 3, 257, 385)])
@pytest.mark.parametrize("causal", [False, True])
def test_whole_keys_equal_the_256_row_kernel_bit_for_bit(lib, cuda, dtype, D, B, H, Sq, Skv, causal):
    from cfk_b200 import TUNE_FMHA_SCHED
    if (Sq, Skv) != (161, 257):            # which is beyond the rule for most types: the 256-row kernel on both sides
        assert fmha_plan(lib, dtype, B, H, Sq, Skv, D, causal) == (ONE_TILE, 1, 0, 0)
    low, _, scales = make_qkv(dtype, B, Sq, Skv, H, D, seed=B)
    got, stats = run_fmha(lib, low, scales, dtype, causal)
    try:
        lib.set_tunable(TUNE_FMHA_SCHED, 1 if dtype == 2 else 0)        # the defaults of the types
        assert fmha_plan(lib, dtype, B, H, Sq, Skv, D, causal) == (BLOCK, 0, 0, 0)
        want, wstats = run_fmha(lib, low, scales, dtype, causal)
    finally:
        lib.set_tunable(TUNE_FMHA_SCHED, -1)
    assert np.array_equal(got, want)
    for name in stats:
        assert np.array_equal(stats[name], wstats[name]), name


# parts of the keys per tile: 8, 8 (parts of one or two tiles), 4, 2, 8
@pytest.mark.parametrize("B,H,Sq,Skv", [(1, 4, 256, 2048), (1, 1, 777, 2100), (2, 4, 1024, 1024), (1, 8, 2048, 2048),
                                        (1, 2, 129, 1921)])
@pytest.mark.parametrize("dtype,D", [(0, 64), (0, 128), (1, 64), (1, 128), (2, 64), (2, 128)])
@pytest.mark.parametrize("causal", [False, True])
def test_split_keys_match_the_oracle(lib, cuda, oracle, dtype, D, B, H, Sq, Skv, causal):
    parts = {(256, 2048): 8, (777, 2100): 8, (1024, 1024): 4, (2048, 2048): 2, (129, 1921): 8}[Sq, Skv]
    assert fmha_plan(lib, dtype, B, H, Sq, Skv, D, causal) == (ONE_TILE, parts, 0, 0)
    low, f32, scales = make_qkv(dtype, B, Sq, Skv, H, D, seed=Skv)
    got, stats = run_fmha(lib, low, scales, dtype, causal)
    check(oracle, got, stats, f32, 1.0 / math.sqrt(D), causal, dtype)


def test_split_keys_with_low_scores_in_most_parts(lib, cuda, oracle):
    """Rows whose visible keys lie in the first part only, and scores hundreds of units apart between the parts: the weights
    of the other parts underflow to zero and must not reach the result."""
    low, _, scales = make_qkv(0, 1, 1024, 1024, 2, 128, seed=4)
    q, k, v = low
    k[0, 512:] *= 0.01
    k[0, :128] = q[0, :128] * 12
    f32 = [x.float().numpy() for x in (q, k, v)]
    for causal in (False, True):
        got, stats = run_fmha(lib, (q, k, v), scales, 0, causal)
        check(oracle, got, stats, f32, 1.0 / math.sqrt(128), causal, 0, max_abs=4e-3)


def very_negative(dtype, Sq, Skv, H, D, seed):
    """make_qkv with every scaled score near -120: Q around +c, K around -c in every element, c^2 sqrt(D) = 120."""
    low, _, _ = make_qkv(0, 1, Sq, Skv, H, D, seed=seed)
    c = math.sqrt(120 / math.sqrt(D))
    q, k, v = low[0].float() * 0.3 + c, low[1].float() * 0.3 - c, low[2].float()
    if dtype == 2:
        scales = [float(x.abs().max()) / 448.0 for x in (q, k, v)]
        low = [(x / s).to(torch.float8_e4m3fn) for x, s in zip((q, k, v), scales)]
    else:
        scales = [1.0, 1.0, 1.0]
        low = [x.to((torch.float16, torch.bfloat16)[dtype]) for x in (q, k, v)]
    return low, [(x.float() * s).numpy() for x, s in zip(low, scales)], scales


# Four parts, and a diagonal that falls into the middle of a key tile: the last tiles of a block are invisible to its first
# rows, so that a part has key tiles but no visible key for a row (84 and 204 pairs of row and part per head).
@pytest.mark.parametrize("Sq,Skv", [(1000, 1100), (900, 960)])
@pytest.mark.parametrize("dtype,D", [(0, 64), (0, 128), (1, 64), (1, 128), (2, 64), (2, 128)])
def test_parts_with_keys_but_none_visible_to_a_row_have_no_weight(lib, cuda, oracle, dtype, D, Sq, Skv):
    """Against maxima far below zero: such a part must not pass for one whose largest score is zero."""
    assert fmha_plan(lib, dtype, 1, 4, Sq, Skv, D, True) == (ONE_TILE, 4, 0, 0)
    low, f32, scales = very_negative(dtype, Sq, Skv, 4, D, seed=Sq)
    got, stats = run_fmha(lib, low, scales, dtype, True)
    check(oracle, got, stats, f32, 1.0 / math.sqrt(D), True, dtype)


@pytest.mark.parametrize("dtype", [0, 1])
def test_a_part_whose_scores_are_all_minus_infinity_has_no_weight(lib, cuda, oracle, dtype):
    """Keys 512 to 1023 (two of eight parts) at -inf against positive Q: as if they were not there, V included."""
    low, f32, scales = very_negative(dtype, 512, 2048, 4, 128, seed=3)
    low[1][:, 512:1024] = -math.inf
    got, stats = run_fmha(lib, low, scales, dtype, False)
    keep = np.r_[0:512, 1024:2048]
    check(oracle, got, stats, [f32[0], np.ascontiguousarray(f32[1][:, keep]), np.ascontiguousarray(f32[2][:, keep])],
          1.0 / math.sqrt(128), False, dtype)


@pytest.mark.parametrize("what", ["value of a key without weight", "value", "key", "query", "score"])
@pytest.mark.parametrize("bad", [math.nan, math.inf])
@pytest.mark.parametrize("dtype,Sq", [(0, 256), (1, 256), (0, 20), (1, 20)])
def test_nan_and_infinity_reach_the_outputs_they_reach_with_whole_keys(lib, cuda, dtype, Sq, bad, what):
    """Split keys (256 rows: eight parts of one tile; 20 rows: the few-rows kernel) against the 256-row kernel, which takes all
    keys of a row in order: the same elements of O and lse are finite.  Keys from 512 on score about -120, so that their
    probability is zero next to the others'."""
    from cfk_b200 import TUNE_FMHA_SCHED
    low, _, scales = very_negative(dtype, Sq, 2048, 2, 128, seed=1)
    q, k, v = low
    k[:, :512] = make_qkv(dtype, 1, Sq, 512, 2, 128, seed=2)[0][1] * 0.1
    if what == "value of a key without weight":
        v[0, 1000, 1, 5] = bad
    elif what == "value":
        v[0, 100, 1, 5] = bad
    elif what == "key":
        k[0, 1100, 0] = bad
    elif what == "query":
        q[0, 17, 1] = bad
    else:                                  # one score of +inf (NaN after the maximum is taken away)
        k[0, 1500, 0] = math.inf if bad == math.inf else 0
        k[0, 1500, 0, 0] = bad
    got, stats = run_fmha(lib, low, scales, dtype, False)
    try:
        lib.set_tunable(TUNE_FMHA_SCHED, 0)
        want, wstats = run_fmha(lib, low, scales, dtype, False)
    finally:
        lib.set_tunable(TUNE_FMHA_SCHED, -1)
    assert not np.isfinite(want).all()
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    assert np.array_equal(np.isfinite(stats["lse"]), np.isfinite(wstats["lse"]))


@pytest.mark.parametrize("D", [64, 128])
def test_hybrid_and_a_head_range_split(lib, cuda, oracle, D):
    """e4m3 Q and K with fp16 V, heads 1 and 2 of five, keys split: strides of the whole tensor; the rest of O stays."""
    B, H, HT, Sq, Skv = 1, 2, 5, 200, 1500
    (q, k, _), (qf, kf, _), (qs, ks, _) = make_qkv(2, B, Sq, Skv, HT, D, seed=77)
    v = torch.randn(B, Skv, HT, D, generator=torch.Generator().manual_seed(78)).half()
    qd, kd, vd = q.cuda(), k.cuda(), v.cuda()
    o = torch.full((B, Sq, HT, D), -7.0, dtype=torch.float16, device="cuda")
    at = [t.data_ptr() + D * t.element_size() for t in (qd, kd, vd, o)]
    sq, skv = (Sq * HT * D, HT * D, D), (Skv * HT * D, HT * D, D)
    lib.fmha_forward(*at, dtype=2, batch=B, heads=H, seqlen_q=Sq, seqlen_kv=Skv, head_dim=D, softmax_scale=D ** -0.5,
                     causal=True, q_descale=qs, k_descale=ks, v_fp16=True, q_stride=sq, k_stride=skv, v_stride=skv,
                     o_stride=sq)
    lib.check_device()
    cut = lambda x: np.ascontiguousarray(x[:, :, 1:3])    # noqa: E731
    check(oracle, cut(o.float().cpu().numpy()), {}, (cut(qf), cut(kf), cut(v.float().numpy())), D ** -0.5, True, 0)
    o[:, :, 1:3] = -7.0
    assert bool((o == -7.0).all())


# nine, one, two and 31 rows behind the last whole block, which without a mask run in the few-rows kernel as a second launch
@pytest.mark.parametrize("B,H,Sq,Skv,D", [(3, 16, 777, 1300, 128), (4, 3, 3073, 1000, 128), (12, 1, 3074, 2600, 64),
                                          (12, 1, 3103, 2600, 128)])
@pytest.mark.parametrize("dtype", [0, 1, 2])
def test_a_short_remainder_of_rows_matches_the_oracle(lib, cuda, oracle, dtype, B, H, Sq, Skv, D):
    plan = fmha_plan(lib, dtype, B, H, Sq, Skv, D, False)
    rest = Sq % (256 if plan[0] == BLOCK else 128)
    assert plan[2] == rest
    low, f32, scales = make_qkv(dtype, B, Sq, Skv, H, D, seed=Sq)
    got, stats = run_fmha(lib, low, scales, dtype, False)
    pick = np.random.default_rng(Sq).permutation(B)[:2]      # two batch entries; the others have the same rows
    check(oracle, got[pick], {k: v[pick] for k, v in stats.items()}, [x[pick] for x in f32], 1.0 / math.sqrt(D), False, dtype)
    # the remainder of every entry, which is the second launch, and that every row of the others was written
    check(oracle, got[:, -rest:], {k: v[:, :, -rest:] for k, v in stats.items()},
          [np.ascontiguousarray(f32[0][:, -rest:]), f32[1], f32[2]], 1.0 / math.sqrt(D), False, dtype)
    assert np.isfinite(got).all() and (got != -1.0).any(axis=3).all()
