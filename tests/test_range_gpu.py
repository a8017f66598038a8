"""The forward on scores and values of unusual size: far above the exponent's offset, infinite, NaN."""

import numpy as np
import pytest
import torch

from nanobrain_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def bf16(*shape, seed, mul=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * mul).to(torch.bfloat16)


def exact_forward(q, k, v, scale=0.125):
    q, k, v = q.double(), k.double(), v.double()
    s = q @ k.transpose(-1, -2) * scale
    return torch.softmax(s, -1) @ v, torch.logsumexp(s, -1)


@pytest.mark.parametrize("lk", [256, 300])
@pytest.mark.parametrize("score", [100.0, 200.0, 500.0])
def test_one_key_far_above_the_first_ones_takes_all_the_weight(lk, score):
    # One sequence per column at which the dominating key can be: every score is 0 but that one, so the
    # output is that key's value (exp(-100) of the others), exactly.
    cols = lk - 64
    q = torch.zeros(cols, 1, 70, 64, device=DEV, dtype=torch.bfloat16)
    q[..., 0] = 8.0
    k = torch.zeros(cols, 1, lk, 64, device=DEV, dtype=torch.bfloat16)
    k[torch.arange(cols), 0, torch.arange(cols) + 64, 0] = score
    v = torch.arange(lk, device=DEV, dtype=torch.float32)[None, None, :, None].expand(cols, 1, lk, 64).to(torch.bfloat16)
    out, lse = ops.sdpa_fwd(q, k, v, 0.125)
    ops.check_status()
    want = v[0, 0, 64:, 0][:, None, None, None].expand_as(out)
    assert torch.equal(out, want), torch.nonzero((out != want).any(-1).any(-1).any(-1)).flatten().tolist()
    # (fp32 of a score of 722 in log2 units: half a unit in the last place is 3e-5)
    np.testing.assert_allclose(lse.cpu().numpy(), score, rtol=1e-6, atol=0)


def test_a_nan_key_row_shows_in_every_query_row():
    lk = 200
    q = bf16(lk, 1, 70, 64, seed=1)
    k, v = bf16(lk, 1, lk, 64, seed=2), bf16(lk, 1, lk, 64, seed=3)
    k[torch.arange(lk), 0, torch.arange(lk)] = float("nan")
    out, lse = ops.sdpa_fwd(q, k, v, 0.125)
    ops.check_status()
    seen = torch.isnan(out).all(-1).all(-1).all(-1) & torch.isnan(lse).all(-1).all(-1)
    assert bool(seen.all()), torch.nonzero(~seen).flatten().tolist()


def test_bias_of_the_log_sum_exp():
    # The polynomial's error is 5.1e-6 on average (7.5e-5 at most), for one key in eight: a bias of 6.4e-7
    # over many keys, to which the roundings of fp32 sums (unbiased) add little.
    q, k, v = (bf16(2, 8, 4096, 64, seed=s) for s in (4, 5, 6))
    lse = ops.sdpa_fwd(q, k, v, 0.125)[1]
    err = lse.double() - exact_forward(q, k, v)[1]
    assert abs(float(err.mean())) <= 8.5e-7 and float(err.pow(2).mean().sqrt()) <= 1.1e-6


@pytest.mark.parametrize("shape,mul", [((4, 8, 128), 1.0), ((2, 4, 820), 1.0), ((2, 4, 300), 3.0), ((2, 4, 1000), 4.0), ((1, 2, 3476), 3.0)])
def test_rounding_of_p_weighs_little_where_one_key_dominates(shape, mul):
    # P is rounded to bf16 (relative error d_j of key j, independent, 2^-8 at most) and O is divided by the sum of
    # the same rounded values, so its error is sum_j w_j d_j (v_j - O), plus its own rounding to bf16. A
    # relative rounding error of a number with evenly spread logarithm has the variance 2^-14 / 12 x 0.541
    # (spacing 2^-7 at 1, and the mean of 1 / m^2 over its mantissas m).
    q, k = (bf16(*shape, 64, seed=s, mul=mul) for s in (7, 8))
    v = bf16(*shape, 64, seed=9)
    out = ops.sdpa_fwd(q, k, v, 0.125)[0].double()
    want = exact_forward(q, k, v)[0]
    w = torch.softmax(q.double() @ k.double().transpose(-1, -2) * 0.125, -1)
    v = v.double()
    spread = (w**2) @ v**2 - 2 * ((w**2) @ v) * want + (w**2).sum(-1, keepdim=True) * want**2
    rounding = (want.to(torch.bfloat16).double() - want) ** 2
    bound = (spread.sum() * 2.0**-14 / 12 * 0.541 + rounding.sum()).sqrt() / want.norm()
    assert float((out - want).norm() / want.norm()) <= 1.05 * float(bound)


@pytest.mark.parametrize("lk", [512, 4000])  # the second one is cut between CTAs
@pytest.mark.parametrize("exponent", [60, 90, 112])
def test_large_values_behind_rising_scores(exponent, lk):
    # P of the keys 35 nats above the first ones is 2^50: times V that is beyond fp32, the result is not.
    q = torch.zeros(1, 1, 140, 64, device=DEV, dtype=torch.bfloat16)
    q[..., 0] = 8.0
    k = torch.zeros(1, 1, lk, 64, device=DEV, dtype=torch.bfloat16)
    k[0, 0, 300:302, 0], k[0, 0, 70, 0] = 35.0, 20.0
    v = torch.full((1, 1, lk, 64), 2.0**exponent, device=DEV).to(torch.bfloat16)
    out = ops.sdpa_fwd(q, k, v, 0.125)[0]
    ops.check_status()
    assert torch.equal(out, v[:, :, :1].expand_as(out))


@pytest.mark.parametrize("lk,first", [(256, 64), (256, 128), (256, 200), (300, 17), (4096, 128), (4096, 2100)])
def test_scores_of_minus_infinity_have_no_weight(lk, first):
    # q.k of the first keys is below fp32's range, all other scores are 0. (4096: cut between CTAs.)
    q = torch.full((1, 1, 128, 64), 1e30, device=DEV, dtype=torch.bfloat16)
    k = torch.zeros(1, 1, lk, 64, device=DEV, dtype=torch.bfloat16)
    k[0, 0, :first] = -1e30
    v = bf16(1, 1, lk, 64, seed=10)
    out, lse = ops.sdpa_fwd(q, k, v, 0.125)
    ops.check_status()
    want = v[0, 0, first:].double().mean(0)
    # P = 1 exactly, so O has its own rounding to bf16 alone: half of a spacing of 2^-7 at most
    assert bool(((out.double() - want).abs() <= 2.0**-8 * 1.001 * want.abs()).all())
    # the polynomial gives 1 - 7.2e-5 at 0, for at most one in seven of the keys that are left: 1.03e-5
    np.testing.assert_allclose(lse.cpu().numpy(), np.log(lk - first), rtol=0, atol=1.2e-5)
