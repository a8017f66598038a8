"""The backward where one CTA takes all key tiles of a (sequence, head) and sums dQ up in tiles of its
own, next to sequences whose key tiles are spread over the CTAs, against the CPU oracle."""

import ctypes as C

import numpy as np
import pytest
import torch

import nanobrain_b200
from nanobrain_b200 import _lib, ops
from oracle import attn_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def check(names, got, want):
    # bf16 results of bf16 products with fp32 accumulation, as for every other configuration
    for name, a, b in zip(names, got, want):
        b = np.asarray(b, dtype=np.float32)
        err = np.abs(a.detach().float().cpu().numpy() - b)
        assert np.isfinite(err).all(), name
        assert err.max() <= 2e-2 * max(1.0, np.abs(b).max()) and err.mean() <= 2e-3 * max(1.0, np.abs(b).max()), name


@pytest.mark.parametrize("lengths_q,lengths_k,heads,spare", [
    ([200] * 14 + [700], None, 100, 0),                       # two query tiles: neighbouring additions to a tile
    ([130, 0, 256, 257, 1, 128, 140, 500] * 3, None, 100, 70),  # all kinds, and rows past the last sequence
    ([1153, 1100], [150, 129], 400, 0),                       # nine and ten
    ([300] * 5, None, 170, 1),                                # 5.7 rounds over the SMs: the last sequence is single tiles
    ([64, 1, 128, 0, 100], None, 120, 30),                    # one tile at most
    ([300, 100, 0, 260, 128] * 4, [50, 400, 200, 0, 129] * 4, 150, 5),
    ([140] * 3, [1000, 1024, 513], 210, 0),                   # more key than query tiles
    ([1300, 900, 1024], [140, 130, 129], 200, 0),             # more query tiles than a CTA keeps, and as many
])
def test_packed_runs(lengths_q, lengths_k, heads, spare):
    lengths_k = lengths_q if lengths_k is None else lengths_k
    g = torch.Generator().manual_seed(sum(lengths_q))
    tq, tk = sum(lengths_q) + spare, sum(lengths_k) + spare
    # Calls of fewer steps are spread over the CTAs altogether.
    assert max(lengths_k) <= 128 or tq * tk * heads >= 30 * 148 * 128 ** 2 * len(lengths_q)
    q, d_out = (torch.randn(tq, heads, 64, generator=g).to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(tk, heads, 64, generator=g).to(torch.bfloat16) for _ in range(2))
    cu_q, cu_k = (torch.tensor([0] + list(x)).cumsum(0).to(DEV, torch.int32) for x in (lengths_q, lengths_k))
    want = [np.zeros((n, heads, 64), np.float32) for n in (tq, tk, tk)]
    at_q = at_k = 0
    for nq, nk in zip(lengths_q, lengths_k):
        if nq and nk:
            sq, sk = slice(at_q, at_q + nq), slice(at_k, at_k + nk)
            one = lambda t, s: t[s].float().numpy().transpose(1, 0, 2)[None]
            grads = O.sdpa_fwd_bwd(one(q, sq), one(k, sk), one(v, sk), one(d_out, sq))[2:5]
            for w, s, x in zip(want, (sq, sk, sk), grads):
                w[s] = x[0].transpose(1, 0, 2)
        at_q, at_k = at_q + nq, at_k + nk
    for _ in range(2):
        qd, kd, vd = (t.to(DEV).requires_grad_(True) for t in (q, k, v))
        out = nanobrain_b200.sdpa_varlen(qd, kd, vd, cu_q, cu_k, max(lengths_q), max(lengths_k))
        out.backward(d_out.to(DEV))
        ops.check_status()
        check(("dq", "dk", "dv"), (qd.grad, kd.grad, vd.grad), want)


def test_an_invalid_packing_is_reported_and_nothing_runs():
    # The rule for runs is looked for before the packing is known to be one.
    heads, n = 200, 8
    t = torch.randn(n * 300, heads, 64, device=DEV).to(torch.bfloat16)
    good = torch.arange(0, n * 300 + 1, 300, dtype=torch.int32, device=DEV)
    bad = good.clone()
    bad[3], bad[4] = 1300, 900
    out, lse = ops.sdpa_varlen_fwd(t, t, t, good, good, 300, 300, 0.125)
    dq, _, _ = ops.sdpa_varlen_bwd(t, t, t, t, out, lse, bad, bad, 400, 400, 0.125)
    with pytest.raises(RuntimeError, match="cu_seqlens"):
        ops.check_status()
    assert int(dq.count_nonzero()) == 0
    ops.sdpa_varlen_bwd(t, t, t, t, out, lse, good, good, 300, 300, 0.125)
    ops.check_status()


def backward(lengths_q, lengths_k, heads, lead=0, spare=0, full=True):
    """Forward and backward of random packed sequences through the C ABI, ``lead`` rows before the first and ``spare`` behind
    the last, with the larger workspace or the one that a call has to have. dQ, dK and dV start as NaN."""
    cu_q, cu_k = (torch.tensor([lead] + list(x)).cumsum(0).to(DEV, torch.int32) for x in (lengths_q, lengths_k))
    tq, tk = lead + sum(lengths_q) + spare, lead + sum(lengths_k) + spare
    g = torch.Generator(device=DEV).manual_seed(tq + tk)
    q, d_out = (torch.randn(tq, heads, 64, generator=g, device=DEV).to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(tk, heads, 64, generator=g, device=DEV).to(torch.bfloat16) for _ in range(2))
    out, lse = ops.sdpa_varlen_fwd(q, k, v, cu_q, cu_k, max(lengths_q), max(lengths_k), 0.125)
    dq, dk, dv = (torch.full_like(t, float("nan")) for t in (q, k, v))
    shape = _lib.Shape(len(lengths_q), heads, 64, max(lengths_q), max(lengths_k), tq, tk, cu_q.data_ptr(), cu_k.data_ptr(),
                       0.125)
    least, most = _lib.bwd_workspace_bytes(shape), _lib.bwd_full_workspace_bytes(shape)
    assert most > least  # the larger one is for runs
    ws = torch.empty(most if full else least, dtype=torch.uint8, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    d = lambda t: _lib.Tensor(t.data_ptr(), 0, t.stride(0), t.stride(1))
    args = _lib.BwdArgs(shape, d(q), d(k), d(v), d(out), d(d_out), d(dq), d(dk), d(dv), lse.data_ptr(), ws.data_ptr(),
                        ws.numel(), status.data_ptr(), None, None)
    _lib.check(_lib.load().nb_attn_bwd(C.byref(args), C.c_void_p(torch.cuda.current_stream().cuda_stream)), "nb_attn_bwd")
    assert int(status.item()) == 0
    return dq, dk, dv


@pytest.mark.parametrize("lengths", [[200] * 14 + [700], [1500] + [200] * 20])  # the first one is a run, or single tiles
def test_dq_of_rows_before_the_first_sequence_is_zero(lengths):
    for full in (False, True):
        dq, dk, dv = backward(lengths, lengths, 100, lead=70, spare=33, full=full)
        assert int(dq[:70].count_nonzero()) == 0 and int(dq[-33:].count_nonzero()) == 0
        assert torch.isfinite(dq.float()).all()
        assert torch.isfinite(dk[70:].float()).all() and torch.isfinite(dv[70:].float()).all()


@pytest.mark.parametrize("lengths,heads,spare,runs", [
    ([200] * 45, 12, 9000, False),     # nine steps per SM, 36 if the spare rows were sequences
    ([200] * 45, 12, 0, False),
    ([200] * 140, 12, 14000, True),    # 28 steps per SM, 63 if they were
    ([200] * 300, 12, 0, True),
    ([200] * 300, 12, 400000, True),   # eleven tiles per sequence if they were
])
def test_spare_rows_do_not_decide_about_runs(lengths, heads, spare, runs):
    total = sum(lengths) + spare
    cu = torch.zeros(len(lengths) + 1, dtype=torch.int32, device=DEV)
    shape = _lib.Shape(len(lengths), heads, 64, max(lengths), max(lengths), total, total, cu.data_ptr(), cu.data_ptr(), 0.125)
    assert (_lib.load().nb_attn_bwd_split_workspace_bytes(C.byref(shape)) > 0) == runs
