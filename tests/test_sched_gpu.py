"""The varlen tile scheduler on the GPU: the device-built work list against the host version of
the same rule, parity of the attention kernels on skewed length mixes (where the list order
matters most), and the device-side validation of cu_seqlens."""

import numpy as np
import pytest
import torch

import nanobrain_b200
from nanobrain_b200 import _lib, ops, schedule
from nanobrain_b200 import workloads as W
from oracle import attn_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"
MAX_ABS, MEAN_ABS = 2e-2, 2e-3


def lists(lengths_q, lengths_k, side, total_q=None, total_k=None, max_q=None, max_k=None):
    lq, lk = torch.tensor(lengths_q), torch.tensor(lengths_k)
    cu_q, cu_k = W.cu_seqlens_from_lengths(lq), W.cu_seqlens_from_lengths(lk)
    args = (max_q or int(lq.max()), max_k or int(lk.max()), total_q or int(lq.sum()), total_k or int(lk.sum()))
    host = schedule.work_list_host(cu_q, cu_k, *args, side)
    dev, status = schedule.work_list_device(cu_q.to(DEV), cu_k.to(DEV), *args, 12, side)
    torch.cuda.synchronize()
    return host, dev.cpu(), int(status[0])


@pytest.mark.parametrize("lengths", [
    [820], [1], [127, 129, 256, 1, 0, 700], [200] * 30 + [2000],
    W.draw_lengths(W.WORKLOADS["vitb_encoder_varlen"]).tolist(),
    torch.randint(0, 3000, (1500,), generator=torch.Generator().manual_seed(1)).tolist(),
])
def test_device_list_equals_host_list_up_to_order_inside_a_cost_class(lengths):
    for side in (0, 1):
        host, dev, status = lists(lengths, lengths, side)
        assert status == 0 and host.shape == dev.shape
        h, d = schedule.decode(host), schedule.decode(dev)
        assert sorted(h) == sorted(d)                                  # the same items, each once
        n_used = len(h)
        assert bool((dev[n_used:, 0] < 0).all())                       # unused entries at the end
        assert sorted(map(tuple, host[:n_used].tolist())) == sorted(map(tuple, dev[:n_used].tolist()))
        # same cost (steps) and same kind (full before ragged) at every position
        steps = [(l + 127) // 128 for l in lengths] + [0]
        lens = list(lengths) + [0]
        kind = lambda it: (steps[it[0]], it[1] == lens[it[0]] // 128 and lens[it[0]] % 128 != 0)
        assert [kind(x) for x in h] == [kind(x) for x in d]


def test_device_list_with_cross_lengths_and_spare_rows():
    host, dev, status = lists([130, 5, 64], [3, 900, 129], 1, total_q=400, total_k=2000)
    assert status == 0 and sorted(schedule.decode(host)) == sorted(schedule.decode(dev))
    assert (3, 0) in schedule.decode(dev)                               # the rows past the last sequence


@pytest.mark.parametrize("case", ["too_long", "beyond_total", "decreasing"])
def test_invalid_cu_seqlens_are_reported_and_nothing_runs(case):
    lengths = torch.tensor([100, 200])
    cu = W.cu_seqlens_from_lengths(lengths)
    max_len, total = 200, 300
    if case == "too_long":
        max_len = 150          # max_seqlen must be a true upper bound: no tile is silently dropped
    elif case == "beyond_total":
        total = 299
    else:
        cu = torch.tensor([0, 200, 100], dtype=torch.int32)
    _, status = schedule.work_list_device(cu.to(DEV), cu.to(DEV), max_len, max_len, total, total, 2, 0)
    torch.cuda.synchronize()
    assert int(status[0]) == _lib.STATUS_BAD_SEQLENS
    # through the op: the kernels leave the outputs alone and the next call (or check_status) raises
    t = torch.randn(300, 2, 64, device=DEV).to(torch.bfloat16)
    cud = cu.to(DEV)
    out, _ = ops.sdpa_varlen_fwd(t[:total], t[:total], t[:total], cud, cud, max_len, max_len, 0.125)
    with pytest.raises(RuntimeError, match="cu_seqlens"):
        ops.check_status()
    ops.check_status()         # the word was cleared by the raise
    out = nanobrain_b200.sdpa_varlen(t, t, t, W.cu_seqlens_from_lengths(lengths).to(DEV),
                                     W.cu_seqlens_from_lengths(lengths).to(DEV), 200, 200)
    ops.check_status()
    assert torch.isfinite(out.float()).all()


def run_varlen(lengths, heads, seed):
    q, k, v, g = (t.to(torch.bfloat16).float() for t in W.make_packed_inputs(lengths, heads, seed=seed))
    cu = W.cu_seqlens_from_lengths(lengths)
    qd, kd, vd = (t.to(DEV, torch.bfloat16).requires_grad_(True) for t in (q, k, v))
    out = nanobrain_b200.sdpa_varlen(qd, kd, vd, cu.to(DEV), cu.to(DEV), int(lengths.max()), int(lengths.max()))
    out.backward(g.to(DEV, torch.bfloat16))
    ops.check_status()
    want = O.varlen_fwd_bwd(q.numpy(), k.numpy(), v.numpy(), g.numpy(), cu.numpy(), cu.numpy(), dtype=np.float32)
    return (out, qd.grad, kd.grad, vd.grad), (want[0], want[2], want[3], want[4])


@pytest.mark.parametrize("lengths", [
    [200] * 30 + [2000],                   # one long sequence among many short ones
    [2000] + [200] * 30,
    [16, 1500, 17, 129, 640, 15, 1, 128],  # ragged tiles of every size next to full ones
    [129, 130, 144, 145, 820],             # lengths around the 16-row trimming granularity
])
def test_skewed_length_mixes_match_the_oracle(lengths):
    got, want = run_varlen(torch.tensor(lengths), heads=2, seed=len(lengths))
    for name, a, b in zip(("out", "dq", "dk", "dv"), got, want):
        err = np.abs(a.detach().float().cpu().numpy() - b)
        assert np.isfinite(err).all(), name
        assert err.max() <= MAX_ABS * max(1.0, np.abs(b).max()) and err.mean() <= MEAN_ABS, (name, err.max(), err.mean())


def test_many_short_units_per_persistent_cta_match_the_oracle():
    # 500 sequences of 1..300 tokens and 3 heads: about 2400 backward work units of one, two or three
    # steps for the 148 persistent CTAs, so that every CTA runs a dozen units back to back (K buffer
    # alternation, one-step units, dV / dK leaving while the next unit has started) and the forward
    # runs several waves of short CTAs.
    g = torch.Generator().manual_seed(7)
    lengths = torch.randint(1, 301, (500,), generator=g)
    got, want = run_varlen(lengths, heads=3, seed=11)
    for name, a, b in zip(("out", "dq", "dk", "dv"), got, want):
        err = np.abs(a.detach().float().cpu().numpy() - b)
        assert np.isfinite(err).all(), name
        assert err.max() <= MAX_ABS * max(1.0, np.abs(b).max()) and err.mean() <= MEAN_ABS, (name, err.max(), err.mean())



@pytest.mark.parametrize("lengths,spare", [
    ([820], 0), ([127, 129, 256, 1, 0, 700], 0), ([200] * 30 + [2000], 70),
    (torch.randint(0, 1500, (400,), generator=torch.Generator().manual_seed(2)).tolist(), 300),
])
def test_the_lists_that_the_calls_build(lengths, spare):
    # What a forward and a backward leave in their workspaces: every tile once, most expensive first, in one cost class
    # the full tiles before the ragged ones, the first entry's counters as in a new list (forward).
    import ctypes as C

    heads, total = 2, sum(lengths) + spare
    g = torch.Generator(device=DEV).manual_seed(len(lengths))
    q, k, v, d_out = (torch.randn(total, heads, 64, generator=g, device=DEV).to(torch.bfloat16) for _ in range(4))
    out, dq, dk, dv = (torch.empty_like(q) for _ in range(4))
    lse = torch.empty(heads, total, device=DEV)
    cu = torch.tensor([0] + lengths).cumsum(0).to(DEV, torch.int32)
    shape = _lib.Shape(len(lengths), heads, 64, max(lengths), max(lengths), total, total, cu.data_ptr(), cu.data_ptr(), 0.125)
    fwd_ws = torch.empty(_lib.fwd_workspace_bytes(shape), dtype=torch.uint8, device=DEV)
    bwd_ws = torch.empty(_lib.bwd_workspace_bytes(shape), dtype=torch.uint8, device=DEV)
    d = lambda t: _lib.Tensor(t.data_ptr(), 0, t.stride(0), t.stride(1))
    lib, stream = _lib.load(), C.c_void_p(torch.cuda.current_stream().cuda_stream)
    fwd = _lib.FwdArgs(shape, d(q), d(k), d(v), d(out), lse.data_ptr(), None, fwd_ws.data_ptr(), fwd_ws.numel())
    bwd = _lib.BwdArgs(shape, d(q), d(k), d(v), d(out), d(d_out), d(dq), d(dk), d(dv), lse.data_ptr(), bwd_ws.data_ptr(),
                       bwd_ws.numel(), None, None, None)
    _lib.check(lib.nb_attn_fwd(C.byref(fwd), stream), "nb_attn_fwd")
    _lib.check(lib.nb_attn_bwd(C.byref(bwd), stream), "nb_attn_bwd")
    torch.cuda.synchronize()
    n = schedule.capacity(total, len(lengths))
    lists_ = [fwd_ws.view(torch.int32).reshape(-1, 8), bwd_ws[-n * 32:].view(torch.int32).reshape(-1, 8)]
    starts = cu.tolist()
    own = list(lengths) + [spare]
    cost = [(length + 127) // 128 for length in lengths] + [0]
    want = [(i, t) for i, length in enumerate(own) for t in range((length + 127) // 128)]
    for items in lists_:
        rows = items.cpu().tolist()
        used = [r for r in rows if r[0] >= 0]
        assert rows[:len(used)] == used and len(rows) == n             # unused entries at the end
        assert sorted((r[0], r[1]) for r in used) == want              # every tile, once
        for seq, _, own_begin, own_len, other_begin, other_len, *_ in used:
            assert (own_begin, own_len) == (starts[seq], own[seq])
            assert seq == len(lengths) or (other_begin, other_len) == (starts[seq], lengths[seq])
        order = [(-cost[r[0]], r[1] == own[r[0]] // 128) for r in used]  # (cost class, ragged)
        assert order == sorted(order)
        assert all(r[6:] == [0, 0] for r in rows[1:])
    assert lists_[0][0, 6:].tolist() == [0, 0]
