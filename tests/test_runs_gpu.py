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
SENTINEL = -12345.0


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


def packed_shape(lengths_q, lengths_k, heads, cu_q, cu_k, lead=0, spare=0):
    return _lib.Shape(len(lengths_q), heads, 64, max(lengths_q), max(lengths_k), lead + sum(lengths_q) + spare,
                      lead + sum(lengths_k) + spare, cu_q.data_ptr(), cu_k.data_ptr(), 0.125)


def in_a_frame(t):
    """``t`` in memory with a gap behind every token and 8 tokens of it before and after; and that memory."""
    rows, width = t.shape[0], t.shape[1] * 64
    frame = torch.full((rows + 16, width + 64), SENTINEL, dtype=torch.bfloat16, device=DEV)
    view = frame[8:8 + rows, :width].unflatten(1, (-1, 64))
    view.copy_(t)
    return view, frame


def backward(lengths_q, lengths_k, heads, lead=0, spare=0, full=True, frames=False):
    """Forward and backward of random packed sequences through the C ABI, ``lead`` rows before the first and ``spare`` behind
    the last, with the larger workspace or the one that a call has to have; ``frames``: all tensors and the workspace
    inside of memory that nobody may write. dQ, dK and dV start as NaN. Returns them and the workspace."""
    cu_q, cu_k = (torch.tensor([lead] + list(x)).cumsum(0).to(DEV, torch.int32) for x in (lengths_q, lengths_k))
    shape = packed_shape(lengths_q, lengths_k, heads, cu_q, cu_k, lead, spare)
    tq, tk = shape.total_q, shape.total_k
    g = torch.Generator(device=DEV).manual_seed(tq + tk)
    q, d_out = (torch.randn(tq, heads, 64, generator=g, device=DEV).to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(tk, heads, 64, generator=g, device=DEV).to(torch.bfloat16) for _ in range(2))
    out, lse = ops.sdpa_varlen_fwd(q, k, v, cu_q, cu_k, max(lengths_q), max(lengths_k), 0.125)
    dq, dk, dv = (torch.full_like(t, float("nan")) for t in (q, k, v))
    tensors, around = [q, k, v, out, d_out, dq, dk, dv], []
    if frames:
        tensors, around = zip(*map(in_a_frame, tensors))
    least, most = _lib.bwd_workspace_bytes(shape), _lib.bwd_full_workspace_bytes(shape)
    assert most > least  # the larger one is for runs
    n = most if full else least
    ws_frame = torch.full((n + 8192,), 0xA5, dtype=torch.uint8, device=DEV)
    ws = ws_frame[4096:4096 + n]
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    descs = [_lib.Tensor(t.data_ptr(), 0, t.stride(0), t.stride(1)) for t in tensors]
    args = _lib.BwdArgs(shape, *descs, lse.data_ptr(), ws.data_ptr(), n, status.data_ptr(), None, None)
    _lib.check(_lib.load().nb_attn_bwd(C.byref(args), C.c_void_p(torch.cuda.current_stream().cuda_stream)), "nb_attn_bwd")
    assert int(status.item()) == 0
    assert bool((ws_frame[:4096] == 0xA5).all() and (ws_frame[4096 + n:] == 0xA5).all())
    for view, frame in zip(tensors, around):
        view_of = torch.zeros_like(frame, dtype=torch.bool)
        view_of[8:8 + view.shape[0], :heads * 64] = True
        assert bool((frame[~view_of] == torch.tensor(SENTINEL, dtype=torch.bfloat16)).all())
    return *tensors[5:], ws


def runs_of(lengths_q, lengths_k, heads):
    """The sequences that are runs: the rule of the library, for packings that may have runs."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles_q, tiles_k = ([(n + 127) // 128 for n in x] for x in (lengths_q, lengths_k))
    single = {i for i, (a, b) in enumerate(zip(tiles_q, tiles_k)) if b == 1 and a}
    if max(tiles_k) == 1:
        return single
    most = min(max(tiles_q), 10 if len(lengths_q) * heads >= 5 * sms else 9)
    share = sum(a * b for a, b in zip(tiles_q, tiles_k)) * heads // sms
    cost = {i: a * b for i, (a, b) in enumerate(zip(tiles_q, tiles_k)) if 1 < a <= most and b > 1 and a * b <= share}
    if not cost:
        return single
    average = -(-sum(cost.values()) // len(cost))
    rounds = share // average
    if rounds and share - rounds * average < average // 2:
        rounds -= 1
    budget = max(rounds * average, share // max(cost.values()) * max(cost.values())) * sms // heads
    used, runs = 0, set(single)
    for i in sorted(cost):
        used += cost[i]
        if used > budget:
            break
        runs.add(i)
    return runs


def check_lists(ws, lengths_q, lengths_k, heads, lead, spare, runs):
    """The work list and the list of the rows of no run that a backward has left in its workspace."""
    tq, tk = lead + sum(lengths_q) + spare, lead + sum(lengths_k) + spare
    up = lambda n: (n + 255) // 256 * 256
    at, n = up(tq * heads * 260), (tk // 128 + len(lengths_k) + 1) * 32
    items = ws[at:at + n].view(torch.int32).reshape(-1, 8).cpu().tolist()
    tiles = [(i, t) for i, k in enumerate(list(lengths_k) + [spare]) if i not in runs for t in range((k + 127) // 128)]
    assert sorted((seq, tile) for seq, tile, *_ in items if seq >= 0) == sorted(tiles + [(i, -1) for i in runs])
    at = up(at + n)
    words = ws[at:at + 16 + 8 * (len(lengths_q) + 1)].view(torch.int32).cpu().tolist()
    rest, begin = list(range(lead)), lead
    for i, length in enumerate(list(lengths_q) + [spare]):
        if i not in runs:
            rest += range(begin, begin + length)
        begin += length
    got, x = [], 0
    for end, shift in zip(words[4::2], words[5::2]):
        got += range(x + shift, end + shift)
        x = max(x, end)
    assert words[0] == len(rest) and got == rest


@pytest.mark.parametrize("lengths", [[200] * 14 + [700], [1500] + [200] * 20])  # the first one is a run, or single tiles
def test_dq_of_rows_before_the_first_sequence_is_zero(lengths):
    for full in (False, True):
        dq, dk, dv, _ = backward(lengths, lengths, 100, lead=70, spare=33, full=full)
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
    cu = torch.zeros(len(lengths) + 1, dtype=torch.int32, device=DEV)
    shape = packed_shape(lengths, lengths, heads, cu, cu, spare=spare)
    assert (_lib.load().nb_attn_bwd_split_workspace_bytes(C.byref(shape)) > 0) == runs


CASES = [  # query lengths, key lengths (None: the same), heads, rows before and behind
    ([600] * 3, None, 150, 0, 0),                                      # five query tiles: the least room between additions
    ([700, 640, 650], [700, 1500, 1400], 150, 0, 9),                   # six and five, more key tiles than that
    ([300, 384, 257], [1000, 900, 1100], 150, 0, 0),                   # three, the same
    ([850, 790, 800], None, 150, 40, 40),                              # seven
    ([1100, 1152, 1030], None, 150, 0, 0),                             # nine
    ([1280, 1200, 1153, 1250], None, 200, 0, 0),                       # ten
    ([300, 0, 260, 140, 513, 1] * 4, [200, 130, 0, 300, 700, 129] * 4, 60, 5, 300),
    ([130 + 41 * i % 171 for i in range(30)], None, 100, 0, 1),
    ([100 + 37 * i % 301 for i in range(600)], None, 4, 3, 70),        # more sequences than a block has threads
    ([150 + i % 3 for i in range(2048)], None, 2, 0, 0),               # as many as may have runs
]


@pytest.mark.parametrize("lengths_q,lengths_k,heads,lead,spare", CASES)
def test_runs_against_single_tiles(lengths_q, lengths_k, heads, lead, spare):
    lengths_k = lengths_q if lengths_k is None else lengths_k
    runs = runs_of(lengths_q, lengths_k, heads)
    assert any(lengths_k[i] > 128 for i in runs)
    *want, _ = backward(lengths_q, lengths_k, heads, lead, spare, full=False)
    for frames in (False, True):
        *got, ws = backward(lengths_q, lengths_k, heads, lead, spare, frames=frames)
        check_lists(ws, lengths_q, lengths_k, heads, lead, spare, runs)
        assert torch.equal(got[1][lead:], want[1][lead:]) and torch.equal(got[2][lead:], want[2][lead:])
        # The same fp32 terms added up in another order, rounded to bf16: neighbouring values at most.
        a, b = got[0].float(), want[0].float()
        assert torch.isfinite(a).all() and bool(((a - b).abs() <= 2.0 ** -7 * b.abs() + 1e-4).all())


def test_packings_of_more_sequences_have_no_runs():
    cu = torch.zeros(2050, dtype=torch.int32, device=DEV)
    for n, runs in ((2048, True), (2049, False)):
        shape = packed_shape([150] * n, [150] * n, 2, cu, cu)
        assert (_lib.load().nb_attn_bwd_split_workspace_bytes(C.byref(shape)) > 0) == runs


def test_a_captured_backward_decides_about_runs_on_every_replay():
    heads, total, most = 100, 20 * 300, 700
    g = torch.Generator(device=DEV).manual_seed(5)
    q, k, v, d_out = (torch.randn(total, heads, 64, generator=g, device=DEV).to(torch.bfloat16) for _ in range(4))
    packings = [[300] * 20, [500, 100] * 10, [130, 700] + [300] * 16 + [170, 200], [0] * 5 + [400] * 15]
    cus = [torch.tensor([0] + x).cumsum(0).to(DEV, torch.int32) for x in packings]
    assert len({frozenset(runs_of(x, x, heads)) for x in packings}) > 1
    cu = cus[0].clone()
    run = lambda: (lambda o, l: ops.sdpa_varlen_bwd(d_out, q, k, v, o, l, cu, cu, most, most, 0.125))(
        *ops.sdpa_varlen_fwd(q, k, v, cu, cu, most, most, 0.125))
    run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = run()
    for x in cus + cus[:1]:
        cu.copy_(x)
        graph.replay()
        want = run()
        ops.check_status()
        assert torch.equal(captured[1], want[1]) and torch.equal(captured[2], want[2])
        a, b = captured[0].float(), want[0].float()  # as above
        assert bool(((a - b).abs() <= 2.0 ** -7 * b.abs() + 1e-4).all())
