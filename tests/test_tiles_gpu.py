"""The kernels at the edges of their tiles: key and query counts around the 64-column halves and the
128-row tiles the main kernels work in, one and several of them, against the CPU oracle."""

import ctypes as C

import numpy as np
import pytest
import torch

import nanobrain_b200
from nanobrain_b200 import _lib, ops
from oracle import attn_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def dense_shape(batch, heads, lq, lk):
    return _lib.Shape(batch, heads, 64, lq, lk, batch * lq, batch * lk, None, None, 0.125)


def check(names, got, want):
    for name, a, b in zip(names, got, want):
        b = np.asarray(b, dtype=np.float32)
        err = np.abs(a.detach().float().cpu().numpy() - b)
        assert np.isfinite(err).all(), name
        assert err.max() <= 2e-2 * max(1.0, np.abs(b).max()) and err.mean() <= 2e-3 * max(1.0, np.abs(b).max()), name


@pytest.mark.parametrize("lk", [1, 15, 16, 17, 63, 64, 65, 127, 128, 129, 191, 192, 193, 320, 321])
@pytest.mark.parametrize("lq", [1, 129])
def test_half_tile_edges(lq, lk):
    g = torch.Generator().manual_seed(1000 * lq + lk)
    q, d_out = (torch.randn(2, 2, lq, 64, generator=g).to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(2, 2, lk, 64, generator=g).to(torch.bfloat16) for _ in range(2))
    want = O.sdpa_fwd_bwd(*(t.float().numpy() for t in (q, k, v, d_out)))
    qd, kd, vd = (t.to(DEV).requires_grad_(True) for t in (q, k, v))
    out = nanobrain_b200.sdpa(qd, kd, vd)
    out.backward(d_out.to(DEV))
    ops.check_status()
    check(("out", "dq", "dk", "dv"), (out, qd.grad, kd.grad, vd.grad), (want[0], *want[2:5]))


@pytest.mark.parametrize("lk", [129, 192, 200, 256, 321])
def test_second_pass_over_the_keys(lk):
    # Scores that rise by far more than 2^60 after the first half tile: the forward walks the keys a
    # second time with a running max. The last tile has one or two halves, ragged or full.
    g = torch.Generator().manual_seed(lk)
    q = torch.randn(1, 2, 140, 64, generator=g)
    k = torch.randn(1, 2, lk, 64, generator=g)
    v = torch.randn(1, 2, lk, 64, generator=g).to(torch.bfloat16)
    k[:, :, 70:] *= 20.0
    k[:, :, 128:] *= 2.0
    q, k = q.to(torch.bfloat16), k.to(torch.bfloat16)
    want, lse = O.sdpa_forward(*(t.float().numpy() for t in (q, k, v)))[:2]
    out, got_lse = ops.sdpa_fwd(q.to(DEV), k.to(DEV), v.to(DEV), 0.125)
    ops.check_status()
    check(("out",), (out,), (want,))
    np.testing.assert_allclose(got_lse.cpu().numpy(), lse, rtol=2e-3, atol=2e-3)


@pytest.mark.parametrize("batch,heads,lq,lk,rising", [
    (1, 1, 130, 2000, False), (1, 1, 1, 2500, False), (1, 2, 300, 1537, False), (2, 1, 64, 4096, False),
    (1, 6, 900, 2500, False), (1, 1, 200, 1900, True),
])
def test_query_tiles_cut_between_ctas(batch, heads, lq, lk, rising):
    # Few query tiles and many keys: the dense forward gives every CTA an equal run of key tiles and
    # puts the parts of a query tile together afterwards; `rising` scores need the second walk as well.
    assert _lib.load().nb_attn_fwd_split_workspace_bytes(C.byref(dense_shape(batch, heads, lq, lk))) > 0
    g = torch.Generator().manual_seed(lq + lk)
    q = torch.randn(batch, heads, lq, 64, generator=g)
    k, v = (torch.randn(batch, heads, lk, 64, generator=g) for _ in range(2))
    if rising:
        k[:, :, 300:] *= 20.0
        k[:, :, 1000:] *= 2.0
    q, k, v = (t.to(torch.bfloat16) for t in (q, k, v))
    want, lse = O.sdpa_forward(*(t.float().numpy() for t in (q, k, v)))[:2]
    for _ in range(2):
        out, got_lse = ops.sdpa_fwd(q.to(DEV), k.to(DEV), v.to(DEV), 0.125)
        ops.check_status()
        check(("out",), (out,), (want,))
        np.testing.assert_allclose(got_lse.cpu().numpy(), lse, rtol=2e-3, atol=2e-3)


@pytest.mark.parametrize("batch,heads,lq,lk", [
    (1, 1, 900, 130), (1, 1, 1000, 1), (2, 1, 1537, 300), (1, 2, 4096, 64), (1, 6, 900, 1500), (2, 12, 820, 820),
])
def test_key_tiles_cut_between_ctas(batch, heads, lq, lk):
    # Few key tiles and many queries: the dense backward gives every CTA an equal run of query tiles and
    # the epilogue adds up the parts of a key tile's dK and dV.
    assert _lib.load().nb_attn_bwd_split_workspace_bytes(C.byref(dense_shape(batch, heads, lq, lk))) > 0
    g = torch.Generator().manual_seed(lq + lk)
    q, d_out = (torch.randn(batch, heads, lq, 64, generator=g).to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(batch, heads, lk, 64, generator=g).to(torch.bfloat16) for _ in range(2))
    want = O.sdpa_fwd_bwd(*(t.float().numpy() for t in (q, k, v, d_out)))
    for _ in range(2):
        qd, kd, vd = (t.to(DEV).requires_grad_(True) for t in (q, k, v))
        nanobrain_b200.sdpa(qd, kd, vd).backward(d_out.to(DEV))
        ops.check_status()
        check(("dq", "dk", "dv"), (qd.grad, kd.grad, vd.grad), want[2:5])


@pytest.mark.parametrize("lengths,heads", [([1], 1), ([130, 0, 64], 2), ([300] * 40 + [2000], 12)])
def test_work_list_used_again(lengths, heads):
    # Fewer units than CTAs, and more: every launch over one list does all of its units.
    total = sum(lengths) + 70  # rows past the last sequence come out as zeros each time
    g = torch.Generator().manual_seed(total)
    q, k, v = (torch.randn(total, heads, 64, generator=g).to(DEV, torch.bfloat16) for _ in range(3))
    cu = torch.tensor([0] + lengths).cumsum(0).to(DEV, torch.int32)
    want, _ = ops.sdpa_varlen_fwd(q, k, v, cu, cu, max(lengths), max(lengths), 0.125)
    lib, lse = _lib.load(), torch.empty(heads, total, device=DEV)
    desc = lambda t: _lib.Tensor(t.data_ptr(), 0, t.stride(0), t.stride(1))
    shape = _lib.Shape(len(lengths), heads, 64, max(lengths), max(lengths), total, total, cu.data_ptr(), cu.data_ptr(),
                       0.125)
    ws = torch.empty(_lib.fwd_workspace_bytes(shape), dtype=torch.uint8, device=DEV)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for call in (lib.nb_attn_fwd, lib.nb_attn_fwd_again, lib.nb_attn_fwd_again):
        out = torch.full_like(q, float("nan"))
        args = _lib.FwdArgs(shape, desc(q), desc(k), desc(v), desc(out), lse.data_ptr(), None, ws.data_ptr(), ws.numel())
        _lib.check(call(C.byref(args), stream), "nb_attn_fwd")
        assert torch.equal(out, want)


@pytest.mark.parametrize("heads,length,cut", [(8, 1500, True), (8, 1800, False), (8, 2048, False), (4, 2000, True)])
def test_query_tiles_with_an_sm_each_are_cut_where_that_is_faster(heads, length, cut):
    shape = dense_shape(1, heads, length, length)
    assert (_lib.load().nb_attn_fwd_split_workspace_bytes(C.byref(shape)) > 0) == cut
