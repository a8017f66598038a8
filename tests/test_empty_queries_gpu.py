"""The packed backward with many key tiles that have no queries: sequences without queries, and a buffer
with many rows past its last sequence."""

import numpy as np
import pytest
import torch

import nanobrain_b200
from nanobrain_b200 import ops
from oracle import attn_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("lengths_q,lengths_k,heads,spare", [
    ([200, 50], [200, 50], 16, 4200),                              # 33 tiles past the last sequence
    ([300, 0, 100, 0, 0, 129] * 3, [50, 700, 130, 1, 256, 40] * 3, 24, 3),
    ([300, 0, 100, 0, 0, 129] * 5, [50, 700, 130, 1, 256, 40] * 5, 24, 3),
])
def test_units_without_queries_in_a_row(lengths_q, lengths_k, heads, spare):
    g = torch.Generator().manual_seed(sum(lengths_q))
    tq, tk = sum(lengths_q) + spare, sum(lengths_k) + spare
    q, d_out = (torch.randn(tq, heads, 64, generator=g).to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(tk, heads, 64, generator=g).to(torch.bfloat16) for _ in range(2))
    cu_q, cu_k = (torch.tensor([0] + list(x)).cumsum(0).to(DEV, torch.int32) for x in (lengths_q, lengths_k))
    want = [np.zeros((n, heads, 64), np.float32) for n in (tq, tk, tk)]
    at_q = at_k = 0
    for nq, nk in zip(lengths_q, lengths_k):
        if nq:
            sq, sk = slice(at_q, at_q + nq), slice(at_k, at_k + nk)
            one = lambda t, s: t[s].float().numpy().transpose(1, 0, 2)[None]
            for w, s, x in zip(want, (sq, sk, sk), O.sdpa_fwd_bwd(one(q, sq), one(k, sk), one(v, sk), one(d_out, sq))[2:5]):
                w[s] = x[0].transpose(1, 0, 2)
        at_q, at_k = at_q + nq, at_k + nk
    for _ in range(10):
        qd, kd, vd = (t.to(DEV).requires_grad_(True) for t in (q, k, v))
        nanobrain_b200.sdpa_varlen(qd, kd, vd, cu_q, cu_k, max(lengths_q), max(lengths_k)).backward(d_out.to(DEV))
        ops.check_status()  # a wait that gave up would be reported here
        for name, got, w in zip(("dq", "dk", "dv"), (qd.grad, kd.grad, vd.grad), want):
            err = np.abs(got.float().cpu().numpy() - w)
            # bf16 results of bf16 products with fp32 accumulation, as for every other configuration
            assert err.max() <= 2e-2 * max(1.0, np.abs(w).max()) and err.mean() <= 2e-3, name
