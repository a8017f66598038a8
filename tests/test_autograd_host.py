"""What the ops' autograd function owes its callers, on meta tensors (no GPU needed)."""

import pytest
import torch

import nanobrain_b200


def dense(requires_grad=True):
    return [torch.empty(2, 3, 5, 64, dtype=torch.bfloat16, device="meta", requires_grad=requires_grad) for _ in range(3)]


def packed():
    cu = torch.empty(3, dtype=torch.int32, device="meta")
    qkv = [torch.empty(10, 3, 64, dtype=torch.bfloat16, device="meta", requires_grad=True) for _ in range(3)]
    return qkv, lambda q, k, v: nanobrain_b200.sdpa_varlen(q, k, v, cu, cu, 5, 5)


CASES = {"dense": lambda: (dense(), nanobrain_b200.sdpa), "packed": packed}


@pytest.mark.parametrize("case", CASES)
def test_backward_under_compiled_autograd(case):
    from torch._dynamo import compiled_autograd

    qkv, call = CASES[case]()
    out = call(*qkv)
    with compiled_autograd._enable(lambda graph: graph):
        out.sum().backward()
    assert all(t.grad.shape == t.shape and t.grad.dtype == t.dtype for t in qkv)


@pytest.mark.parametrize("case", CASES)
def test_a_graph_can_be_kept_for_a_second_backward(case):
    qkv, call = CASES[case]()
    loss = call(*qkv).sum()
    loss.backward(retain_graph=True)
    loss.backward()
    with pytest.raises(RuntimeError, match="second time"):
        loss.backward()


@pytest.mark.parametrize("case,saved", [("dense", 5), ("packed", 7)])
def test_saved_tensor_hooks_see_what_is_kept(case, saved):
    qkv, call = CASES[case]()
    kept, used = [], []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: kept.append(t) or t, lambda t: used.append(t) or t):
        out = call(*qkv)
    assert len(kept) == saved
    out.sum().backward()
    assert len(used) == saved


def test_what_is_not_implemented_is_refused():
    q, k, v = dense()
    grad = torch.autograd.grad(nanobrain_b200.sdpa(q, k, v).sum(), q, create_graph=True)[0]
    with pytest.raises(RuntimeError):
        grad.sum().backward()  # there is no second derivative
    q, k, v = dense(requires_grad=False)
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: nanobrain_b200.sdpa(t, k, v).float().sum())(q)


@pytest.mark.parametrize("case,name", [("dense", "sdpa_fwd"), ("packed", "sdpa_varlen_fwd")])
def test_torch_function_overrides_see_the_op(case, name):
    from torch.overrides import TorchFunctionMode

    seen = []

    class Mode(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    class Subclass(torch.Tensor):
        @classmethod
        def __torch_function__(cls, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return super().__torch_function__(func, types, args, kwargs or {})

    qkv, call = CASES[case]()
    with Mode():
        call(*qkv)
    assert f"nanobrain_b200.{name}.default" in seen
    qkv = [t.detach().as_subclass(Subclass) for t in qkv]
    seen.clear()
    assert type(call(*qkv)) is Subclass and f"nanobrain_b200.{name}.default" in seen
