"""ops.gmm's native autograd function against the Python one it stands in for."""
import pytest
import torch

from grouped_gemm_b200 import ops

pytestmark = pytest.mark.gpu


def _leaves(trans_b, grad_a=True, grad_b=True):
    gen = torch.Generator(device="cuda").manual_seed(8)
    a = torch.randn(96, 64, device="cuda", generator=gen).bfloat16().requires_grad_(grad_a)
    shape = (3, 72, 64) if trans_b else (3, 64, 72)
    b = torch.randn(*shape, device="cuda", generator=gen).bfloat16().requires_grad_(grad_b)
    return a, b, torch.tensor([50, 0, 46])


@pytest.mark.parametrize("trans_b", [False, True])
@pytest.mark.parametrize("grad_a,grad_b", [(True, True), (True, False), (False, True), (False, False)])
def test_equals_the_python_function(trans_b, grad_a, grad_b):
    results = []
    for fn in (ops.gmm, ops.GroupedGemm.apply):
        a, b, sizes = _leaves(trans_b, grad_a, grad_b)
        out = fn(a, b, sizes, trans_b)
        assert out.requires_grad == (grad_a or grad_b)
        if out.requires_grad:
            out.backward(torch.ones(96, 1, device="cuda", dtype=torch.bfloat16).expand(96, 72))
        results.append((out.detach(), a.grad, b.grad))
    for x, y in zip(*results):
        assert (x is None and y is None) or torch.equal(x, y)


def test_saved_tensor_hooks_see_the_operands():
    packed = []

    def pack(t):
        packed.append(t.shape)
        return t.clone()

    a, b, sizes = _leaves(False)
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        out = ops.gmm(a, b, sizes)
    assert [tuple(s) for s in packed] == [(96, 64), (3, 64, 72), (3,)]
    out.sum().backward()
    assert a.grad is not None and b.grad is not None


def test_operand_changed_in_place_is_refused():
    a, b, sizes = _leaves(False)
    out = ops.gmm(a, b, sizes)
    with torch.no_grad():
        b.mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.sum().backward()


def test_tracing_records_the_product():
    a, b, sizes = _leaves(False, False, False)
    traced = torch.jit.trace(lambda x, y: ops.gmm(x, y, sizes), (a, b), check_trace=False)
    other = torch.randn_like(a)
    assert torch.equal(traced(other, b), ops.gmm(other, b, sizes))


def test_forward_mode_and_vmap_stay_refused():
    import torch.autograd.forward_ad as fwd
    a, b, sizes = _leaves(False, False, False)
    with fwd.dual_level():
        dual = fwd.make_dual(a, torch.ones_like(a))
        with pytest.raises((RuntimeError, NotImplementedError)):
            ops.gmm(dual, b, sizes)
    with pytest.raises((RuntimeError, AssertionError)):
        torch.func.vmap(lambda x: ops.gmm(x, b, sizes))(a[None].repeat(2, 1, 1))
    with pytest.raises((RuntimeError, AssertionError)):
        torch.func.grad(lambda x: ops.gmm(x, b, sizes).sum().float())(a)


@pytest.mark.parametrize("bad", ["a", "b", "sizes"])
def test_wrong_ranks_raise_assertion_errors(bad):
    a, b, sizes = _leaves(False, False, False)
    args = {"a": a, "b": b, "sizes": sizes}
    args[bad] = args[bad][None]
    with pytest.raises(AssertionError):
        ops.gmm(args["a"], args["b"], args["sizes"])
