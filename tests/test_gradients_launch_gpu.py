"""Both gradients of a small product in one launch (b200gmm_run_gradients) against the two
launches that it stands for: the same kernels' code on the same operands, so equal bit for bit.
Sizes on both sides of the line: as many tiles in all as SMs (148)."""
import pytest
import torch

from grouped_gemm_b200 import _capi, backend, ops

pytestmark = pytest.mark.gpu

# experts' rows, k, n, launches of the backward pass with weights [z, k, n]
CASES = [
    ([8], 8, 8, 1),
    ([50, 0, 46], 64, 72, 1),
    ([128, 100, 156, 128], 128, 128, 1),
    ([130, 0, 1, 509, 7, 300], 200, 520, 1),
    ([0, 0, 0], 64, 64, 1),
    ([128], 2048, 2048, 1),          # 16 + 128 tiles
    ([128], 2048, 2304, None),       # 16 + 144
]


@pytest.mark.parametrize("trans_b", [False, True])
@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("counts,k,n,launches", CASES)
def test_equals_two_launches(counts, k, n, launches, host, trans_b):
    gen = torch.Generator(device="cuda").manual_seed(4)
    rows = sum(counts) + 3                      # three rows of no expert
    a = torch.randn(rows, k, device="cuda", generator=gen).bfloat16().requires_grad_()
    shape = (len(counts), n, k) if trans_b else (len(counts), k, n)
    b = torch.randn(*shape, device="cuda", generator=gen).bfloat16().requires_grad_()
    grad = torch.randn(rows, n, device="cuda", generator=gen).bfloat16()
    sizes = torch.tensor(counts, device="cpu" if host else "cuda")
    out = ops.gmm(a, b, sizes, trans_b)
    before = _capi.launch_count()
    a_grad, b_grad = torch.autograd.grad(out, (a, b), grad)
    if launches is not None:
        assert _capi.launch_count() - before == launches
    used = sum(counts)
    x, w = a.detach(), b.detach()
    assert torch.equal(a_grad[:used], backend.gmm(grad, w, sizes, trans_b=not trans_b)[:used])
    lhs, rhs = (grad, x) if trans_b else (x, grad)
    assert torch.equal(b_grad, backend.gmm(lhs, rhs, sizes, trans_a=True))
    assert backend.device_status() == 0
