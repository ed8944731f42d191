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
    ([128], 2048, 2304, 2),          # 16 + 144
    ([3] * 65, 16, 24, 1),           # more host sizes than fit in a kernel's arguments
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
    assert _capi.launch_count() - before == launches
    used = sum(counts)
    x, w = a.detach(), b.detach()
    assert torch.equal(a_grad[:used], backend.gmm(grad, w, sizes, trans_b=not trans_b)[:used])
    lhs, rhs = (grad, x) if trans_b else (x, grad)
    assert torch.equal(b_grad, backend.gmm(lhs, rhs, sizes, trans_a=True))
    assert backend.device_status() == 0


def test_captured_backward_is_two_launches_and_reads_sizes_again():
    """A captured product keeps its own dependencies; a replay follows sizes that changed on the device."""
    counts = [[50, 0, 46], [7, 80, 9]]
    gen = torch.Generator(device="cuda").manual_seed(4)
    a = torch.randn(96, 64, device="cuda", generator=gen).bfloat16()
    b = torch.randn(3, 64, 72, device="cuda", generator=gen).bfloat16()
    grad = torch.randn(96, 72, device="cuda", generator=gen).bfloat16()
    sizes = torch.tensor(counts[0], device="cuda")
    x, w = a.clone().requires_grad_(), b.clone().requires_grad_()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):          # (allocations and lazy work before the capture)
        torch.autograd.grad(ops.gmm(x, w, sizes), (x, w), grad)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    before = _capi.launch_count()
    with torch.cuda.graph(graph, stream=side):
        a_grad, b_grad = torch.autograd.grad(ops.gmm(x, w, sizes), (x, w), grad)
    assert _capi.launch_count() - before == 3      # the product and its two gradients
    for count in counts:
        sizes.copy_(torch.tensor(count))
        graph.replay()
        assert torch.equal(a_grad, backend.gmm(grad, b, sizes, trans_b=True))
        assert torch.equal(b_grad, backend.gmm(a, grad, sizes, trans_a=True))
    assert backend.device_status() == 0
