"""Backward of the gated product: the input gradient as one product over both halves of
the contraction, and rows that belong to no expert."""
import pytest
import torch

from grouped_gemm_b200 import backend

pytestmark = pytest.mark.gpu

SIZES = [5, 0, 64, 130, 300, 1]


@pytest.fixture(params=["1", "2"], ids=["one-cta", "pair"], autouse=True)
def ctas(request, monkeypatch):
    monkeypatch.setenv("B200GMM_CTAS", request.param)


@pytest.mark.parametrize("light", ["0", "1"])
@pytest.mark.parametrize("trans_b", [False, True])
@pytest.mark.parametrize("k,n", [(72, 8), (264, 64), (136, 200)])
def test_input_gradient_against_64_bits(k, n, trans_b, light, monkeypatch):
    """Contraction lengths below, at and past a k-block (64): the second half starts a
    block of its own.  Bound: one rounding to bf16 of an fp32 sum of 2 n products."""
    monkeypatch.setenv("B200GMM_LIGHT", light)
    gen = torch.Generator(device="cuda").manual_seed(2)
    rows = sum(SIZES)
    d = torch.randn(2, rows, n, device="cuda", generator=gen).bfloat16()
    shape = (len(SIZES), k, n) if trans_b else (len(SIZES), n, k)
    w = [(torch.randn(*shape, device="cuda", generator=gen) * 0.1).bfloat16() for _ in range(2)]
    got = backend._gmm_pair_sum(d, w[0], w[1], torch.tensor(SIZES, device="cuda"), trans_b)
    start = 0
    for i, size in enumerate(SIZES):
        x = d[:, start:start + size].double()
        m = [(v[i].t() if trans_b else v[i]).double() for v in w]
        ref = x[0] @ m[0] + x[1] @ m[1]
        mag = x[0].abs() @ m[0].abs() + x[1].abs() @ m[1].abs()
        err = (got[start:start + size].double() - ref).abs()
        assert bool((err <= 2.0 ** -8 * ref.abs() + 2 * n * 2.0 ** -24 * mag + 1e-30).all()), i
        start += size


@pytest.mark.parametrize("left", [0, 1, 77])
def test_rows_of_no_expert_are_zeros(left):
    k, n = 64, 136
    rows = sum(SIZES) + left
    a, dh = (torch.randn(rows, c, device="cuda").bfloat16() for c in (k, n))
    bg, bu = (torch.randn(len(SIZES), k, n, device="cuda").bfloat16() for _ in range(2))
    torch.full((4, rows, n), float("nan"), device="cuda", dtype=torch.bfloat16)   # what the allocator hands out next
    d_gate, d_up = backend.gmm_swiglu_backward(a, bg, bu, dh, torch.tensor(SIZES, device="cuda"))
    assert bool((d_gate[sum(SIZES):] == 0).all()) and bool((d_up[sum(SIZES):] == 0).all())
    assert bool(torch.isfinite(d_gate).all()) and bool(torch.isfinite(d_up).all())


def test_no_experts():
    a = torch.randn(16, 64, device="cuda").bfloat16()
    b = torch.empty(0, 64, 72, device="cuda", dtype=torch.bfloat16)
    dh = torch.randn(16, 72, device="cuda").bfloat16()
    sizes = torch.empty(0, dtype=torch.int64, device="cuda")
    d_gate, d_up = backend.gmm_swiglu_backward(a, b, b, dh, sizes)
    assert bool((d_gate == 0).all()) and bool((d_up == 0).all())
