"""Destination rows that the kernels take as indices: strided, out of range, at the edges
of the output."""
import pytest
import torch

from grouped_gemm_b200 import _capi, backend

pytestmark = pytest.mark.gpu

SIZES = [3, 64, 0, 130, 1]


@pytest.fixture(params=["1", "2", "light"], ids=["one-cta", "pair", "one-cta-transposed-tiles"], autouse=True)
def ctas(request, monkeypatch):
    monkeypatch.setenv("B200GMM_CTAS", "1" if request.param == "light" else request.param)
    monkeypatch.setenv("B200GMM_LIGHT", "1" if request.param == "light" else "0")


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("strided", [False, True])
def test_scatter_writes_the_rows_named_and_no_other(weighted, strided):
    rows, k, n = sum(SIZES), 136, 72
    gen = torch.Generator(device="cuda").manual_seed(9)
    a = torch.randn(rows, k, device="cuda", generator=gen).bfloat16()
    b = torch.randn(len(SIZES), k, n, device="cuda", generator=gen).bfloat16()
    sizes = torch.tensor(SIZES, device="cuda")
    whole = torch.full((rows + 4, n), 7.0, device="cuda", dtype=torch.bfloat16)
    out = whole[1:-1]                                   # room on both sides: nothing may land there
    index = torch.randperm(rows + 2, device="cuda", generator=gen)[:rows].contiguous()
    index[7], index[8], index[9] = -1, rows + 2, 2 ** 40
    given = torch.stack([index, index.flip(0)], 1)[:, 0] if strided else index
    weight = torch.full((rows,), 2.0, device="cuda") if weighted else None
    status = backend.backend.device_status(a.device)
    before = int(status.item())
    backend.gmm_scatter(a, b, sizes, out, given, row_weight=weight)
    assert int(status.item()) & _capi.STATUS_BAD_ROW_DEST
    status.fill_(before)
    y = backend.gmm(a, b, sizes) * (2 if weighted else 1)   # a factor of two rounds nothing
    want = torch.full_like(whole, 7.0)
    ok = (index >= 0) & (index < rows + 2)
    want[1:-1][index[ok]] = y[ok]
    assert torch.equal(whole, want)


def test_scatter_into_no_rows():
    a = torch.ones(4, 64, device="cuda", dtype=torch.bfloat16)
    b = torch.ones(1, 64, 8, device="cuda", dtype=torch.bfloat16)
    out = torch.empty(0, 8, device="cuda", dtype=torch.bfloat16)
    status = backend.backend.device_status(a.device)
    before = int(status.item())
    backend.gmm_scatter(a, b, torch.tensor([4]), out, torch.zeros(4, dtype=torch.int64, device="cuda"))
    assert int(status.item()) & _capi.STATUS_BAD_ROW_DEST
    status.fill_(before)
