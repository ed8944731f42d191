"""C entry points that the Python functions do not go through: rows scattered to addresses
with weights and additions (b200gmm_run_combine) and the gated product's backward that
leaves rows of no expert alone (b200gmm_run_swiglu_backward).  Each is compared bit for
bit with the entry point that the Python functions use."""
import pytest
import torch

from grouped_gemm_b200 import _capi, backend

pytestmark = pytest.mark.gpu

SIZES = [5, 0, 64, 130, 300, 1]


@pytest.fixture(params=["1", "2"], ids=["one-cta", "pair"], autouse=True)
def ctas(request, monkeypatch):
    monkeypatch.setenv("B200GMM_CTAS", request.param)


def _scratch(z):
    nbytes = _capi.workspace_bytes(z)
    return torch.empty(nbytes, dtype=torch.uint8, device="cuda"), nbytes


@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("trans_b", [False, True])
def test_combine_to_addresses_equals_combine_to_rows(trans_b, weighted, accumulate):
    rows, z, k, n = sum(SIZES), len(SIZES), 136, 72
    gen = torch.Generator(device="cuda").manual_seed(4)
    a = torch.randn(rows, k, device="cuda", generator=gen).bfloat16()
    shape = (z, n, k) if trans_b else (z, k, n)
    b = torch.randn(*shape, device="cuda", generator=gen).bfloat16()
    weight = torch.rand(rows, device="cuda", generator=gen) if weighted else None
    sizes = torch.tensor(SIZES, device="cuda")
    index = torch.randperm(rows + 3, device="cuda", generator=gen)[:rows]
    start = torch.randn(rows + 5, n, device="cuda", generator=gen).bfloat16()
    got, want = start.clone(), start.clone()            # the first and the last row lie outside the window
    backend.gmm_scatter(a, b, sizes, want[1:-1], index, trans_b=trans_b, row_weight=weight, accumulate=accumulate)
    window = got[1:-1]
    dest = index * (n * 2) + window.data_ptr()
    # a row below the window, one past it, one that starts inside and is not 16-byte aligned
    for i, address in ((7, window.data_ptr() - n * 2), (8, window.data_ptr() + window.numel() * 2),
                       (9, window.data_ptr() + 8)):
        want[1 + index[i]] = start[1 + index[i]]
        dest[i] = address
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ws, nbytes = _scratch(z)
    rc = _capi.load().b200gmm_run_combine(
        a.data_ptr(), b.data_ptr(), dest.data_ptr(), window.data_ptr(), window.numel() * 2,
        None if weight is None else weight.data_ptr(), 1 if accumulate else 0, sizes.data_ptr(), 1, z, rows, k, n,
        1 if trans_b else 0, ws.data_ptr(), nbytes, status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    assert int(status.item()) == _capi.STATUS_BAD_ROW_DEST
    assert torch.equal(got, want)


@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("trans_b", [False, True])
def test_gated_backward_leaves_rows_of_no_expert_alone(trans_b, host):
    z, k, n, left = len(SIZES), 72, 136, 77
    rows = sum(SIZES) + left
    gen = torch.Generator(device="cuda").manual_seed(5)
    a, dh = (torch.randn(rows, c, device="cuda", generator=gen).bfloat16() for c in (k, n))
    shape = (z, n, k) if trans_b else (z, k, n)
    bg, bu = (torch.randn(*shape, device="cuda", generator=gen).bfloat16() for _ in range(2))
    sizes = torch.tensor(SIZES, device="cpu" if host else "cuda")
    want = backend.gmm_swiglu_backward(a, bg, bu, dh, sizes, trans_b=trans_b)
    got = torch.full((2, rows, n), 7.0, device="cuda", dtype=torch.bfloat16)
    ws, nbytes = _scratch(z)
    rc = _capi.load().b200gmm_run_swiglu_backward(
        a.data_ptr(), bg.data_ptr(), bu.data_ptr(), dh.data_ptr(), got.data_ptr(), sizes.data_ptr(), 0 if host else 1, z,
        rows, k, n, 1 if trans_b else 0, ws.data_ptr(), nbytes, None, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    used = sum(SIZES)
    for half in range(2):
        assert torch.equal(got[half, :used], want[half][:used])
        assert bool((got[half, used:] == 7.0).all())
