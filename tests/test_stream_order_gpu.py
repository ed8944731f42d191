"""What a launch may read and when: host batch_sizes that the stream itself fills, and
chains of launches that overlap the one before them."""
import pytest
import torch

from grouped_gemm_b200 import _capi, backend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("z", [3, 64, 65])
def test_pinned_host_sizes_are_read_when_the_stream_gets_there(z):
    """Earlier work of the stream fills the pinned array after the call has returned;
    a pageable array is read by the call itself, and may change right after it."""
    lib = _capi.load()
    rows, k, n = 5 * z, 72, 40
    a = torch.randn(rows, k, device="cuda").bfloat16()
    b = torch.randn(z, k, n, device="cuda").bfloat16()
    sizes = torch.tensor([(3 * i) % 11 for i in range(z)], device="cuda")   # sums to at most 5 z + 6
    sizes[-1] = 0
    want = torch.zeros(rows, n, device="cuda", dtype=torch.bfloat16)
    backend.gmm(a, b, sizes, c=want)
    nbytes = _capi.workspace_bytes(z)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")

    def run(host):
        c = torch.zeros(rows, n, device="cuda", dtype=torch.bfloat16)
        return c, lib.b200gmm_run(a.data_ptr(), b.data_ptr(), c.data_ptr(), host.data_ptr(), 0, z, rows, k, n, 0, 0,
                                  ws.data_ptr(), nbytes, None, torch.cuda.current_stream().cuda_stream)

    pinned = torch.zeros(z, dtype=torch.int64).pin_memory()
    torch.cuda.synchronize()
    torch.cuda._sleep(40_000_000)          # about 20 ms: the call below returns long before the copy
    pinned.copy_(sizes, non_blocking=True)
    got, rc = run(pinned)
    assert rc == 0
    torch.cuda.synchronize()
    assert torch.equal(got, want)

    pageable = sizes.cpu()
    torch.cuda._sleep(40_000_000)
    got, rc = run(pageable)
    pageable.zero_()
    assert rc == 0
    torch.cuda.synchronize()
    assert torch.equal(got, want)
