"""Launches that draw no tile positions and take batch_sizes as an argument: both sides
of each line of the rule, and what must not change with it."""
import pytest
import torch

from grouped_gemm_b200 import _capi, backend

pytestmark = pytest.mark.gpu


def _check(sizes, k, n, host, trans_a=False):
    gen = torch.Generator(device="cuda").manual_seed(1)
    rows, z = sum(sizes), len(sizes)
    a = torch.randn(rows, k, device="cuda", generator=gen).bfloat16()
    b = torch.randn(*((rows, n) if trans_a else (z, k, n)), device="cuda", generator=gen).bfloat16()
    bs = torch.tensor(sizes, dtype=torch.int64, device="cpu" if host else "cuda")
    got = backend.gmm(a, b, bs, trans_a=trans_a)
    start, refs = 0, []
    for i, size in enumerate(sizes):
        x = a[start:start + size].double()
        refs.append(x.t() @ b[start:start + size].double() if trans_a else x @ b[i].double())
        start += size
    ref = torch.stack(refs) if trans_a else torch.cat(refs)
    # one rounding to bf16 of an fp32 sum of terms ~ N(0, 1) products: 2^-8 relative plus
    # length * 2^-24 * the largest sum of absolute values (below 2 per term on average)
    length = max(sizes) if trans_a else k
    bound = 2.0 ** -8 * ref.abs() + length * 2.0 ** -24 * 2 * length + 1e-30
    assert bool(((got.double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("z", [1, 63, 64, 65, 200])
def test_experts_around_the_inline_limit(z, host):
    _check([(7 * i) % 5 for i in range(z)], 72, 40, host)
    _check([(7 * i) % 5 for i in range(z)], 72, 40, host, trans_a=True)


@pytest.mark.parametrize("columns", [256 * 73, 256 * 74, 256 * 75, 256 * 147, 256 * 148, 256 * 149])
@pytest.mark.parametrize("ctas", ["1", "2"])
def test_tiles_around_one_wave(columns, ctas, monkeypatch):
    """One expert: as many tiles as column tiles (times two: the bound counts a partial
    row tile), from below a single wave of a 148-SM device to past it."""
    monkeypatch.setenv("B200GMM_CTAS", ctas)
    _check([100], 64, columns, False)
    _check([100], 64, columns // 2, False)
    _check([100], 64, columns, True, trans_a=True)


def test_bad_host_sizes_raise_the_same_status():
    lib = _capi.load()
    for sizes in ([100, -5, 100], [2 ** 40, 1, 1], [-2 ** 62, 2 ** 62, 7]):
        found = []
        for host in (False, True):
            a = torch.ones(150, 64, device="cuda", dtype=torch.bfloat16)
            b = torch.ones(3, 64, 64, device="cuda", dtype=torch.bfloat16)
            c = torch.zeros(150, 64, device="cuda", dtype=torch.bfloat16)
            bs = torch.tensor(sizes, device="cpu" if host else "cuda")
            status = torch.zeros(1, dtype=torch.int32, device="cuda")
            nbytes = _capi.workspace_bytes(3)
            ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
            assert lib.b200gmm_run(a.data_ptr(), b.data_ptr(), c.data_ptr(), bs.data_ptr(), 0 if host else 1, 3, 150, 64, 64,
                                   0, 0, ws.data_ptr(), nbytes, status.data_ptr(),
                                   torch.cuda.current_stream().cuda_stream) == 0
            found.append((int(status.item()), c))
        assert found[0][0] == found[1][0] != 0
        assert torch.equal(found[0][1], found[1][1])


def test_back_to_back_launches_depend_on_one_another():
    """A chain in which every launch reads what the one before it wrote."""
    z, k = 4, 256
    eye = torch.eye(k, device="cuda", dtype=torch.bfloat16).repeat(z, 1, 1)
    host = torch.tensor([100, 30, 0, 126])
    for sizes in (host, host.cuda()):
        x = torch.randn(256, k, device="cuda").bfloat16()
        y = x
        for _ in range(50):
            y = backend.gmm(y, eye, sizes)
        assert torch.equal(x, y)


def test_captured_call_reads_host_sizes_at_replay():
    a = torch.ones(64, 64, device="cuda", dtype=torch.bfloat16)
    b = torch.stack([torch.full((64, 64), float(i + 1)) for i in range(2)]).bfloat16().cuda()
    sizes = torch.tensor([64, 0])
    c = torch.zeros(64, 64, device="cuda", dtype=torch.bfloat16)
    backend.gmm(a, b, sizes, c=c)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        backend.gmm(a, b, sizes, c=c)
        d = backend.gmm(c, b, sizes)
    graph.replay()
    torch.cuda.synchronize()
    assert bool((c == 64).all()) and bool((d == 64 * 64).all())
    sizes.copy_(torch.tensor([0, 64]))
    graph.replay()
    torch.cuda.synchronize()
    assert bool((c == 128).all())


def test_row_transfer_in_a_small_launch_uses_the_whole_device(monkeypatch):
    """A product of six rows that carries 86 MB of row transfer.  The same transfer as a
    launch of its own takes about 45 us, inside the product about 200; dealt over the
    product's four thread blocks alone it took 6500.  The bound, about 1000, lies between."""
    lib = _capi.load()
    monkeypatch.setenv("B200GMM_PUSH_TMA", "1")
    sizes, k, n, items, columns = [3, 1, 0, 2], 64, 72, 4000, 10752
    z, rows = len(sizes), sum(sizes)
    a = torch.randn(rows, k, device="cuda").bfloat16()
    b = torch.randn(z, k, n, device="cuda").bfloat16()
    want = backend.gmm(a, b, torch.tensor(sizes))
    bs = torch.tensor(sizes, device="cuda")
    out = torch.zeros(rows, n, device="cuda", dtype=torch.bfloat16)
    dest = torch.arange(rows, device="cuda") * (n * 2) + out.data_ptr()
    src = torch.randn(items, columns, device="cuda").bfloat16()
    dst = torch.zeros_like(src)
    row = torch.arange(items, device="cuda")
    rank = torch.zeros(items, dtype=torch.int32, device="cuda")
    table = torch.tensor([dst.data_ptr()], device="cuda")
    nbytes = _capi.workspace_bytes(z)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    head = (a.data_ptr(), b.data_ptr(), dest.data_ptr(), out.data_ptr(), out.numel() * 2, bs.data_ptr(), 1, z, rows, k, n, 0)
    push = (src.data_ptr(), columns * 2, items, None, rank.data_ptr(), row.data_ptr(), table.data_ptr())

    def fused():
        assert lib.b200gmm_run_scatter_push(*head, *push, ws.data_ptr(), nbytes, None, stream) == 0

    def separate():
        assert lib.b200gmm_run_scatter(*head, ws.data_ptr(), nbytes, None, stream) == 0
        assert lib.b200gmm_push_rows(*push, 0, stream) == 0

    def microseconds(launch):
        times = []
        for _ in range(8):
            begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            begin.record()
            launch()
            end.record()
            end.synchronize()
            times.append(begin.elapsed_time(end) * 1e3)
        return sorted(times)[len(times) // 2]

    alone = microseconds(separate)
    dst.zero_()
    together = microseconds(fused)
    assert torch.equal(out, want) and torch.equal(dst, src)
    assert together < 20 * alone + 100, (together, alone)
