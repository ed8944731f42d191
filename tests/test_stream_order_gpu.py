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


def _sizes(z, rows, gen):
    """A ragged split of `rows` rows over z experts, some of them empty."""
    ids = torch.randint(0, max(1, z - z // 4), (rows,), generator=gen)
    return torch.bincount(ids, minlength=z)


def _step(case, x, buffers, waits):
    """One chain: every launch reads what the launch before it wrote.  With `waits` the
    device is drained between the launches, so that nothing can overlap."""
    z, k, n, sizes, source, weight, w1, w2, bw1, bw2 = (case[key] for key in (
        "z", "k", "n", "sizes", "source", "weight", "w1", "w2", "bw1", "bw2"))
    done = (lambda: torch.cuda.synchronize()) if waits else (lambda: None)
    results = []

    def add(t):
        results.append(t)
        done()
        return t

    y = add(backend.gmm(x, w1, sizes, c=buffers["y"]))                          # [T, n]
    dw = add(backend.gmm(x, y, sizes, trans_a=True, c=buffers["dw"]))            # wgrad of a fresh forward output
    back = add(backend.gmm(y, dw, sizes, trans_b=True, c=buffers["x"]))          # fresh weights, [T, k]
    got = add(backend.gmm_gather(back, source, w1, sizes, c=buffers["y2"]))      # gathers fresh rows
    gw = add(backend.gmm_gather_wgrad(back, source, got, sizes, c=buffers["dw"]))
    h = add(backend.gmm_swiglu(back, gw, w1, sizes))                             # fresh gate weights
    d = backend.gmm_swiglu_backward(back, w1, w2, h, sizes)                      # fresh output gradient
    add(d[0]), add(d[1])
    out = buffers["out"]
    backend.gmm_scatter(d[0], bw1, sizes, out, source, row_weight=weight)        # every row once: no order of additions
    add(out)
    backend.gmm_scatter(d[1], bw2, sizes, out, source, accumulate=True)          # onto the rows just written
    add(out)
    return [t.clone() for t in results]


@pytest.mark.parametrize("ctas", ["1", "2"])
@pytest.mark.parametrize("where", ["device", "host"])
@pytest.mark.parametrize("z,rows,k,n", [(5, 700, 136, 264),          # one wave: no counter kernel
                                        (9, 20000, 264, 1032),       # several waves, the counter kernel between the products
                                        (70, 9000, 200, 520)])       # more host sizes than travel with a launch: a copy as well
def test_chains_of_launches_equal_the_same_launches_one_at_a_time(z, rows, k, n, where, ctas, monkeypatch):
    """Exact: the kernels are deterministic, so a launch that read a buffer before the
    launch ahead of it had written it would show.  Every pass has other inputs, in
    the same buffers, so that stale contents differ from the right ones."""
    monkeypatch.setenv("B200GMM_CTAS", ctas)
    cpu = torch.Generator().manual_seed(z)
    gen = torch.Generator(device="cuda").manual_seed(z)

    def normal(*shape, scale=1.0):
        return (torch.randn(*shape, device="cuda", generator=gen) * scale).bfloat16()

    sizes = _sizes(z, rows, cpu)
    case = {"z": z, "k": k, "n": n, "sizes": sizes.cuda() if where == "device" else sizes,
            "source": torch.randperm(rows, generator=cpu).cuda(), "weight": torch.rand(rows, device="cuda", generator=gen),
            "w1": normal(z, k, n, scale=k ** -0.5), "w2": normal(z, k, n, scale=k ** -0.5),
            "bw1": normal(z, n, k, scale=n ** -0.5), "bw2": normal(z, n, k, scale=n ** -0.5)}

    def buffers():
        shapes = {"y": (rows, n), "y2": (rows, n), "dw": (z, k, n), "x": (rows, k), "out": (rows, k)}
        return {name: torch.zeros(*shape, device="cuda", dtype=torch.bfloat16) for name, shape in shapes.items()}

    inputs = [normal(rows, k, scale=0.02 * (1 + i / 8)) for i in range(6)]
    free, drained = buffers(), buffers()
    torch.cuda.synchronize()
    got = [_step(case, x, free, False) for x in inputs]
    want = [_step(case, x, drained, True) for x in inputs]
    for i, (g, w) in enumerate(zip(got, want)):
        for j, (u, v) in enumerate(zip(g, w)):
            assert torch.equal(u, v), (i, j)
