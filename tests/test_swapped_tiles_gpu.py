"""Tiles of few rows, which the forward / dgrad kernels compute with their operands
swapped (schedule.cuh: swapped_rows), at the row counts where the form of a tile or of
its stores changes, against 64-bit sums.

Bound: one rounding to bf16 (2^-8 relative) of an fp32 sum of k products, whose own
error is at most k * 2^-24 times the sum of the products' absolute values; a scattered
row with a weight is rounded once as well.  Adding to the destination (accumulate) is
one more rounding.  The gated product multiplies two such sums: its bound is stated there.

The rule (b200gmm.cu: swap_rows) goes by the mean rows of an expert, the length of the
contraction and the number of tiles: every case here lies on a stated side of a line, and
each line has cases on both sides.  Idle experts make the mean.  The gathered product does
not have the form, and pairs only in launches of more tiles (test_wide_tiles_gpu.py): they run the same
rows here as plain tiles.
"""
import pytest
import torch

from grouped_gemm_b200 import backend

pytestmark = pytest.mark.gpu

# 1 .. 64 of 128 rows are swapped; 16 / 32: the step of the row count and of the stores;
# last: full tiles followed by a remainder of each kind.
ROWS = [1, 15, 16, 17, 0, 31, 32, 33, 48, 63, 64, 65, 96, 127, 128, 129, 128 + 40, 256 + 1, 256 + 128, 256 + 130]
SIZES = ROWS + [0] * 110     # 15.8 rows an expert


def _idle_to(experts):
    """ROWS (2060 of them) over `experts` experts."""
    return ROWS + [0] * (experts - len(ROWS))


def _operands(k, n, trans_b, seed=3, counts=SIZES):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rows = sum(counts)
    a = torch.randn(rows, k, device="cuda", generator=gen).bfloat16()
    shape = (len(counts), n, k) if trans_b else (len(counts), k, n)
    b = (torch.randn(*shape, device="cuda", generator=gen) * 0.1).bfloat16()
    return a, b, torch.tensor(counts, device="cuda")


def _sums(a, b, trans_b, counts=SIZES):
    """The products in 64 bits and the sums of their terms' absolute values."""
    out, mag, start = [], [], 0
    for i, size in enumerate(counts):
        w = (b[i].t() if trans_b else b[i]).double()
        x = a[start:start + size].double()
        out.append(x @ w)
        mag.append(x.abs() @ w.abs())
        start += size
    return torch.cat(out), torch.cat(mag)


def _bound(ref, mag, k):
    return 2.0 ** -8 * ref.abs() + k * 2.0 ** -24 * mag + 1e-30


@pytest.fixture(params=["1", "2"], ids=["one-cta", "pair"], autouse=True)
def ctas(request, monkeypatch):
    monkeypatch.setenv("B200GMM_CTAS", request.param)


@pytest.mark.parametrize("trans_b", [False, True])
@pytest.mark.parametrize("k,n", [(64, 264),        # short contraction: plain tiles
                                 (504, 264), (512, 264), (520, 72),   # around the line of 512
                                 (4088, 8), (4096, 264), (4104, 72)])
def test_rows_around_every_step(trans_b, k, n):
    a, b, sizes = _operands(k, n, trans_b)
    ref, mag = _sums(a, b, trans_b)
    got = torch.full((a.shape[0] + 1, n), 7.0, device="cuda", dtype=torch.bfloat16)
    backend.gmm(a, b, sizes, trans_b=trans_b, c=got[:-1])
    assert bool(((got[:-1].double() - ref).abs() <= _bound(ref, mag, k)).all())
    assert bool((got[-1] == 7.0).all()), "a row past the last was written"
    source = torch.arange(a.shape[0], device="cuda").flip(0)
    gathered = backend.gmm_gather(a.flip(0).contiguous(), source, b, sizes, trans_b=trans_b)
    assert torch.equal(gathered, got[:-1])


@pytest.mark.parametrize("experts", [32, 33, 42, 43])
@pytest.mark.parametrize("gated", [False, True])
def test_launches_around_the_line_of_rows(gated, experts):
    """64 rows an expert: 33 experts are below, 32 above.  The gated product: 48, 43 and 42."""
    k, n, counts = 520, 520, _idle_to(experts)
    a, b, sizes = _operands(k, n, False, counts=counts)
    ref, mag = _sums(a, b, False, counts)
    if not gated:
        got = backend.gmm(a, b, sizes)
        assert bool(((got.double() - ref).abs() <= _bound(ref, mag, k)).all())
        return
    bu = _operands(k, n, False, seed=4, counts=counts)[1]
    up, mag_up = _sums(a, bu, False, counts)
    got = backend.gmm_swiglu(a, b, bu, sizes)
    want, bound = _gated(ref, up, k * 2.0 ** -24 * mag, k * 2.0 ** -24 * mag_up)
    assert bool(((got.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("columns", [256 * 73, 256 * 74, 128 * 98, 128 * 99])
def test_launches_around_the_line_of_tiles(columns):
    """One expert of 40 rows: as many tiles as column tiles.  A plain product needs half as
    many as SMs (74 of 148), the gated product, whose tiles are 128 columns wide, two thirds (99)."""
    k = 512
    gen = torch.Generator(device="cuda").manual_seed(8)
    a = torch.randn(40, k, device="cuda", generator=gen).bfloat16()
    bg, bu = ((torch.randn(1, k, columns, device="cuda", generator=gen) * 0.1).bfloat16() for _ in range(2))
    sizes = torch.tensor([40], device="cuda")
    (g, mg), (u, mu) = _sums(a, bg, False, [40]), _sums(a, bu, False, [40])
    assert bool(((backend.gmm(a, bg, sizes).double() - g).abs() <= _bound(g, mg, k)).all())
    want, bound = _gated(g, u, k * 2.0 ** -24 * mg, k * 2.0 ** -24 * mu)
    assert bool(((backend.gmm_swiglu(a, bg, bu, sizes).double() - want).abs() <= bound).all())


@pytest.mark.parametrize("k", [72, 4104])
@pytest.mark.parametrize("accumulate", [False, True])
def test_scattered_and_weighted_rows(accumulate, k):
    n = 136
    a, b, sizes = _operands(k, n, False)
    ref, mag = _sums(a, b, False)
    gen = torch.Generator(device="cuda").manual_seed(5)
    index = torch.randperm(a.shape[0], device="cuda", generator=gen)
    weight = torch.rand(a.shape[0], device="cuda", generator=gen)
    out = torch.ones(a.shape[0], n, device="cuda", dtype=torch.bfloat16)
    backend.gmm_scatter(a, b, sizes, out, index, row_weight=weight, accumulate=accumulate)
    w = weight.double()[:, None]
    ref, bound = ref * w, _bound(ref * w, mag * w, k + 1)
    if accumulate:
        ref = ref + 1.0
        bound = bound + 2.0 ** -8 * ref.abs()
    assert bool(((out[index].double() - ref).abs() <= bound).all())


def _gated(g, u, eg, eu):
    """silu(g) * u and its bound, eg and eu being those of g and u: silu has a slope of at
    most 1.1, __expf and __fdividef err by a few 2^-22 and the result is rounded once."""
    ref = g * torch.sigmoid(g) * u
    return ref, 2.0 ** -8 * ref.abs() + 1.1 * eg * u.abs() + eu * g.abs() + 2.0 ** -18 * (ref.abs() + 1e-6)


@pytest.mark.parametrize("k", [8, 72, 4104])
@pytest.mark.parametrize("trans_b", [False, True])
def test_gated_product_and_its_backward(trans_b, k):
    """_gated for the product; of its gradients silu' has a slope of at most 0.5."""
    n = 136
    a, bg, sizes = _operands(k, n, trans_b)
    bu = _operands(k, n, trans_b, seed=4)[1]
    (g, mg), (u, mu) = _sums(a, bg, trans_b), _sums(a, bu, trans_b)
    eg, eu = k * 2.0 ** -24 * mg, k * 2.0 ** -24 * mu
    s = torch.sigmoid(g)
    tiny = 2.0 ** -18
    ref, bound = _gated(g, u, eg, eu)
    got = backend.gmm_swiglu(a, bg, bu, sizes, trans_b=trans_b)
    assert bool(((got.double() - ref).abs() <= bound).all())
    dh = torch.randn(a.shape[0], n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(6)).bfloat16()
    d_gate, d_up = backend.gmm_swiglu_backward(a, bg, bu, dh, sizes, trans_b=trans_b)
    d = dh.double()
    slope = s * (1.0 + g * (1.0 - s))
    ref = d * u * slope
    bound = 2.0 ** -8 * ref.abs() + d.abs() * (1.1 * eu + 0.5 * eg * u.abs()) + tiny * (d * u).abs() + 1e-6
    assert bool(((d_gate.double() - ref).abs() <= bound).all())
    ref = d * g * s
    bound = 2.0 ** -8 * ref.abs() + 1.1 * eg * d.abs() + tiny * (d * g).abs() + 1e-6
    assert bool(((d_up.double() - ref).abs() <= bound).all())
