"""Tiles of a CTA pair: two accumulators of 256 columns side by side (gmm_kernel.cuh:
wide_tile), where their form changes: column tiles of one and of two accumulators, k-blocks
fewer than, as many as and more than the skew of the two takes at both ends, launches whose
last tiles are taken as halves, and tiles with swapped operands.  A launch of few tiles has them one
accumulator wide: SIZES as they are, unless a test says otherwise.  MANY and STEPS are what
it takes to have wide and swapped ones, and those tests say which forms they mean to run.

Operands are whole numbers of at most 3 in size, so every sum of products below is one of
whole numbers under 2^24, exact in fp32 in any order, and the result is its rounding to bf16: the
comparison is for equality."""
import pytest
import torch

from grouped_gemm_b200 import _capi, backend

pytestmark = pytest.mark.gpu

SIZES = [300, 0, 1, 255, 513, 64, 256]


@pytest.fixture(autouse=True)
def pairs(monkeypatch):
    monkeypatch.setenv("B200GMM_CTAS", "2")


def _whole(*shape, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(-3, 4, shape, device="cuda", generator=gen).bfloat16()


def _products(a, b, sizes):
    out, start = [], 0
    for w, size in zip(b, sizes):
        out.append(a[start:start + size].double() @ w.double())
        start += size
    return torch.cat(out)


def _check(sizes, k, n):
    rows = sum(sizes)
    a, b, g = _whole(rows, k, seed=1), _whole(len(sizes), k, n, seed=2), _whole(rows, n, seed=3)
    bs = torch.tensor(sizes, device="cuda")
    bt = b.transpose(1, 2).contiguous()
    want = _products(a, b, sizes).bfloat16()
    index = torch.randperm(rows, device="cuda")
    source = torch.empty_like(a)
    source[index] = a
    assert torch.equal(backend.gmm(a, b, bs), want)
    assert torch.equal(backend.gmm(a, bt, bs, trans_b=True), want)
    assert torch.equal(backend.gmm_gather(source, index, b, bs), want)
    out = torch.zeros(rows, n, device="cuda", dtype=torch.bfloat16)
    backend.gmm_scatter(a, b, bs, out, index)
    assert torch.equal(out[index], want)
    wgrad = torch.stack([x.double().t() @ y.double() for x, y in zip(a.split(sizes), g.split(sizes))]).bfloat16()
    assert torch.equal(backend.gmm(a, g, bs, trans_a=True), wgrad)
    assert torch.equal(backend.gmm_gather_wgrad(source, index, g, bs), wgrad)
    pair = torch.stack([a, a.flip(1)]).contiguous()
    assert torch.equal(backend._gmm_pair_sum(pair, b, b, bs, False), (_products(a, b, sizes) + _products(pair[1], b, sizes)).bfloat16())


@pytest.mark.parametrize("n", [8, 248, 256, 264, 504, 512, 520, 768, 776, 1032])
def test_columns_of_one_and_two_accumulators(n):
    _check(SIZES, 200, n)


@pytest.mark.parametrize("k", [8, 64, 72, 128, 136, 192, 200, 256, 264, 328, 584])
def test_k_blocks_around_the_skew(k):
    _check(SIZES, k, 776)


@pytest.mark.parametrize("row_tiles", [12, 24, 25, 30, 37, 49, 62])
def test_last_tiles_as_halves(row_tiles):
    """1288 columns: two wide column tiles and one of a single accumulator, whose second half
    does not exist.  On 74 pairs the leftover tiles run from few to more than half a round."""
    _check([256 * (row_tiles // 2) - 7, 256 * (row_tiles - row_tiles // 2) - 100], 72, 1288)


@pytest.mark.parametrize("n", [8, 120, 128, 136, 256, 264, 392])
def test_gated_product_and_its_backward(n):
    """The gated product needs rounding: 64-bit sums of the same whole numbers, scaled so that the
    gate is of order one; bound of one rounding to bf16 and the few 2^-20 of __expf and __fdividef."""
    k, rows = 136, sum(SIZES)
    a = _whole(rows, k, seed=1) / 16
    bg, bu = _whole(len(SIZES), k, n, seed=2) / 4, _whole(len(SIZES), k, n, seed=3) / 4
    bs = torch.tensor(SIZES, device="cuda")
    g, u = _products(a, bg, SIZES), _products(a, bu, SIZES)   # multiples of 1/64: exact in fp32
    s = torch.sigmoid(g)
    want = g * s * u
    got = backend.gmm_swiglu(a, bg, bu, bs).double()
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -18 * (g * u).abs() + 1e-6).all())
    dh = _whole(rows, n, seed=4)
    dg, du = backend.gmm_swiglu_backward(a, bg, bu, dh, bs)
    d = dh.double()
    want_g, want_u = d * u * s * (1 + g * (1 - s)), d * g * s
    assert bool(((dg.double() - want_g).abs() <= 2.0 ** -8 * want_g.abs() + 2.0 ** -18 * (d * u * (1 + g.abs())).abs() + 1e-6).all())
    assert bool(((du.double() - want_u).abs() <= 2.0 ** -8 * want_u.abs() + 2.0 ** -18 * (d * g).abs() + 1e-6).all())


MANY = SIZES * 8    # 72 row tiles of 256
# the remainders of a row tile around every step of a swapped tile's rows (32, up to 192), and of its stores
STEPS = [1, 31, 32, 33, 63, 64, 65, 95, 96, 97, 159, 160, 161, 191, 192, 193, 255, 256, 257, 0] * 4


def _forms(sizes, k, n, **kw):
    return _capi.launch_forms(sizes, k, n, **kw)


@pytest.mark.parametrize("k", [8, 64, 72, 128, 136, 192, 200, 264, 584])
def test_wide_tiles_k_blocks_around_the_skew(k):
    """One to ten k-blocks; the weight gradient's are the rows of its experts."""
    for kw in ({}, {"trans_b": True}, {"features": _capi.FORM_GATHER}, {"trans_a": True}):
        forms = _forms(MANY, k, 776, **kw)
        assert forms.wide > 74 and forms.swapped == 0, kw
    _check(MANY, k, 776)


@pytest.mark.parametrize("n,swapped", [(264, False), (512, False), (1032, True), (1288, True), (1544, True)])
def test_wide_tiles_columns(n, swapped):
    """The last column tile: two accumulators (8 and 256 columns in the second) or one."""
    forms = _forms(MANY, 200, n)
    assert forms.wide >= 72 and (forms.swapped > 0) == swapped and (forms.narrow > 0) == (n in (1032, 1544))
    _check(MANY, 200, n)


@pytest.mark.parametrize("n", [1288, 1544])
@pytest.mark.parametrize("k", [72, 584])
def test_swapped_tiles_of_a_pair(k, n):
    """Rows around every step, wide tiles and narrow ones (scattered rows of a short contraction)."""
    for kw in ({}, {"trans_b": True}, {"features": _capi.FORM_SCATTER}):
        forms = _forms(STEPS, k, n, **kw)
        assert forms.ctas == 2 and forms.swapped > 148 and (forms.wide == 0) == ("features" in kw)
    _check(STEPS, k, n)


@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("k,n", [(136, 1288), (8200, 1288)])
def test_swapped_tiles_scattered_weighted_and_accumulated(k, n, accumulate):
    """Weights are powers of two, so that only the roundings to bf16 are left: of the weighted row, and
    of its sum with what was there.  Wide tiles need the long contraction."""
    sizes = STEPS
    forms = _forms(sizes, k, n, features=_capi.FORM_SCATTER)
    assert forms.swapped > 50 and (forms.wide > 0) == (k > 8192)
    rows = sum(sizes)
    a, b = _whole(rows, k, seed=1), _whole(len(sizes), k, n, seed=2)
    bs = torch.tensor(sizes, device="cuda")
    index = torch.randperm(rows, device="cuda")
    weight = 2.0 ** torch.randint(-2, 3, (rows,), device="cuda").float()
    out = _whole(rows, n, seed=5)
    there = out[index].double()
    backend.gmm_scatter(a, b, bs, out, index, row_weight=weight, accumulate=accumulate)
    want = (_products(a, b, sizes) * weight.double()[:, None]).bfloat16()
    if accumulate:
        want = (want.double() + there).bfloat16()
    assert torch.equal(out[index], want)


@pytest.mark.parametrize("trans_b", [False, True])
@pytest.mark.parametrize("sizes,n", [(MANY, 512), (MANY, 776), (STEPS, 520), (STEPS, 776)])
def test_wide_gated_product_and_its_backward(sizes, n, trans_b):
    """As test_gated_product_and_its_backward, on wide tiles, swapped ones among them."""
    k, rows = 136, sum(sizes)
    forms = _forms(sizes, k, n, trans_b=trans_b, features=_capi.FORM_GATED)
    assert forms.wide > 74 and (forms.swapped > 0) == (sizes is STEPS or n == 776)
    assert _forms(sizes, k, n, trans_b=trans_b, features=_capi.FORM_GATED_BACKWARD).wide > 74
    a = _whole(rows, k, seed=1) / 16
    bg, bu = _whole(len(sizes), k, n, seed=2) / 4, _whole(len(sizes), k, n, seed=3) / 4
    wg, wu = (w.transpose(1, 2).contiguous() if trans_b else w for w in (bg, bu))
    bs = torch.tensor(sizes, device="cuda")
    g, u = _products(a, bg, sizes), _products(a, bu, sizes)
    s = torch.sigmoid(g)
    want = g * s * u
    got = backend.gmm_swiglu(a, wg, wu, bs, trans_b=trans_b).double()
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -18 * (g * u).abs() + 1e-6).all())
    dh = _whole(rows, n, seed=4)
    dg, du = backend.gmm_swiglu_backward(a, wg, wu, dh, bs, trans_b=trans_b)
    d = dh.double()
    want_g, want_u = d * u * s * (1 + g * (1 - s)), d * g * s
    assert bool(((dg.double() - want_g).abs() <= 2.0 ** -8 * want_g.abs() + 2.0 ** -18 * (d * u * (1 + g.abs())).abs() + 1e-6).all())
    assert bool(((du.double() - want_u).abs() <= 2.0 ** -8 * want_u.abs() + 2.0 ** -18 * (d * g).abs() + 1e-6).all())
