"""CPU-only checks of the C-ABI library: it loads, exports every symbol the
header declares, rejects bad arguments with the documented codes before touching
CUDA, and its host replay of the tile schedule covers every output exactly once."""
import ctypes
import os
import re

import numpy as np
import pytest

from grouped_gemm_b200 import _capi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "include", "b200gmm.h")


def _header_symbols():
    text = open(HEADER).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(b200gmm_\w+)\s*\(", text)))


def test_header_symbols_all_exported():
    lib = ctypes.CDLL(_capi.LIB_PATH)
    names = _header_symbols()
    assert len(names) >= 7
    for name in names:
        assert hasattr(lib, name), f"{name} declared in include/b200gmm.h but not exported"
    assert set(names) == set(_capi.SIGNATURES), "ctypes prototypes out of step with the header"


def test_strerror_and_tile_shape():
    assert _capi.strerror(0) == "ok"
    assert "trans_a" in _capi.strerror(-1)
    assert _capi.tile_shape(1) == (128, 256, 64)
    assert _capi.tile_shape(2) == (256, 256, 64)


def test_workspace_bytes():
    maps = 256 * 8 * 2 * 128  # per-CTA tensor-map copies for wgrad
    assert _capi.workspace_bytes(0) == 128 + maps
    assert _capi.workspace_bytes(8) == 128 + maps
    assert _capi.workspace_bytes(100) == 896 + maps  # 800 + 16 rounded up to 128
    with pytest.raises(RuntimeError):
        _capi.workspace_bytes(_capi.MAX_EXPERTS + 1)


@pytest.mark.parametrize("kwargs,code", [
    (dict(trans_a=1, trans_b=1), -1),
    (dict(d1=100), -2),            # not a multiple of 8
    (dict(n=12), -2),
    (dict(z=2000), -3),
    (dict(tokens=-1), -1),
    (dict(tokens=2 ** 31), -3),
])
def test_run_rejects_bad_arguments_before_cuda(kwargs, code):
    args = dict(z=4, tokens=512, d1=128, n=128, trans_a=0, trans_b=0)
    args.update(kwargs)
    lib = _capi.load()
    rc = lib.b200gmm_run(None, None, None, None, 0, args["z"], args["tokens"], args["d1"], args["n"],
                         args["trans_a"], args["trans_b"], None, 0, None, None)
    assert rc == code


def test_run_with_no_work_is_ok_without_gpu():
    lib = _capi.load()
    # z == 0, and non-transposed with zero rows: nothing to do, no CUDA call made.
    assert lib.b200gmm_run(None, None, None, None, 0, 0, 0, 128, 128, 0, 0, None, 0, None, None) == 0
    bs = np.zeros(4, dtype=np.int64)
    assert lib.b200gmm_run(None, None, None, bs.ctypes.data, 0, 4, 0, 128, 128, 0, 0, None, 0, None, None) == 0


def test_fused_entry_points_reject_bad_arguments_before_cuda():
    """Argument checks of the scatter / combine / gather / swiglu entry points
    that return before any CUDA call (so they can run without a GPU)."""
    lib = _capi.load()
    bs = np.array([64, 64], dtype=np.int64)
    dummy = np.zeros(64, dtype=np.int64).ctypes.data  # any non-null, 16-byte aligned address
    # scatter and combine need a destination table
    assert lib.b200gmm_run_scatter(dummy, dummy, None, None, 0, bs.ctypes.data, 0, 2, 128, 64, 64, 0, None, 0, None, None) == -1
    assert lib.b200gmm_run_combine(dummy, dummy, None, None, 0, None, 1, bs.ctypes.data, 0, 2, 128, 64, 64, 0, None, 0, None, None) == -1
    # combine: weights must be 4-byte aligned; k == 0 overwrite has nothing to write through
    assert lib.b200gmm_run_combine(dummy, dummy, dummy, None, 0, dummy + 2, 1, bs.ctypes.data, 0, 2, 128, 64, 64, 0, None, 0, None, None) == -2
    assert lib.b200gmm_run_combine(dummy, dummy, dummy, None, 0, None, 0, bs.ctypes.data, 0, 2, 128, 0, 64, 0, None, 0, None, None) == -1
    assert lib.b200gmm_run_combine(dummy, dummy, dummy, None, 0, None, 1, bs.ctypes.data, 0, 2, 128, 0, 64, 0, None, 0, None, None) == 0
    # gather: row index table, a non-empty source below 2^31 rows, an output of some kind
    assert lib.b200gmm_run_gather(dummy, 100, None, dummy, dummy, None, None, 0, bs.ctypes.data, 0, 2, 128, 64, 64, 0, None, 0, None, None) == -1
    assert lib.b200gmm_run_gather(dummy, 0, dummy, dummy, dummy, None, None, 0, bs.ctypes.data, 0, 2, 128, 64, 64, 0, None, 0, None, None) == -1
    assert lib.b200gmm_run_gather(dummy, 2 ** 31, dummy, dummy, dummy, None, None, 0, bs.ctypes.data, 0, 2, 128, 64, 64, 0, None, 0, None, None) == -1
    assert lib.b200gmm_run_gather(dummy, 100, dummy, dummy, None, None, None, 0, bs.ctypes.data, 0, 2, 128, 64, 64, 0, None, 0, None, None) == -1
    # swiglu: both weight tensors, an output, column count a multiple of 8
    assert lib.b200gmm_run_swiglu(dummy, dummy, None, dummy, None, None, 0, bs.ctypes.data, 0, 2, 128, 64, 64, 0, None, 0, None, None) == -1
    assert lib.b200gmm_run_swiglu(dummy, dummy, dummy, None, None, None, 0, bs.ctypes.data, 0, 2, 128, 64, 64, 0, None, 0, None, None) == -1
    assert lib.b200gmm_run_swiglu(dummy, dummy, dummy, dummy, None, None, 0, bs.ctypes.data, 0, 2, 128, 64, 60, 0, None, 0, None, None) == -2
    assert lib.b200gmm_run_swiglu(dummy, dummy, dummy + 8, dummy, None, None, 0, bs.ctypes.data, 0, 2, 128, 64, 64, 0, None, 0, None, None) == -2
    # a destination window needs a destination table
    assert lib.b200gmm_run_gather(dummy, 100, dummy, dummy, dummy, None, dummy, 64, bs.ctypes.data, 0, 2, 128, 64, 64, 0, None, 0, None, None) == -1
    # the static-scratch entry point refuses more experts than its scratch holds
    assert lib.b200gmm_run_static(dummy, dummy, dummy, bs.ctypes.data, 0, 257, 128, 64, 64, 0, 0, None, None) == -3


def _schedule(sizes, tokens, d1, n, trans_a, trans_b, ctas=1):
    lib = _capi.load()
    bs = np.asarray(sizes, dtype=np.int64)
    count = ctypes.c_int64(0)
    ptr = bs.ctypes.data if len(sizes) else None
    rc = lib.b200gmm_schedule_host(ptr, len(sizes), tokens, d1, n, trans_a, trans_b, ctas, None, 0,
                                   ctypes.byref(count))
    assert rc == 0
    out = np.zeros((count.value, _capi.SCHEDULE_FIELDS), dtype=np.int64)
    rc = lib.b200gmm_schedule_host(ptr, len(sizes), tokens, d1, n, trans_a, trans_b, ctas,
                                   out.ctypes.data, count.value, ctypes.byref(count))
    assert rc == 0
    return out


SIZE_SETS = [
    [128] * 4,
    [219, 2246, 5, 8103, 1, 1117, 4693, 0],
    [0, 0, 0],
    [1],
    [3400, 1030, 17412, 1225, 363, 5908, 1691, 1739],
    [7, 0, 300, 129, 128, 127, 0, 1025],
    [64, 65, 192, 193, 16, 17],
]


@pytest.mark.parametrize("sizes", SIZE_SETS)
@pytest.mark.parametrize("trans_b", [0, 1])
@pytest.mark.parametrize("n", [128, 256, 328, 1536])
@pytest.mark.parametrize("ctas", [1, 2])
@pytest.mark.parametrize("light", ["0", "1"])
def test_schedule_covers_rows_and_columns_once(sizes, trans_b, n, ctas, light, monkeypatch):
    """Every output element belongs to exactly one tile: 128-column granularity,
    since the transposed tiles of the one-CTA variant (B200GMM_LIGHT=1) are 128
    columns wide."""
    monkeypatch.setenv("B200GMM_LIGHT", light)
    tokens = sum(sizes)
    tile_m = 128 * ctas
    tiles = _schedule(sizes, tokens, 512, n, 0, trans_b, ctas)
    cover = np.zeros((tokens, (n + 127) // 128), dtype=np.int32)
    starts = np.concatenate([[0], np.cumsum(sizes)])
    for e, row0, col0, valid, stages, kind in tiles:
        width = 128 if kind else 256
        assert col0 % width == 0 and col0 < n
        assert starts[e] <= row0 and row0 + valid <= starts[e + 1], "tile leaves its expert's rows"
        if kind:
            assert light == "1" and ctas == 1 and 0 < valid <= 64 and stages == 512 // 128
            assert row0 == starts[e] and row0 + valid == starts[e + 1], "a transposed tile holds a whole small expert"
        else:
            assert 0 < valid <= tile_m and stages == 512 // 64
            if ctas == 1 and light == "1":
                assert sizes[e] > 64, "experts of at most 64 rows go to transposed tiles"
        cover[row0:row0 + valid, col0 // 128:(col0 + width + 127) // 128] += 1
    assert (cover == 1).all()


# z, rows, k, n, layout, features, CTAs a tile: the faster of the two on a B200 by a tenth and more
CHOICES = [
    (200, 30000, 512, 512, "nn", 0, 1), (200, 30000, 512, 512, "nn", _capi.FORM_GATED, 1),
    (256, 65536, 7168, 2048, "nn", 0, 2), (256, 65536, 2048, 7168, "nt", 0, 2), (200, 51200, 4096, 2048, "nn", _capi.FORM_GATED, 2),
    (64, 16384, 2048, 4096, "nn", 0, 2), (128, 16384, 4096, 2048, "nn", 0, 2), (64, 16384, 1024, 4096, "nn", 0, 1),
    (6, 6012, 2016, 264, "nn", _capi.FORM_GATED, 2), (1, 1084, 552, 1936, "nn", _capi.FORM_GATED, 1),
    (1, 1041, 2200, 4120, "nn", 0, 2), (1, 1041, 2200, 4120, "nn", _capi.FORM_GATED, 2),
    (19, 54879, 9736, 96, "nn", 0, 2), (19, 54879, 9736, 96, "nn", _capi.FORM_SCATTER, 2),
    (16, 6170, 1416, 11392, "nn", _capi.FORM_GATED_BACKWARD, 1), (16, 6170, 1416, 11392, "nn", _capi.FORM_GATHER, 1),
    (64, 8192, 4088, 8184, "nn", 0, 2), (64, 8192, 4088, 8184, "nt", 0, 2), (7, 3001, 2504, 1000, "nt", 0, 2),
    (49, 98681, 72, 2000, "nn", 0, 1), (9, 1966, 952, 128, "nn", 0, 1),
    (18, 34044, 3592, 552, "tn", 0, 2), (25, 100842, 368, 5768, "tn", 0, 2), (7, 22823, 880, 1344, "tn", 0, 2),
    (7, 3001, 1000, 2504, "tn", 0, 1), (8, 32768, 4096, 14336, "nn", 0, 2), (8, 32768, 4096, 14336, "tn", 0, 2),
]


@pytest.mark.parametrize("z,rows,k,n,layout,features,ctas", CHOICES)
def test_choice_between_one_cta_and_pairs(z, rows, k, n, layout, features, ctas, monkeypatch):
    monkeypatch.delenv("B200GMM_CTAS", raising=False)
    sizes = [rows // z + (i < rows % z) for i in range(z)]
    assert _capi.launch_forms(sizes, k, n, layout == "tn", layout == "nt", features).ctas == ctas
    # a device on which pairs do not fit has none, and the device's own count of pairs is what is asked
    assert _capi.launch_forms(sizes, k, n, layout == "tn", layout == "nt", features, pair_ctas=0).ctas == 1


@pytest.mark.parametrize("sizes", SIZE_SETS + [[256 * (t // 2) - 7, 256 * (t - t // 2) - 100] for t in (25, 37, 62, 150)])
@pytest.mark.parametrize("n", [256, 264, 776, 1288, 4104])
@pytest.mark.parametrize("layout", [(0, 0), (0, 1), (1, 0)])
@pytest.mark.parametrize("pair_ctas", [148, 4])
def test_positions_of_a_pair_launch_fill_every_accumulator_once(sizes, n, layout, pair_ctas, monkeypatch):
    """Wide tiles, narrow ones and halves of wide ones, in whatever order the launch has them, and
    halves that do not exist only where the last column tile is one accumulator wide."""
    monkeypatch.setenv("B200GMM_CTAS", "2")
    m = 200 if layout[0] else None
    positions = np.full((20000, 5), -1, dtype=np.int64)
    forms = _capi.launch_forms(sizes, 200, n, *layout, pair_ctas=pair_ctas, positions=positions)
    count = forms.wide + forms.narrow + forms.empty
    if sum(sizes) == 0:
        assert count == 0
        return
    assert count < len(positions) and (positions[count:] == -1).all()
    starts = np.concatenate([[0], np.cumsum(sizes)])
    seen = set()
    for expert, row0, col0, valid, units in positions[:count]:
        if units == 0:
            assert n % 512 in range(1, 257) and col0 >= n
            continue
        assert valid == min(256, (m if m else starts[expert + 1]) - row0) and (row0 - (0 if m else starts[expert])) % 256 == 0
        for unit in range(units):
            key = (expert, row0, col0 // 256 + unit)
            assert col0 % 256 == 0 and key[2] * 256 < n and key not in seen
            seen.add(key)
    row_tiles = len(sizes) if m else sum((size + 255) // 256 for size in sizes)
    assert len(seen) == row_tiles * ((n + 255) // 256) == 2 * forms.wide + forms.narrow
    if forms.all_narrow:
        assert forms.wide == forms.empty == 0


@pytest.mark.parametrize("sizes", SIZE_SETS)
@pytest.mark.parametrize("ctas", [1, 2])
def test_schedule_wgrad_full_grid_for_every_expert(sizes, ctas):
    tokens, m, n = sum(sizes), 320, 520
    tile_m = 128 * ctas
    tiles = _schedule(sizes, tokens, m, n, 1, 0, ctas)
    per_expert = ((m + tile_m - 1) // tile_m) * ((n + 255) // 256)
    assert len(tiles) == per_expert * len(sizes)
    for e, size in enumerate(sizes):
        mine = tiles[tiles[:, 0] == e]
        cover = np.zeros(((m + tile_m - 1) // tile_m, (n + 255) // 256), dtype=np.int32)
        for _, row0, col0, valid, stages, kind in mine:
            assert kind == 0
            assert valid == min(tile_m, m - row0)
            assert stages == (size + 63) // 64  # 0 for an empty expert: zero-fill tile
            cover[row0 // tile_m, col0 // 256] += 1
        assert (cover == 1).all()


def test_schedule_order_largest_experts_first_for_wgrad():
    """wgrad launch order: experts sorted by rows, largest first (ties keep their
    index order), so that the launch ends on the shortest tiles."""
    sizes = [10, 500, 0, 70, 3000, 200]
    tiles = _schedule(sizes, sum(sizes), 128, 256, 1, 0, 1)     # one tile per expert
    assert tiles[:, 0].tolist() == [4, 1, 5, 3, 0, 2]
    tiles = _schedule([64, 64, 64, 64], 256, 128, 256, 1, 0, 1)
    assert tiles[:, 0].tolist() == [0, 1, 2, 3]
    # the forward layouts keep the experts in index order
    for ctas in (1, 2):
        tiles = _schedule([600, 100, 900], 1600, 128, 256, 0, 0, ctas)
        assert (np.diff(tiles[:, 0]) >= 0).all()


def test_schedule_clamps_rows_past_tokens():
    # sum(batch_sizes) > tokens must never schedule a row >= tokens
    for ctas in (1, 2):
        tiles = _schedule([100, 100, 100], 150, 128, 256, 0, 0, ctas)
        assert int((tiles[:, 1] + tiles[:, 3]).max()) <= 150


def test_variant_choice_depends_on_shapes_only(monkeypatch):
    """cluster_ctas=0 asks for the variant b200gmm_run would use: pairs for
    experts with many rows, single CTAs for fine-grained groups."""
    monkeypatch.setenv("B200GMM_LIGHT", "1")
    big = _schedule([4096] * 8, 32768, 512, 512, 0, 0, 0)
    small = _schedule([64] * 64, 4096, 512, 512, 0, 0, 0)
    assert int(big[:, 3].max()) == 256 and int(small[:, 3].max()) == 64
    assert (small[:, 5] == 1).all(), "64-row experts run as transposed tiles"


def test_overlapped_kernel_has_no_read_only_inputs():
    """gmm_kernel starts while the kernel before it may still write its inputs, so no input
    that it reads with ordinary loads may take the read-only path: the output is the only
    __restrict__ parameter, and neither it nor build_schedule uses __ldg."""
    path = os.path.join(ROOT, "grouped_gemm_b200", "csrc", "gmm_kernel.cuh")
    text = re.sub(r"//[^\n]*", "", open(path).read())
    signature = re.search(r"\bgmm_kernel\((.*?)\)\s*\{", text, flags=re.S).group(1)
    restricted = [p.strip() for p in signature.split(",") if "__restrict__" in p]
    assert restricted == ["__nv_bfloat16* __restrict__ c"]
    schedule = re.search(r"\bvoid build_schedule\((.*?)\)\s*\{", text, flags=re.S).group(1)
    assert "__restrict__" not in schedule
    assert "__ldg" not in text


def test_pair_sum_refuses_what_its_32_bit_numbers_cannot_hold():
    """Both parts of the contraction, each a whole number of k-blocks of 64, and the rows of
    both parts of a_pair: below 2^31 each, refused before any CUDA call (the addresses
    are dummies; sizes that fit would go on to ask for the device)."""
    lib = _capi.load()
    dummy = np.zeros(64, dtype=np.int64)
    at = (dummy.ctypes.data + 15) // 16 * 16
    bs = np.array([8], dtype=np.int64)

    def run(tokens, d1, b1=at, n=8):
        return lib.b200gmm_run_pair_sum(at, at, b1, at, bs.ctypes.data, 0, 1, tokens, d1, n, 0, None, 0, None, None)

    assert run(8, 2 ** 30 - 64) == -3
    assert run(8, 2 ** 31 - 264) == -3
    assert run(2 ** 30 - 128, 64) == -3
    assert run(8, 64, b1=None) == -1
    assert run(8, 64, b1=at + 8) == -2
    assert run(8, 60) == -2
    assert run(0, 2 ** 30 - 64) == 0 and run(8, 2 ** 30 - 64, n=0) == 0     # nothing to do


def test_row_index_and_gated_backward_entries_reject_bad_arguments_before_cuda():
    """The entry points that gmm_scatter and the gated backward use."""
    lib = _capi.load()
    bs = np.array([64, 64], dtype=np.int64)
    room = np.zeros(64, dtype=np.int64)
    at = (room.ctypes.data + 15) // 16 * 16   # any non-null, 16-byte aligned address

    def rows(index=at, out=at, out_rows=128, weight=None, accumulate=0, tokens=128, k=64, n=64):
        return lib.b200gmm_run_combine_rows(at, at, index, out, out_rows, weight, accumulate, bs.ctypes.data, 0, 2, tokens, k,
                                            n, 0, None, 0, None, None)

    assert rows(index=None) == -1
    assert rows(out_rows=-1) == -1
    assert rows(out=None) == -1
    assert rows(weight=at + 2) == -2
    assert rows(k=60) == -2 and rows(n=60) == -2
    assert rows(k=0) == -1                      # nothing to overwrite the rows with
    assert rows(k=0, accumulate=1) == 0         # adding nothing
    assert rows(tokens=0) == 0 and rows(n=0) == 0

    for entry in (lib.b200gmm_run_swiglu_backward, lib.b200gmm_run_swiglu_backward_full):
        def gated(up=at, grad=at, products=at, tokens=128, k=64, n=64):
            return entry(at, at, up, grad, products, bs.ctypes.data, 0, 2, tokens, k, n, 0, None, 0, None, None)

        assert gated(products=None) == -1
        assert gated(grad=None) == -1
        assert gated(up=None) == -1
        assert gated(up=at + 8) == -2
        assert gated(grad=at + 8) == -1
        assert gated(n=60) == -2 and gated(k=60) == -2
        assert gated(tokens=0) == 0 and gated(n=0) == 0
