"""The unit-vector correlation (block sizes 4 and 8) against the CUDA-core kernel: the same
records, byte for byte, at the edges of its tiles (32 ranges, 128 domains) and on planes that
leave its quick test: flat and nearly flat blocks, ties, saturated and high-contrast ones."""
import time

import numpy as np
import pytest
import torch

import mars_b200 as mb

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def unit_form_at_any_size(monkeypatch):
    monkeypatch.setenv("MARS_UNIT_TILES", "0")


@pytest.fixture(scope="module")
def both():
    a, b = mb.Context(0), mb.Context(0)
    b.set_search_path("simt")
    yield a, b
    a.close()
    b.close()


def _plane(kind, w, h, seed=11):
    rng = np.random.default_rng(seed)
    yy, xx = np.mgrid[0:h, 0:w]
    if kind == "noise":
        p = rng.integers(0, 256, (h, w))
    elif kind == "flat":
        p = np.full((h, w), 77)
        p[h // 2:, : w // 3] = 12
    elif kind == "faint":  # 128 +- 1
        p = 128 + rng.integers(-1, 2, (h, w))
    elif kind == "ties":  # a pattern that repeats at every domain stride
        p = 255 * ((xx // 4 + yy // 4) % 2)
    elif kind == "saturated":
        p = np.clip(300.0 * np.sin(xx / 9.0) * np.cos(yy / 7.0) + 128, 0, 255)
    else:  # a smooth field with one textured corner
        p = np.where((xx < w // 4) & (yy < h // 4), rng.integers(0, 256, (h, w)), (xx + yy) % 200)
    return np.ascontiguousarray(p, dtype=np.uint8)


KINDS = ("noise", "flat", "faint", "ties", "saturated", "mixed")


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("size,w,h,shift", [
    (4, 8, 8, 2),        # one domain
    (4, 70, 38, 2),      # a last domain tile of a few
    (4, 65, 47, 4),
    (8, 46, 30, 2),      # 128 domains exactly: 16 x 8
    (8, 129, 67, 2),
    (8, 160, 96, 16),
])
def test_records_equal_the_cuda_core_kernel(both, kind, size, w, h, shift):
    img = _plane(kind, w, h)
    params = mb.make_params(shift=shift)
    rows, cols = np.meshgrid(np.arange(h // size) * size, np.arange(w // size) * size,
                             indexing="ij")
    rows, cols = rows.ravel(), cols.ravel()
    for n in (1, 31, 32, 33, len(rows)):
        got, want = (c.search_blocks(img, size, shift, params, rows[:n], cols[:n]) for c in both)
        assert got[0].tobytes() == want[0].tobytes(), (kind, n)
        assert np.array_equal(got[1], want[1])


@pytest.mark.parametrize("w,h,shift", [(136, 72, 2), (129, 127, 4)])
def test_plans_mix_the_forms(both, w, h, shift):
    # Sizes 4 and 8 in the unit launch, 16 and 32 in the integer one, side by side.
    img = _plane("mixed", w, h, 3)
    params = mb.make_params(min_size=4, max_size=32, shift=shift)
    plan = both[0].search_plan(w, h, params)
    for _ in range(2):
        got, want = plan.run(img), both[1].search_provider(img, params)
        for size in (4, 8, 16, 32):
            rows, cols = (a.ravel() for a in np.meshgrid(np.arange(h // size) * size,
                                                         np.arange(w // size) * size,
                                                         indexing="ij"))
            x, y = (t.search_many(rows, cols, size, shift) for t in (got, want))
            assert x[0].tobytes() == y[0].tobytes() and np.array_equal(x[1], y[1]), size
        got.close()
        want.close()
    plan.close()


@pytest.mark.parametrize("size", [4, 8])
@pytest.mark.parametrize("alfa_bits,beta_bits,max_alfa", [(1, 1, 0.3), (4, 7, 3.0), (8, 10, 1.0)])
def test_other_quantisers(both, size, alfa_bits, beta_bits, max_alfa):
    img = _plane("mixed", 96, 64, 5)
    params = mb.make_params(shift=2, bits_alfa=alfa_bits, bits_beta=beta_bits, max_alfa=max_alfa)
    got, want = (c.search_grid(img, size, 2, params) for c in both)
    assert got[0].tobytes() == want[0].tobytes()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("size,w,h,n", [
    (4, 400, 300, 33),     # 227 tiles, the last group of three: 14 splits a range tile
    (4, 400, 300, 2000),   # two splits
    (8, 404, 300, 70),     # 218 tiles: the last group of two
])
def test_several_splits_a_range_tile(both, kind, size, w, h, n):
    # Splits share champions as they find them, in whatever order they run: again and again.
    img = _plane(kind, w, h)
    params = mb.make_params(shift=2)
    rows, cols = np.meshgrid(np.arange(h // size) * size, np.arange(w // size) * size,
                             indexing="ij")
    pick = np.random.default_rng(n).permutation(rows.size)[:n]
    rows, cols = rows.ravel()[pick], cols.ravel()[pick]
    want = both[1].search_blocks(img, size, 2, params, rows, cols)
    for _ in range(5):
        got = both[0].search_blocks(img, size, 2, params, rows, cols)
        assert got[0].tobytes() == want[0].tobytes()
        assert np.array_equal(got[1], want[1])


@pytest.mark.parametrize("alfa_bits,beta_bits,max_alfa", [(4, 7, 1.0), (1, 1, 3.0), (2, 3, 0.3),
                                                          (8, 2, 2.0)])
@pytest.mark.parametrize("kind", ["ties", "faint", "noise"])
@pytest.mark.parametrize("size", [4, 8])
def test_ranges_that_nothing_fits_better_than_flat(both, size, kind, alfa_bits, beta_bits, max_alfa):
    # Champions of contrast 0, W far below zero where the offset's steps are coarse; the first
    # domain's flat quarter at (0, 0) included.
    img = _plane(kind, 180, 132, 7)
    for plane in (img, np.where(np.add.outer(np.arange(132), np.arange(180)) < 40, 90, img)):
        plane = np.ascontiguousarray(plane, dtype=np.uint8)
        params = mb.make_params(shift=2, bits_alfa=alfa_bits, bits_beta=beta_bits, max_alfa=max_alfa)
        got, want = (c.search_grid(plane, size, 2, params) for c in both)
        assert got[0].tobytes() == want[0].tobytes()


@pytest.mark.parametrize("side,shift", [(512, 2), (1024, 8)])
def test_no_slower_than_the_integer_form_where_nothing_fits(monkeypatch, side, shift):
    # A checkerboard of 4 x 4 squares in blocks of 8: no domain correlates with any block.
    plane = torch.from_numpy(_plane("ties", side, side)).cuda()
    params = mb.make_params(min_size=8, max_size=8, shift=shift)
    n = mb.C.c_size_t()
    times, records = [], []
    for tiles in ("0", str(1 << 40)):  # the unit form, the fold
        monkeypatch.setenv("MARS_UNIT_TILES", tiles)
        with mb.Context(0) as ctx:
            args = (ctx.handle, plane.data_ptr(), side, side, mb.C.byref(params))
            mb.check(mb.lib().mars_search_nodes_device(*args, None, 0, mb.C.byref(n), None))
            out = torch.zeros(n.value, 80, dtype=torch.uint8, device="cuda")
            best = float("inf")
            for _ in range(5):
                torch.cuda.synchronize()
                t = time.perf_counter()
                mb.check(mb.lib().mars_search_nodes_device(*args, out.data_ptr(), n.value,
                                                           mb.C.byref(n), None))
                torch.cuda.synchronize()
                best = min(best, time.perf_counter() - t)
            times.append(best)
            records.append(out.cpu().numpy().tobytes())
    assert records[0] == records[1]
    assert times[0] < 1.5 * times[1]
