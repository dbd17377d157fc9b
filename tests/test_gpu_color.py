"""The colour input and metric kernels (color.cu) against the oracle, bit-exact, and the
colour encode/decode pipeline (color.rs:400-528 without regions) end to end."""
import time

import numpy as np
import pytest

import mars_b200 as mb
from mars_b200 import color, synthetic
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = mb.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("shape", [(64, 64), (37, 53), (1, 7), (3, 2), (256, 384)])
def test_ycbcr_both_ways(ctx, shape):
    rng = np.random.default_rng(sum(shape))
    r, g, b = (rng.integers(0, 256, shape, dtype=np.uint8) for _ in range(3))
    got = ctx.ycbcr(r, g, b)
    want = orc.ycbcr(r, g, b)
    for x, y in zip(got, want):
        assert np.array_equal(x, y)
    back = ctx.rgb_from_ycbcr(*got)
    for x, y in zip(back, orc.rgb_from_ycbcr(*want)):
        assert np.array_equal(x, y)


def test_every_rgb_value_on_one_axis(ctx):
    # All 2^24 colours would be 48 MB per plane; every (r, g, b) with r, g, b in 0..255 in
    # steps covers the rounding boundaries of each coefficient.
    v = np.arange(256, dtype=np.uint8)
    r, g, b = np.meshgrid(v, v[::3], v[::5], indexing="ij")
    got = ctx.ycbcr(r, g, b)
    for x, y in zip(got, orc.ycbcr(r, g, b)):
        assert np.array_equal(x, y)
    for x, y in zip(ctx.rgb_from_ycbcr(r, g, b), orc.rgb_from_ycbcr(r, g, b)):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("shape", [(64, 64), (37, 53), (1, 1), (1, 9), (513, 257)])
def test_downsample_and_upsample(ctx, shape):
    rng = np.random.default_rng(shape[0] * 7 + shape[1])
    p = rng.integers(0, 256, shape, dtype=np.uint8)
    d = ctx.downsample_box(p)
    assert np.array_equal(d, orc.downsample_box(p))
    h, w = shape
    assert np.array_equal(ctx.upsample_nearest(d, w, h), orc.upsample_nearest(d, w, h))


def test_every_colour(ctx):
    # All 2^24: every value that lies near a half, the exact halves among them.
    v = np.arange(1 << 24, dtype=np.uint32)
    r, g, b = ((v >> s & 255).astype(np.uint8).reshape(4096, 4096) for s in (0, 8, 16))
    for x, y in zip(ctx.ycbcr(r, g, b), orc.ycbcr(r, g, b)):
        assert np.array_equal(x, y)
    for x, y in zip(ctx.rgb_from_ycbcr(r, g, b), orc.rgb_from_ycbcr(r, g, b)):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("offset", [0, 1, 4, 8, 13])
@pytest.mark.parametrize("shape", [(2, 15), (3, 16), (5, 33), (8, 64), (7, 130)])
def test_planes_at_any_address(ctx, shape, offset):
    # Word loads and stores at every alignment; a byte on either side of each output stays.
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(shape[1] + offset)
    h, w = shape
    hw, hh = (w + 1) // 2, (h + 1) // 2
    host = [rng.integers(0, 256, (h, w), dtype=np.uint8) for _ in range(3)]

    def place(a):
        buf = torch.full((a.size + 32,), 77, dtype=torch.uint8, device="cuda:0")
        buf[offset: offset + a.size] = torch.from_numpy(a.ravel()).cuda()
        return buf

    def out(n):
        return torch.full((n + 32,), 77, dtype=torch.uint8, device="cuda:0")

    def taken(buf, shape):
        n = shape[0] * shape[1]
        got = buf.cpu().numpy()
        assert (got[:offset] == 77).all() and (got[offset + n:] == 77).all()
        return got[offset: offset + n].reshape(shape)

    L = mb.lib()
    src = [place(a) for a in host]
    dst, down, up = [out(h * w) for _ in range(3)], out(hh * hw), out(h * w)
    torch.cuda.synchronize()
    mb.check(L.mars_ycbcr_device(ctx.handle, *(t.data_ptr() + offset for t in src), h * w,
                                 *(t.data_ptr() + offset for t in dst)))
    mb.check(L.mars_downsample_box_device(ctx.handle, src[0].data_ptr() + offset, w, h,
                                          down.data_ptr() + offset))
    mb.check(L.mars_upsample_nearest_device(ctx.handle, down.data_ptr() + offset, hw, hh,
                                            up.data_ptr() + offset, w, h))
    mse = mb.C.c_double()
    mb.check(L.mars_mse_device(ctx.handle, src[0].data_ptr() + offset, up.data_ptr() + offset,
                               h * w, mb.C.byref(mse)))
    for x, y in zip(dst, orc.ycbcr(*host)):
        assert np.array_equal(taken(x, shape), y)
    want = orc.downsample_box(host[0])
    assert np.array_equal(taken(down, (hh, hw)), want)
    want = orc.upsample_nearest(want, w, h)
    assert np.array_equal(taken(up, shape), want)
    assert mse.value == orc.mse(host[0], want)


@pytest.mark.parametrize("inverse", [False, True])
def test_conversion_at_odd_addresses_in_time(ctx, inverse):
    # A 4K frame whose planes start one byte off: 2.2 times as long as a byte a thread was, and
    # 3.2 times the aligned time, before four bytes shared a conversion.
    torch = pytest.importorskip("torch")
    n = 3840 * 2160
    bufs = [torch.randint(0, 256, (n + 16,), dtype=torch.uint8, device="cuda:0") for _ in range(6)]
    call = mb.lib().mars_rgb_from_ycbcr_device if inverse else mb.lib().mars_ycbcr_device
    times, outs = [], []
    for off in (0, 1):
        if off:
            for b in bufs[:3]:
                b[1:] = b[:-1].clone()
        at = [b.data_ptr() + off for b in bufs]
        best = float("inf")
        for _ in range(5):
            torch.cuda.synchronize()
            t = time.perf_counter()
            for _ in range(100):
                mb.check(call(ctx.handle, *at[:3], n, *at[3:]))
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        times.append(best)
        outs.append([b[off: n + off].clone() for b in bufs[3:]])
    assert all(torch.equal(x, y) for x, y in zip(*outs))
    assert times[1] < 2.5 * times[0]


@pytest.mark.parametrize("n", [1, 15, 16, 17, 4096, 1 << 20, (1 << 20) + 3])
def test_mse(ctx, n):
    rng = np.random.default_rng(n)
    a = rng.integers(0, 256, (1, n), dtype=np.uint8)
    b = rng.integers(0, 256, (1, n), dtype=np.uint8)
    assert ctx.mse(a, b) == orc.mse(a, b)
    assert ctx.mse(a, a) == 0.0
    assert ctx.mse(np.zeros((1, n), np.uint8), np.full((1, n), 255, np.uint8)) == 65025.0


def test_color_pipeline_matches_the_oracle_pipeline(ctx):
    # Config 3 in miniature: RGB -> Y + 4:2:0 Cb/Cr -> per-plane encodes -> MARC container,
    # then decode back; the oracle path runs the same steps with its own restatements.
    rgb = synthetic.rgb(96, 64, 2)
    y_p = dict(min_size=4, max_size=16, shift=2, lam=200.0)
    c_p = dict(min_size=4, max_size=16, shift=2, lam=400.0)
    params = color.ColorEncodeParams(mb.make_params(**y_p), mb.make_params(**c_p))
    data, stats = color.encode_color(ctx, rgb, params)

    y, cb, cr = orc.ycbcr(rgb[..., 0], rgb[..., 1], rgb[..., 2])
    streams = []
    for plane, kw in ((y, y_p), (orc.downsample_box(cb), c_p), (orc.downsample_box(cr), c_p)):
        h, l, res, _, _ = orc.encode(plane, orc.make_params(**kw), allowed_modes=(1, 1, 1, 1))
        streams.append(mb.format_write(mb.Header(*[getattr(h, f) for f, _ in h._fields_]), l, res))
    assert data == color.write_container(color.MODE_RGB_420, streams)
    assert stats.cb_bytes == len(streams[1])

    out = color.decode_color(ctx, data, 10)
    assert out.shape == rgb.shape
    planes = []
    for s in streams:
        h, l, res = mb.format_read(s)
        planes.append(orc.decode(orc.Header(*[getattr(h, f) for f, _ in h._fields_]), l, 10, res))
    H, W = planes[0].shape
    ref = orc.rgb_from_ycbcr(planes[0], orc.upsample_nearest(planes[1], W, H),
                             orc.upsample_nearest(planes[2], W, H))
    assert np.array_equal(out, np.stack(ref, axis=-1))
    assert mb.psnr_from_mse(ctx.mse(out[..., 1], rgb[..., 1])) > 15.0


def test_zoomed_and_auto_colour_decodes(ctx):
    rgb = synthetic.rgb(96, 64, 5)
    kw = dict(min_size=4, max_size=16, shift=2, lam=200.0)
    params = color.ColorEncodeParams(mb.make_params(**kw), mb.make_params(**kw))
    data, _ = color.encode_color(ctx, rgb, params)
    mode, streams = color.read_container(data)
    oplanes = []
    for s in streams:
        h, l, res = mb.format_read(s)
        oh = orc.Header(*[getattr(h, f) for f, _ in h._fields_])
        zh, zl = orc.zoom_leaves(oh, l, 2.0)
        oplanes.append(orc.decode(zh, zl, 10))
    H, W = oplanes[0].shape
    ref = np.stack(orc.rgb_from_ycbcr(oplanes[0], orc.upsample_nearest(oplanes[1], W, H),
                                      orc.upsample_nearest(oplanes[2], W, H)), axis=-1)
    assert np.array_equal(color.decode_color_zoomed(ctx, data, 10, 2.0), ref)
    out, used = color.decode_color_auto(ctx, data, 1, 40)
    uses = []
    oplanes = []
    for s in streams:
        h, l, res = mb.format_read(s)
        oh = orc.Header(*[getattr(h, f) for f, _ in h._fields_])
        p, n = orc.decode_until_stable(oh, l, 1, 40, res)
        oplanes.append(p)
        uses.append(n)
    H, W = oplanes[0].shape
    ref = np.stack(orc.rgb_from_ycbcr(oplanes[0], orc.upsample_nearest(oplanes[1], W, H),
                                      orc.upsample_nearest(oplanes[2], W, H)), axis=-1)
    assert used == max(uses) and np.array_equal(out, ref)


@pytest.mark.parametrize("offset", [0, 1, 4, 13])
@pytest.mark.parametrize("shape", [(1301, 1623), (523, 511), (511, 513), (65, 33)])
def test_ragged_planes_by_chunks_and_by_bytes(ctx, shape, offset):
    # Rows that are no whole chunks, on either side of the sizes that go by bytes.
    torch = pytest.importorskip("torch")
    h, w = shape
    hw, hh = (w + 1) // 2, (h + 1) // 2
    host = np.random.default_rng(w + offset).integers(0, 256, (h, w), dtype=np.uint8)
    src = torch.from_numpy(np.pad(host.ravel(), (offset, 16))).cuda()
    down, up = (torch.full((n + 32,), 77, dtype=torch.uint8, device="cuda:0")
                for n in (hh * hw, h * w))
    torch.cuda.synchronize()
    L = mb.lib()
    mb.check(L.mars_downsample_box_device(ctx.handle, src.data_ptr() + offset, w, h,
                                          down.data_ptr() + offset))
    mb.check(L.mars_upsample_nearest_device(ctx.handle, down.data_ptr() + offset, hw, hh,
                                            up.data_ptr() + offset, w, h))
    torch.cuda.synchronize()
    half = orc.downsample_box(host)
    for buf, want in ((down, half), (up, orc.upsample_nearest(half, w, h))):
        got = buf.cpu().numpy()
        end = offset + want.size
        assert (got[:offset] == 77).all() and (got[end:] == 77).all()
        assert np.array_equal(got[offset:end].reshape(want.shape), want)
