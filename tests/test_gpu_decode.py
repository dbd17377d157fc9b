"""Parity of the decode gather (mars_decode, mars_decode_plan_*) against the oracle's
decode_iterative (crates/mars-codec/src/ifs.rs:281-309, 406-484), bit-exact."""
import time

import numpy as np
import pytest

import mars_b200 as mb
from mars_b200 import synthetic
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = mb.Context(0)
    yield c
    c.close()


def _hdr(w, h, bits_alfa=4, bits_beta=7, int_max_alfa=32):
    return mb.Header(bits_alfa, bits_beta, 4, 32, 2, w, h, int_max_alfa)


def _ohdr(hdr):
    return orc.Header(*[getattr(hdr, f) for f, _ in orc.Header._fields_])


@pytest.mark.parametrize("w,h,seed", [(256, 256, 1), (260, 200, 2), (512, 384, 3), (64, 96, 4)])
def test_synthetic_quadtree_maps(ctx, w, h, seed):
    # Modes 0/1/2, all isometries; (260, 200) leaves a border no leaf covers (written 0).
    leaves = synthetic.quadtree_leaves(w, h, seed)
    hdr = _hdr(w, h)
    for iters in (1, 2, 10):
        assert np.array_equal(ctx.decode(hdr, leaves, iters), orc.decode(_ohdr(hdr), leaves, iters))


@pytest.mark.parametrize("bits_alfa,bits_beta,int_max_alfa", [(2, 5, 32), (6, 9, 64), (16, 16, 255),
                                                               (0, 1, 32)])
def test_header_bit_widths(ctx, bits_alfa, bits_beta, int_max_alfa):
    w = h = 128
    leaves = synthetic.quadtree_leaves(w, h, 7, bits_alfa=bits_alfa, bits_beta=bits_beta)
    hdr = _hdr(w, h, bits_alfa, bits_beta, int_max_alfa)
    assert np.array_equal(ctx.decode(hdr, leaves, 6), orc.decode(_ohdr(hdr), leaves, 6))


def test_unaligned_leaves_one_pixel_cells(ctx):
    # Leaves of size 5 at multiples of 5: the owner map falls back to 1x1 cells.
    w = h = 30
    rng = np.random.default_rng(5)
    rows = []
    for r in range(0, h, 5):
        for c in range(0, w, 5):
            mode = int(rng.integers(0, 3))
            qalfa = int(rng.integers(1, 17)) if mode == 2 else 0
            dr, dc = int(rng.integers(0, h - 10 + 1)), int(rng.integers(0, w - 10 + 1))
            rows.append((r, c, 5, mode, qalfa, int(rng.integers(0, 128)), int(rng.integers(0, 8)),
                         dr if mode == 2 else 0, dc if mode == 2 else 0,
                         int(rng.integers(-80, 81)) if mode == 1 else 0,
                         int(rng.integers(-80, 81)) if mode == 1 else 0))
    leaves = np.array(rows, dtype=mb.LEAF_DTYPE)
    hdr = _hdr(w, h)
    for iters in (1, 4):
        assert np.array_equal(ctx.decode(hdr, leaves, iters), orc.decode(_ohdr(hdr), leaves, iters))


def _mode3(leaves, rng, p_zero=0.5):
    """Turn the domain leaves into mode-3 leaves, half of them with qalfa = 0 (no domain
    read, the residual still added: ifs.rs:459-479), with random residual levels."""
    out = leaves.copy()
    pool = []
    for k in range(len(out)):
        if out["mode"][k] != 2:
            continue
        out["mode"][k] = 3
        if rng.random() < p_zero:
            out["qalfa"][k] = 0
        n = int(out["size"][k]) ** 2
        lv = np.zeros(n, np.int32)
        nz = rng.choice(n, size=min(n, 6), replace=False)
        lv[nz] = rng.integers(-20, 21, size=len(nz))
        pool.append(lv)
    return out, (np.concatenate(pool) if pool else np.zeros(0, np.int32))


@pytest.mark.parametrize("w,h,seed", [(128, 96, 11), (30, 30, 12)])
def test_zero_alpha_residual_leaves(ctx, w, h, seed):
    rng = np.random.default_rng(seed)
    if w == 30:  # size-5 leaves: the one-pixel-cell kernel
        rows = []
        for r in range(0, h, 5):
            for c in range(0, w, 5):
                dr, dc = int(rng.integers(0, h - 9)), int(rng.integers(0, w - 9))
                rows.append((r, c, 5, 2, int(rng.integers(1, 17)), int(rng.integers(0, 128)),
                             int(rng.integers(0, 8)), dr, dc, 0, 0))
        base = np.array(rows, dtype=mb.LEAF_DTYPE)
    else:
        base = synthetic.quadtree_leaves(w, h, seed)
    leaves, pool = _mode3(base, rng)
    assert (leaves["mode"] == 3).any() and ((leaves["mode"] == 3) & (leaves["qalfa"] == 0)).any()
    hdr = _hdr(w, h)
    for iters in (1, 5):
        assert np.array_equal(ctx.decode(hdr, leaves, iters, pool),
                              orc.decode(_ohdr(hdr), leaves, iters, pool))


def test_later_leaves_overwrite_earlier(ctx):
    # decode_step writes leaves in order, so a later leaf wins where two overlap.
    w = h = 64
    base = synthetic.quadtree_leaves(w, h, 9)
    extra = synthetic.quadtree_leaves(w, h, 10, max_size=16)[:20]
    leaves = np.concatenate([base, extra])
    hdr = _hdr(w, h)
    for iters in (1, 5):
        assert np.array_equal(ctx.decode(hdr, leaves, iters), orc.decode(_ohdr(hdr), leaves, iters))


def test_empty_leaf_list_decodes_to_zero(ctx):
    hdr = _hdr(32, 16)
    out = ctx.decode(hdr, np.zeros(0, dtype=mb.LEAF_DTYPE), 3)
    assert out.shape == (16, 32) and not out.any()
    assert np.array_equal(out, orc.decode(_ohdr(hdr), np.zeros(0, dtype=mb.LEAF_DTYPE), 3))


@pytest.mark.parametrize("iters", [0, 1, 2, 7, 10])
def test_decode_plan_matches_decode(ctx, iters):
    import torch
    w, h = 320, 256
    leaves = synthetic.quadtree_leaves(w, h, 11)
    hdr = _hdr(w, h)
    plan = ctx.decode_plan(hdr, leaves)
    dev = torch.empty(w * h, dtype=torch.uint8, device="cuda:0")
    for _ in range(2):  # a plan runs any number of times
        dev.fill_(7)
        torch.cuda.synchronize()
        plan.run(iters, dev.data_ptr())
        torch.cuda.synchronize()
        got = dev.cpu().numpy().reshape(h, w)
        assert np.array_equal(got, ctx.decode(hdr, leaves, iters))
        assert np.array_equal(got, orc.decode(_ohdr(hdr), leaves, iters))
    plan.close()


def test_decode_rejects_out_of_range_leaves(ctx):
    hdr = _hdr(64, 64)
    leaves = synthetic.quadtree_leaves(64, 64, 12)
    k = int(np.flatnonzero(leaves["mode"] == 2)[0])
    bad = leaves.copy()
    bad["qalfa"][k] = 17  # above 2^bits_alfa
    with pytest.raises(mb.MarsError) as e:
        ctx.decode(hdr, bad, 2)
    assert e.value.code == -1
    bad = leaves.copy()
    bad["qbeta"][k] = 128  # above 2^bits_beta - 1
    with pytest.raises(mb.MarsError) as e:
        ctx.decode(hdr, bad, 2)
    assert e.value.code == -1
    bad = leaves.copy()
    bad["mode"][k] = 3  # a mode-3 leaf without its residual levels
    with pytest.raises(mb.MarsError, match="residual pool") as e:
        ctx.decode(hdr, bad, 2)
    assert e.value.code == -1
    bad["mode"][k] = 4
    with pytest.raises(mb.MarsError) as e:
        ctx.decode(hdr, bad, 2)
    assert e.value.code == -1
    with pytest.raises(mb.MarsError) as e:
        ctx.decode_plan(_hdr(70000, 8), np.zeros(0, dtype=mb.LEAF_DTYPE))
    assert e.value.code == -1


@pytest.mark.parametrize("threshold", [0, 1, 3, 255])
def test_until_stable_matches_the_oracle(ctx, threshold):
    # Aligned maps take the 4x4-cell kernel, the size-5 map the one-pixel kernel.
    rng = np.random.default_rng(9)
    maps = [(synthetic.quadtree_leaves(160, 96, 21), 160, 96, None)]
    base = synthetic.quadtree_leaves(128, 96, 22)
    leaves3, pool = _mode3(base, rng, p_zero=0.3)
    maps.append((leaves3, 128, 96, pool))
    rows = []
    for r in range(0, 30, 5):
        for c in range(0, 30, 5):
            rows.append((r, c, 5, 2, int(rng.integers(1, 17)), int(rng.integers(0, 128)),
                         int(rng.integers(0, 8)), int(rng.integers(0, 21)), int(rng.integers(0, 21)),
                         0, 0))
    maps.append((np.array(rows, dtype=mb.LEAF_DTYPE), 30, 30, None))
    for leaves, w, h, res in maps:
        hdr = _hdr(w, h)
        got, used = ctx.decode_until_stable(hdr, leaves, threshold, 40, res)
        want, oused = orc.decode_until_stable(_ohdr(hdr), leaves, threshold, 40, res)
        assert used == oused and np.array_equal(got, want)


def test_plan_until_stable_on_the_device(ctx):
    import torch
    leaves = synthetic.quadtree_leaves(256, 192, 23)
    hdr = _hdr(256, 192)
    plan = ctx.decode_plan(hdr, leaves)
    out = torch.zeros(256 * 192, dtype=torch.uint8, device="cuda:0")
    used = mb.C.c_uint32()
    mb.check(mb.lib().mars_decode_plan_run_until_stable(plan._h, 2, 30, out.data_ptr(),
                                                        mb.C.byref(used)))
    torch.cuda.synchronize()
    want, oused = orc.decode_until_stable(_ohdr(hdr), leaves, 2, 30)
    assert used.value == oused
    assert np.array_equal(out.cpu().numpy().reshape(192, 256), want)
    plan.close()


@pytest.mark.parametrize("factor", [2.0, 1.5, 0.5])
def test_zoomed_decode_matches_the_oracle(ctx, factor):
    img = synthetic.gray(128, 96, 24)
    hdr, leaves, res, _ = ctx.encode(img, mb.make_params(min_size=4, max_size=16, shift=4, lam=200.0),
                                     allowed_modes=(1, 1, 1, 1))
    zh, zl = mb.zoom_leaves(hdr, leaves, factor)
    ozh, ozl = orc.zoom_leaves(_ohdr(hdr), leaves, factor)
    assert zl.tobytes() == ozl.tobytes()
    got = ctx.decode(zh, zl, 10)
    assert got.shape == (round(96 * factor), round(128 * factor))
    assert np.array_equal(got, orc.decode(ozh, ozl, 10))


@pytest.mark.parametrize("w,h,seed", [(320, 256, 11), (1024, 768, 13), (516, 302, 14),
                                      (2500, 300, 15), (2052, 148, 16)])
def test_source_ordered_plan_steps_match_the_oracle(ctx, monkeypatch, w, h, seed):
    """The source-ordered steps large planes take (domain cells gathered in the order of their
    windows' source rows into a cell buffer, then placed in output order) give the cell
    kernel's bytes: forced on here for planes small enough for the oracle; (516, 302) leaves a
    border no leaf covers and a last cell row cut by the plane's edge."""
    import torch
    monkeypatch.setenv("MARS_DECODE_SORTED", "1")
    leaves = synthetic.quadtree_leaves(w, h, seed)
    hdr = _hdr(w, h)
    plan = ctx.decode_plan(hdr, leaves)
    dev = torch.empty(w * h, dtype=torch.uint8, device="cuda:0")
    for iters in (1, 3, 10):
        dev.fill_(7)
        torch.cuda.synchronize()
        plan.run(iters, dev.data_ptr())
        torch.cuda.synchronize()
        got = dev.cpu().numpy().reshape(h, w)
        assert np.array_equal(got, orc.decode(_ohdr(hdr), leaves, iters)), iters
    plan.close()


@pytest.mark.parametrize("w,h,bits_alfa,bits_beta,int_max_alfa",
                         [(64, 64, 4, 7, 32), (132, 92, 4, 7, 32), (96, 64, 5, 7, 64),
                          (96, 64, 3, 1, 8), (96, 64, 5, 16, 32), (64, 64, 6, 7, 255),
                          (1024, 1024, 4, 7, 32), (2048, 1536, 4, 7, 32)])
def test_integer_values_and_one_launch_steps(ctx, w, h, bits_alfa, bits_beta, int_max_alfa):
    # Every contrast and offset of the header's widths (those with an integer form and those
    # without), affine leaves past both ends of a byte, planes on both sides of the largest one
    # whose steps run in one launch; the plan into a buffer at an 8-byte address.
    torch = pytest.importorskip("torch")
    leaves = synthetic.quadtree_leaves(w, h, w + bits_alfa, bits_alfa=bits_alfa,
                                       bits_beta=bits_beta)
    rng = np.random.default_rng(w * bits_beta)
    dom = (leaves["mode"] != 1) & (leaves["qalfa"] != 0)
    leaves["qalfa"][dom] = rng.integers(1, (1 << bits_alfa) + 1, int(dom.sum()))
    leaves["qbeta"] = rng.integers(0, 1 << bits_beta, len(leaves))
    affine = np.flatnonzero(leaves["mode"] == 1)
    leaves["qgx"][affine[::2]] = rng.integers(-5000, 5001, len(affine[::2]))
    leaves["qgy"][affine[1::3]] = rng.integers(-1 << 30, 1 << 30, len(affine[1::3]))
    hdr = _hdr(w, h, bits_alfa, bits_beta, int_max_alfa)
    plan = ctx.decode_plan(hdr, leaves)
    buf = torch.zeros(w * h + 16, dtype=torch.uint8, device="cuda:0")
    torch.cuda.synchronize()
    for iters in (1, 2, 5):
        want = orc.decode(_ohdr(hdr), leaves, iters)
        assert np.array_equal(ctx.decode(hdr, leaves, iters), want)
        for _ in range(2):
            plan.run(iters, buf.data_ptr() + 8)
        ctx.decode(hdr, leaves[:0], 1)  # waits for the context's stream
        assert np.array_equal(buf.cpu().numpy()[8: 8 + w * h].reshape(h, w), want)
    plan.close()


@pytest.mark.parametrize("w,h,min_size,max_size", [(64, 64, 2, 16), (96, 80, 4, 32),
                                                   (256, 128, 4, 64), (512, 256, 8, 128)])
def test_residuals_of_every_size(ctx, w, h, min_size, max_size):
    # Mode-3 leaves of each size: rebuilt on the device up to 64, on the host beyond; levels of
    # every magnitude and lists of zeros, against the oracle's inverse transform bit for bit.
    leaves = synthetic.quadtree_leaves(w, h, w + max_size, min_size=min_size, max_size=max_size)
    rng = np.random.default_rng(w)
    pick = (leaves["mode"] == 2) & (rng.random(len(leaves)) < 0.7)
    leaves["mode"][pick] = 3
    assert pick.any()
    n = int((leaves["size"][pick].astype(np.int64) ** 2).sum())
    levels = np.where(rng.random(n) < 0.3, rng.integers(-63, 64, n), 0).astype(np.int32)
    hdr = _hdr(w, h)
    want = orc.decode(_ohdr(hdr), leaves, 3, levels)
    assert np.array_equal(ctx.decode(hdr, leaves, 3, levels), want)
    plane, used = ctx.decode_until_stable(hdr, leaves, 1, 6, levels)
    oplane, oused = orc.decode_until_stable(_ohdr(hdr), leaves, 1, 6, levels)
    assert used == oused and np.array_equal(plane, oplane)


@pytest.mark.parametrize("w,h,bits_alfa", [(128, 96, 4), (516, 132, 4), (256, 258, 7)])
def test_source_ordered_steps_with_overwritten_leaves(ctx, monkeypatch, w, h, bits_alfa):
    # Leaves on top of others: a leaf's rows of windows keep holes, down to none of its cells.
    monkeypatch.setenv("MARS_DECODE_SORTED", "1")
    under = synthetic.quadtree_leaves(w, h, w, bits_alfa=bits_alfa)
    over = synthetic.quadtree_leaves(w, h, w + 1, bits_alfa=bits_alfa)
    leaves = np.concatenate([under, over[over["size"] <= 8][::2], under[under["size"] >= 16][::5]])
    hdr = _hdr(w, h, bits_alfa)
    plan = ctx.decode_plan(hdr, leaves)
    torch = pytest.importorskip("torch")
    out = torch.zeros(h, w, dtype=torch.uint8, device="cuda:0")
    torch.cuda.synchronize()
    for iters in (1, 4):
        plan.run(iters, out.data_ptr())
        ctx.decode(hdr, leaves[:0], 1)  # waits for the context's stream
        assert np.array_equal(out.cpu().numpy(), orc.decode(_ohdr(hdr), leaves, iters))
    plan.close()


@pytest.mark.parametrize("w,h,min_size", [(64, 64, 4), (100, 77, 2), (516, 260, 4)])
def test_repeated_plan_runs(ctx, w, h, min_size):
    # A run that repeats the last one's steps and output replays them; others change either, or
    # both, between replays.
    torch = pytest.importorskip("torch")
    leaves = synthetic.quadtree_leaves(w, h, w, min_size=min_size)
    hdr = _hdr(w, h)
    plan = ctx.decode_plan(hdr, leaves)
    outs = [torch.zeros(h, w, dtype=torch.uint8, device="cuda:0") for _ in range(2)]
    want = {n: orc.decode(_ohdr(hdr), leaves, n) for n in (1, 2, 3, 70)}
    torch.cuda.synchronize()
    for k, n in [(0, 3)] * 3 + [(1, 3), (0, 3), (1, 2), (1, 2), (1, 2), (0, 3), (0, 3), (0, 1),
                                (0, 1), (1, 70), (1, 70), (1, 2)]:
        outs[k].fill_(7)
        torch.cuda.synchronize()
        plan.run(n, outs[k].data_ptr())
        torch.cuda.synchronize()
        assert np.array_equal(outs[k].cpu().numpy(), want[n]), (k, n)
    plan.close()


@pytest.mark.parametrize("at", [0, 1, 4, 6])
def test_source_ordered_runs_into_any_address(ctx, monkeypatch, at):
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("MARS_DECODE_SORTED", "1")
    w, h = 516, 260
    leaves = synthetic.quadtree_leaves(w, h, 8, min_size=4)
    hdr = _hdr(w, h)
    plan = ctx.decode_plan(hdr, leaves)
    whole = torch.full((w * h + 16,), 7, dtype=torch.uint8, device="cuda:0")
    torch.cuda.synchronize()
    for n in (1, 2, 7):
        plan.run(n, whole.data_ptr() + at)
        torch.cuda.synchronize()
        got = whole.cpu().numpy()
        assert np.array_equal(got[at: at + w * h].reshape(h, w), orc.decode(_ohdr(hdr), leaves, n))
        assert (got[:at] == 7).all() and (got[at + w * h:] == 7).all()


@pytest.mark.parametrize("w,h,min_size,wide", [(64, 64, 4, None), (100, 77, 2, None),
                                               (516, 260, 4, None), (516, 260, 4, "1")])
def test_plan_runs_of_every_count(ctx, monkeypatch, w, h, min_size, wide):
    # More step counts than a plan keeps graphs for, into three buffers by turns, one of them at an
    # odd address; wide: the source-ordered steps.
    torch = pytest.importorskip("torch")
    if wide:
        monkeypatch.setenv("MARS_DECODE_SORTED", wide)
    leaves = synthetic.quadtree_leaves(w, h, w + 1, min_size=min_size)
    hdr = _hdr(w, h)
    plan = ctx.decode_plan(hdr, leaves)
    apart = (w * h + 256) // 256 * 256
    whole = torch.zeros(3 * apart, dtype=torch.uint8, device="cuda:0")
    starts = (0, apart, 2 * apart - 1)
    torch.cuda.synchronize()
    for n in (3, 2, 10, 1, 65, 7, 4, 10, 2):
        want = orc.decode(_ohdr(hdr), leaves, n)
        for k in (0, 0, 1, 2, 1, 0):
            whole.fill_(7)
            torch.cuda.synchronize()
            plan.run(n, whole.data_ptr() + starts[k])
            torch.cuda.synchronize()
            got = whole.cpu().numpy()
            out = got[starts[k]: starts[k] + w * h].copy()
            assert np.array_equal(out.reshape(h, w), want), (n, k)
            got[starts[k]: starts[k] + w * h] = 7
            assert (got == 7).all()  # nothing beside the output
    plan.close()


def test_runs_into_odd_addresses_in_time(ctx):
    # Only the last step stores there.  (With every other one, one pixel a thread, 2.9 times the
    # aligned time.)
    torch = pytest.importorskip("torch")
    w = h = 1280
    plan = ctx.decode_plan(_hdr(w, h), synthetic.quadtree_leaves(w, h, 5, min_size=4))
    out = torch.zeros(w * h + 8, dtype=torch.uint8, device="cuda:0")
    times = []
    for at in (0, 1):
        best = float("inf")
        for _ in range(5):
            torch.cuda.synchronize()
            t = time.perf_counter()
            for _ in range(50):
                plan.run(10, out.data_ptr() + at)
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        times.append(best)
    assert times[1] < 2.3 * times[0]
    plan.close()
