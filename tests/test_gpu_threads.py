"""Contexts on several host threads at once: every call's records are those it gives alone."""
import threading

import numpy as np
import pytest
import torch

import mars_b200 as mb
from mars_b200 import synthetic

pytestmark = pytest.mark.gpu


def _side_by_side(calls, repeats):
    """Runs each call `repeats` times on a thread of its own; the calls' results, by call."""
    errors, start = [], threading.Barrier(len(calls))
    results = [[] for _ in calls]

    def work(call, out):
        try:
            start.wait(60)
            for _ in range(repeats):
                out.append(call())
        except Exception as e:  # reported on the test's thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=a) for a in zip(calls, results)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors, errors[0]
    return results


@pytest.mark.parametrize("path,first,second", [
    ("auto", (4, 2), (8, 2)),      # the unit form's launch with and without size 8
    ("simt", (16, 2), (16, 16)),   # the CUDA-core kernel's domain tiles, by stride
])
def test_contexts_of_different_levels(monkeypatch, path, first, second):
    monkeypatch.setenv("MARS_UNIT_TILES", "0")
    w = h = 192
    plane = torch.from_numpy(synthetic.gray(w, h, 5)).cuda()
    torch.cuda.synchronize()
    ctxs = [mb.Context(0) for _ in range(4)]

    def call(ctx, size, shift):
        params = mb.make_params(min_size=size, max_size=size, shift=shift)
        n = mb.C.c_size_t()
        mb.check(mb.lib().mars_search_nodes_device(ctx.handle, plane.data_ptr(), w, h,
                                                   mb.C.byref(params), None, 0, mb.C.byref(n),
                                                   None))
        out = torch.zeros(n.value, 80, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()

        def run():
            mb.check(mb.lib().mars_search_nodes_device(ctx.handle, plane.data_ptr(), w, h,
                                                       mb.C.byref(params), out.data_ptr(), n.value,
                                                       mb.C.byref(n), None))

        def records():
            torch.cuda.synchronize()
            return out.cpu().numpy().tobytes()
        return run, records

    for ctx in ctxs:
        ctx.set_search_path(path)
    runs, records = zip(*[call(ctx, *level) for ctx, level in zip(ctxs, 2 * (first, second))])
    for run in runs:
        run()
    alone = [r() for r in records]
    # Calls that only launch: a collision on what they share is a matter of host time alone.
    _side_by_side(runs, 3000)
    assert [r() for r in records] == alone
    for ctx in ctxs:
        ctx.close()


def test_two_contexts_tables_of_different_levels():
    # The integer launch of a table's levels: size 16 alone beside 64.
    img = synthetic.gray(192, 192, 5)
    ctxs = [mb.Context(0) for _ in range(2)]

    def call(ctx, size):
        params = mb.make_params(min_size=size, max_size=size, shift=4)
        grid = [i * size for i in range(192 // size)]
        rows, cols = [r for r in grid for _ in grid], grid * len(grid)

        def run():
            table = ctx.search_provider(img, params)
            records = table.search_many(rows, cols, size, 4)[0].tobytes()
            table.close()
            return records
        return run

    calls = [call(ctx, size) for ctx, size in zip(ctxs, (16, 64))]
    alone = [c() for c in calls]
    for want, got in zip(alone, _side_by_side(calls, 300)):
        assert all(g == want for g in got)
    for ctx in ctxs:
        ctx.close()


def test_one_shot_decodes_while_the_stream_changes():
    w, h = 404, 300
    leaves = synthetic.quadtree_leaves(w, h, 3, min_size=4)
    hdr = mb.Header(bits_alfa=4, bits_beta=7, min_size=4, max_size=32, shift=2, width=w, height=h,
                    int_max_alfa=32)
    leaves["mode"][::3][leaves["mode"][::3] == 2] = 3
    pick = leaves["mode"] == 3
    levels = np.random.default_rng(1).integers(
        -2, 3, int((leaves["size"][pick].astype(np.int64) ** 2).sum())).astype(np.int32)
    ctx = mb.Context(0)
    want = ctx.decode_until_stable(hdr, leaves, 1, 24, levels)
    plan = ctx.decode_plan(hdr, leaves, levels)
    other = torch.cuda.Stream()
    done = threading.Event()

    def switch():
        while not done.is_set():
            ctx.set_stream(other.cuda_stream)
            ctx.set_stream(0)

    def decode():
        plane, used = ctx.decode_until_stable(hdr, leaves, 1, 24, levels)
        made = ctx.decode_plan(hdr, leaves, levels)
        made.close()  # released while the other thread changes the stream
        return used, plane.tobytes()

    turning = threading.Thread(target=switch)
    turning.start()
    try:
        got = _side_by_side([decode, decode], 60)
    finally:
        done.set()
        turning.join(60)
    assert all(g == (want[1], want[0].tobytes()) for side in got for g in side)
    torch.cuda.synchronize()
    plan.close()
    ctx.close()


def test_contexts_come_and_go_beside_each_other():
    # Calls of every context take the device's call streams; the last context out gives them back.
    params = mb.make_params(min_size=4, max_size=16, shift=4, lam=200.0)
    images = [synthetic.gray(112, 80, seed) for seed in range(3)]

    def encode(ctx, img):
        _, leaves, levels, count = ctx.encode(img, params, allowed_modes=(1, 1, 1, 1))
        return leaves.tobytes(), levels.tobytes(), count.search_evals

    with mb.Context(0) as ctx:
        want = [encode(ctx, img) for img in images]
    for _ in range(3):
        ctxs = [mb.Context(0) for _ in images]
        got = _side_by_side([lambda c=c, i=i: encode(c, i) for c, i in zip(ctxs, images)], 8)
        for w, g in zip(want, got):
            assert all(x == w for x in g)
        for ctx in ctxs:
            ctx.close()


@pytest.mark.parametrize("lam,modes", [(None, (1, 0, 1, 0)), (200.0, (1, 0, 1, 0)),
                                       (200.0, (1, 1, 1, 1))])
def test_fisher_encodes_beside_each_other(lam, modes):
    # 4,032 nodes: alone the walks run on the device, beside others without residuals on the host.
    params = mb.make_params(min_size=4, max_size=16, shift=4, lam=lam)
    images = [synthetic.gray(256, 192, seed) for seed in range(3)]

    def encode(ctx, img):
        _, leaves, levels, count = ctx.encode(img, params, allowed_modes=modes, method="fisher")
        return leaves.tobytes(), levels.tobytes(), count.search_evals, count.warmup_evals

    with mb.Context(0) as ctx:
        want = [encode(ctx, img) for img in images]
        again = [encode(ctx, img) for img in images]
        assert again == want
        got = _side_by_side([lambda i=i: encode(ctx, i) for i in images], 8)
        for w, g in zip(want, got):
            assert all(x == w for x in g)
    ctxs = [mb.Context(0) for _ in images]
    got = _side_by_side([lambda c=c, i=i: encode(c, i) for c, i in zip(ctxs, images)], 8)
    for w, g in zip(want, got):
        assert all(x == w for x in g)
    for ctx in ctxs:
        ctx.close()
