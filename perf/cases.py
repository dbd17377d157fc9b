"""Timed workloads of the codec's public calls.

`listed()` names twelve workloads, `draw()` gives more of the same ranges, `prepare()` makes
what a program holds before the call (planes from a seed, a context, a plan), `run()` is one
call, `work()` the bytes and operations it cannot do without, and `exact()` the results in
64-bit arithmetic where they are computed numbers.

The kinds:
  encode   one plane in, leaves out: through a search plan of the geometry, or through
           Context.encode (exhaustive, Fisher-classified or ranked search)
  nodes    the search of every quadtree node, plane and records in device memory
  blocks   the search of one level's blocks, host plane in, records out
  decode   fixed-point iterations of a prepared leaf list into a device buffer
  stable   a one-shot decode until the plane stops changing, host leaves in, host plane out
  refine   the attractor's loss and gradients for one set of contrasts and offsets
  colour   RGB to YCbCr 4:2:0 planes, back to RGB, and the error between the two
"""
import math

import numpy as np
import torch

import mars_b200 as mb
from mars_b200 import synthetic

DEV = "cuda:0"


class State(dict):
    """A case's context, plan and buffers; the plan goes before the context it belongs to."""

    def __del__(self):
        for key in ("plan", "ctx"):
            if key in self:
                self[key].close()


class Rows:
    """An array of fixed length for a result whose length depends on the plane: the result's
    rows, then zeros."""

    def __init__(self, *shape, dtype):
        self.all, self.used = np.zeros(shape, dtype), 0

    def put(self, rows):
        n = len(rows)
        self.all[:n] = rows
        self.all[n: self.used] = 0
        self.used = n
        return self.all


def _most_leaves(case):
    """Whole min_size cells, and pixel leaves along two odd borders."""
    return (case["w"] // 4) * (case["h"] // 4) + 4 * (case["w"] + case["h"])


def listed():
    return [
        # The smallest call: a thumbnail through Context.encode at the command line's
        # defaults (sizes 16..4, stride 4, threshold walk).
        dict(name="encode_thumb_96x80", kind="encode", entry="context", method="exhaustive", k=1,
             w=96, h=80, min=4, max=16, shift=4, lam=0.0, modes="02"),
        # The usual call: one 512x512 plane through its geometry's plan, rate-distortion walk
        # over all four modes.
        dict(name="encode_rd_512", kind="encode", entry="plan", method="exhaustive", k=1,
             w=512, h=512, min=4, max=32, shift=2, lam=200.0, modes="0123"),
        # The largest: a 1.5 Mpixel plane, default modes.
        dict(name="encode_rd_1536x1024", kind="encode", entry="plan", method="exhaustive", k=1,
             w=1536, h=1024, min=4, max=32, shift=2, lam=200.0, modes="02"),
        # The classified search at the colour corpus' luma size, threshold walk.
        dict(name="encode_fisher_768x512", kind="encode", entry="context", method="fisher", k=1,
             w=768, h=512, min=4, max=16, shift=2, lam=0.0, modes="02"),
        # Ranked candidates (three a node) on an odd-sized plane with forced border splits.
        dict(name="encode_ranked_250x190", kind="encode", entry="context", method="exhaustive",
             k=3, w=250, h=190, min=4, max=16, shift=2, lam=200.0, modes="0123"),
        # A device-resident caller: every node of a VGA plane at the default stride.
        dict(name="nodes_640x480", kind="nodes", w=640, h=480, min=4, max=16, shift=4),
        # The fixed-grid search of one level from host memory.
        dict(name="blocks8_384x256", kind="blocks", w=384, h=256, size=8, shift=2, n=1536),
        # A small preview decode: ten steps of a 512x512 leaf list.
        dict(name="decode_512", kind="decode", w=512, h=512, min=4, iters=10, resid=False),
        # A large decode: ten steps of a plane pair larger than L2.
        dict(name="decode_8192", kind="decode", w=8192, h=8192, min=4, iters=10, resid=False),
        # A one-shot decode of a stream with residual leaves, until it is stable.
        dict(name="stable_1000x752", kind="stable", w=1000, h=752, min=4, iters=32, resid=True),
        # The refinement's differentiable pair on one encoded 512x512 plane.
        dict(name="refine_512", kind="refine", w=512, h=512, lam=200.0),
        # The colour path of a 4K frame, both directions, and its metric.
        dict(name="colour_3840x2160", kind="colour", w=3840, h=2160),
    ]


def _between(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _sides(rng, lo, hi):
    """Sides of a plane of lo..hi pixels (log-uniform), aspect 1:2 to 2:1, mostly multiples of
    4 or 16, sometimes any even number, sometimes odd ones."""
    area, aspect = _between(rng, lo, hi), _between(rng, 0.5, 2.0)
    step = rng.choice((16, 16, 4, 4, 2, 1))
    return tuple(max(40, int(s) // step * step)
                 for s in (math.sqrt(area * aspect), math.sqrt(area / aspect)))


def draw(rng):
    kind = rng.choice(("encode", "encode", "encode", "encode", "nodes", "blocks", "decode",
                       "decode", "stable", "refine", "colour"))
    if kind == "encode":
        what = rng.choice(("plan", "plan", "context", "fisher", "ranked"))
        w, h = _sides(rng, 64 * 64, {"fisher": 600e3, "ranked": 250e3}.get(what, 1e6))
        lam = round(_between(rng, 50.0, 800.0), 1)
        if what != "ranked" and rng.random() < 0.4:
            lam = 0.0
        return dict(kind="encode", entry="plan" if what == "plan" else "context",
                    method="fisher" if what == "fisher" else "exhaustive",
                    k=rng.randint(2, 8) if what == "ranked" else 1, w=w, h=h, min=4,
                    max=rng.choice((16, 32)), shift=rng.choice((2, 2, 4, 8)), lam=lam,
                    modes=rng.choice(("02", "0123")))
    if kind == "nodes":
        w, h = _sides(rng, 64 * 64, 800e3)
        return dict(kind=kind, w=w, h=h, min=4, max=rng.choice((16, 32, 64)),
                    shift=rng.choice((2, 4, 4, 8)))
    if kind == "blocks":
        size = rng.choice((4, 8, 16, 32, 64))
        w, h = _sides(rng, 4 * (2 * size + 8) ** 2, 400e3)
        return dict(kind=kind, w=w, h=h, size=size, shift=rng.choice((2, 4, 8)),
                    n=int(_between(rng, 1, (w // size) * (h // size))))
    if kind in ("decode", "stable"):
        w, h = _sides(rng, 128 * 128, 50e6 if kind == "decode" else 4e6)
        return dict(kind=kind, w=w, h=h, min=rng.choice((2, 4, 4, 4, 8)),
                    iters=rng.randint(6, 16) if kind == "decode" else rng.randint(16, 40),
                    resid=kind == "stable" and rng.random() < 0.5)
    if kind == "refine":
        w, h = _sides(rng, 96 * 96, 400e3)
        return dict(kind=kind, w=w, h=h, lam=round(_between(rng, 50.0, 800.0), 1))
    w, h = _sides(rng, 256 * 256, 9e6)
    return dict(kind="colour", w=w, h=h)


# ---- inputs ----

def _params(case, lam):
    return mb.make_params(min_size=case["min"], max_size=case["max"], shift=case["shift"],
                          lam=lam or None)


def _leaf_list(case, seed):
    """A quadtree leaf list as a stream holds it (flat, affine and domain leaves of sizes
    32..min), with a residual on a quarter of the domain leaves when asked."""
    leaves = synthetic.quadtree_leaves(case["w"], case["h"], seed, min_size=case["min"])
    hdr = mb.Header(bits_alfa=4, bits_beta=7, min_size=case["min"], max_size=32, shift=2,
                    width=case["w"], height=case["h"], int_max_alfa=32)
    levels = None
    if case["resid"]:
        rng = np.random.default_rng(seed + 1)
        pick = (leaves["mode"] == 2) & (leaves["size"] <= 16) & (rng.random(len(leaves)) < 0.25)
        leaves["mode"][pick] = 3
        n = int((leaves["size"][pick].astype(np.int64) ** 2).sum())
        levels = np.where(rng.random(n) < 0.1, rng.integers(-3, 4, n), 0).astype(np.int32)
    return hdr, leaves, levels


def _origins(case, seed):
    """The level's grid in raster order, or a sorted sample of it."""
    s = case["size"]
    rows, cols = np.meshgrid(np.arange(case["h"] // s) * s, np.arange(case["w"] // s) * s,
                             indexing="ij")
    pick = np.random.default_rng(seed).permutation(rows.size)[: case["n"]]
    pick.sort()
    return rows.ravel()[pick].astype(np.uint32), cols.ravel()[pick].astype(np.uint32)


def _coded(ctx, case, seed):
    """An encoded plane (flat and domain leaves): what the refinement starts from."""
    img = synthetic.gray(case["w"], case["h"], seed)
    params = mb.make_params(min_size=4, max_size=32, shift=2, lam=case["lam"])
    hdr, leaves, _, _ = ctx.encode(img, params, allowed_modes=(1, 0, 1, 0))
    return img, hdr, leaves


def _rgb(case, seed):
    """A smooth colour gradient with noise, made on the device."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    n = case["w"] * case["h"]
    ramp = torch.linspace(0.0, 1.0, n, device=DEV)
    planes = []
    for _ in range(3):
        a, b = torch.rand(2, generator=g, device=DEV).tolist()
        p = 255.0 * (a + (b - a) * ramp) + 12.0 * torch.randn(n, generator=g, device=DEV)
        planes.append(p.round().clamp(0, 255).to(torch.uint8))
    return planes


def prepare(case, seed):
    kind, w, h = case["kind"], case["w"], case["h"]
    ctx = mb.Context(0)
    st = State(case=case, kind=kind, ctx=ctx)
    if kind == "encode":
        st["img"] = synthetic.gray(w, h, seed)
        st["params"] = _params(case, case["lam"])
        st["modes"] = tuple(int(str(m) in case["modes"]) for m in range(4))
        st["leaves"] = Rows(_most_leaves(case), 11, dtype=np.int32)
        st["levels"] = Rows(w * h, dtype=np.int32)
        if case["entry"] == "plan":
            st["plan"] = ctx.search_plan(w, h, st["params"])
    elif kind == "nodes":
        st["plane"] = torch.from_numpy(synthetic.gray(w, h, seed)).to(DEV)
        st["params"] = _params(case, None)
        n, ev = mb.C.c_size_t(), mb.C.c_uint64()
        mb.check(mb.lib().mars_search_nodes_device(
            ctx.handle, st["plane"].data_ptr(), w, h, mb.C.byref(st["params"]), None, 0,
            mb.C.byref(n), mb.C.byref(ev)))
        st["n"] = n.value
        st["out"] = torch.zeros(n.value, 80, dtype=torch.uint8, device=DEV)
    elif kind == "blocks":
        st["img"] = synthetic.gray(w, h, seed)
        st["params"] = mb.make_params(shift=case["shift"])
        st["rows"], st["cols"] = _origins(case, seed)
    elif kind in ("decode", "stable"):
        st["hdr"], st["leaves"], st["levels"] = _leaf_list(case, seed)
        if kind == "decode":
            st["plan"] = ctx.decode_plan(st["hdr"], st["leaves"])
            st["out"] = torch.zeros(h, w, dtype=torch.uint8, device=DEV)
    elif kind == "refine":
        img, hdr, leaves = _coded(ctx, case, seed)
        st["plan"] = ctx.refine_plan(hdr, leaves, img)
        st["s"], st["o"] = st["plan"].params()
        st["grads"] = [Rows(_most_leaves(case), dtype=np.float32) for _ in range(2)]
    else:
        st["rgb"] = _rgb(case, seed)
        n, half = w * h, ((w + 1) // 2) * ((h + 1) // 2)
        st["ycc"] = [torch.zeros(n, dtype=torch.uint8, device=DEV) for _ in range(3)]
        st["sub"] = [torch.zeros(half, dtype=torch.uint8, device=DEV) for _ in range(2)]
        st["up"] = [torch.zeros(n, dtype=torch.uint8, device=DEV) for _ in range(2)]
        st["back"] = [torch.zeros(n, dtype=torch.uint8, device=DEV) for _ in range(3)]
    torch.cuda.synchronize()  # the context's stream does not wait for torch's
    return st


# ---- one pass ----

def run(st):
    kind, case, ctx = st["kind"], st["case"], st["ctx"]
    if kind == "encode":
        if "plan" in st:
            _, leaves, levels, count = st["plan"].encode(st["img"], allowed_modes=st["modes"])
        else:
            _, leaves, levels, count = ctx.encode(st["img"], st["params"],
                                                  allowed_modes=st["modes"],
                                                  method=case["method"], rd_candidates=case["k"])
        return {"leaves": st["leaves"].put(leaves.view(np.int32).reshape(-1, 11)),
                "levels": st["levels"].put(levels), "count": [len(leaves), len(levels)],
                "evals": [count.search_evals, count.warmup_evals]}
    if kind == "nodes":
        n = mb.C.c_size_t()
        mb.check(mb.lib().mars_search_nodes_device(
            ctx.handle, st["plane"].data_ptr(), case["w"], case["h"], mb.C.byref(st["params"]),
            st["out"].data_ptr(), st["n"], mb.C.byref(n), None))
        return st["out"]
    if kind == "blocks":
        out, evals = ctx.search_blocks(st["img"], case["size"], case["shift"], st["params"],
                                       st["rows"], st["cols"])
        return {"records": out.view(np.int32).reshape(-1, 20), "rms": out["rms"],
                "evals": evals.view(np.int64)}
    if kind == "decode":
        st["plan"].run(case["iters"], st["out"].data_ptr())
        return st["out"]
    if kind == "stable":
        plane, used = ctx.decode_until_stable(st["hdr"], st["leaves"], 1, case["iters"],
                                              st["levels"])
        return {"plane": plane, "used": used}
    if kind == "refine":
        # The gradients' own convergence measure is not compared: it is the difference of two
        # nearly equal vectors.
        loss, steps, x = st["plan"].forward(st["s"], st["o"], want_x=True)
        gs, go, adjoint_steps, _ = st["plan"].backward()
        return {"loss": loss, "x": x, "grad_s": st["grads"][0].put(gs),
                "grad_o": st["grads"][1].put(go), "steps": [steps, adjoint_steps]}
    L, w, h, hw, hh = mb.lib(), case["w"], case["h"], (case["w"] + 1) // 2, (case["h"] + 1) // 2
    r, g, b = (t.data_ptr() for t in st["rgb"])
    y, cb, cr = (t.data_ptr() for t in st["ycc"])
    mb.check(L.mars_ycbcr_device(ctx.handle, r, g, b, w * h, y, cb, cr))
    for full, sub, up in zip((cb, cr), st["sub"], st["up"]):
        mb.check(L.mars_downsample_box_device(ctx.handle, full, w, h, sub.data_ptr()))
        mb.check(L.mars_upsample_nearest_device(ctx.handle, sub.data_ptr(), hw, hh,
                                                up.data_ptr(), w, h))
    mb.check(L.mars_rgb_from_ycbcr_device(ctx.handle, y, st["up"][0].data_ptr(),
                                          st["up"][1].data_ptr(), w * h,
                                          *(t.data_ptr() for t in st["back"])))
    mse = mb.C.c_double()
    mb.check(L.mars_mse_device(ctx.handle, g, st["back"][1].data_ptr(), w * h, mb.C.byref(mse)))
    return {"ycc": st["ycc"], "sub": st["sub"], "up": st["up"], "back": st["back"],
            "mse": mse.value}


# ---- what a pass cannot do without ----

def _level_fits(case, size):
    """Domain positions x 8 isometries of one block of `size`."""
    dy, dx = case["h"] - 2 * size, case["w"] - 2 * size
    if dy < 0 or dx < 0:
        return 0
    return (dy // case["shift"] + 1) * (dx // case["shift"] + 1) * 8


def work(case):
    kind, n = case["kind"], case["w"] * case["h"]
    if kind in ("encode", "nodes"):
        sizes = [s for s in (64, 32, 16, 8, 4) if case["min"] <= s <= case["max"]]
        nodes = {s: (case["w"] // s) * (case["h"] // s) for s in sizes}
        # A fit is size^2 multiply-adds.  The classified search's buckets hold a few percent of
        # the domains (72 classes of uneven sizes).
        share = 0.05 if case.get("method") == "fisher" else 1.0
        flops = sum(2.0 * s * s * nodes[s] * _level_fits(case, s) for s in sizes) * share
        out = 80 * sum(nodes.values()) if kind == "nodes" else 44 * (n // 64)
        return {"bytes": n + out, "flops": flops}
    if kind == "blocks":
        return {"bytes": n + 88 * case["n"],
                "flops": 2.0 * case["size"] ** 2 * case["n"] * _level_fits(case, case["size"])}
    if kind in ("decode", "stable"):
        # Per pixel and step: the four samples' sum, one multiply-add; planes beyond L2 would
        # cross HBM each step, which is not counted: leaves in, one plane out.
        return {"bytes": n + 16 * (n // 170), "flops": 6.0 * n * case["iters"]}
    if kind == "refine":
        # Target in, plane out; some thirty steps each way of six operations a pixel.
        return {"bytes": 5 * n, "flops": 2.0 * 30 * 6 * n}
    return {"bytes": 3 * n + 3 * n + 2 * n + n // 2 + n // 2 + 2 * n + 3 * n + 3 * n + 2 * n,
            "flops": 40.0 * n}


# ---- 64-bit results ----

def _isometries(r):
    """The eight orientations of (n, S, S) blocks."""
    turns = [torch.rot90(r, k, (1, 2)) for k in range(4)]
    return turns + [t.transpose(1, 2) for t in turns]


def _search_rms(img, rows, cols, size, shift, alfa_bits=4, beta_bits=7, max_alfa=1.0):
    """The smallest rms of the quantised affine fit over every domain and orientation."""
    f64 = dict(dtype=torch.float64, device=DEV)
    p = torch.as_tensor(img, **f64)
    h, w = p.shape
    if h < 2 * size or w < 2 * size or not len(rows):
        return torch.zeros(len(rows), **f64)
    half = (p[: h // 2 * 2: 2, : w // 2 * 2: 2] + p[1::2, : w // 2 * 2: 2][: h // 2]
            + p[: h // 2 * 2: 2, 1::2][:, : w // 2] + p[1::2, 1::2]) / 4.0
    dom = half.unfold(0, size, 1).unfold(1, size, 1)
    dy, dx = (h - 2 * size) // shift + 1, (w - 2 * size) // shift + 1
    dom = dom[:: shift // 2, :: shift // 2][:dy, :dx].reshape(-1, size * size)
    s1, s2, s0 = dom.sum(1), (dom * dom).sum(1), float(size * size)
    det = s0 * s2 - s1 * s1
    at_r = torch.as_tensor(rows.astype(np.int64), device=DEV)
    at_c = torch.as_tensor(cols.astype(np.int64), device=DEV)
    span = torch.arange(size, device=DEV)
    blk = p[(at_r[:, None, None] + span[:, None]), (at_c[:, None, None] + span)]
    best = torch.full((len(rows),), math.inf, **f64)
    chunk = max(1, int(2e8) // dom.shape[0])
    aq, bq = float(1 << alfa_bits), float((1 << beta_bits) - 1)
    for a in range(0, len(rows), chunk):
        r = blk[a: a + chunk]
        t0, t2 = r.sum((1, 2))[:, None], (r * r).sum((1, 2))[:, None]
        for turned in _isometries(r):
            t1 = turned.reshape(len(r), -1) @ dom.T
            alfa = torch.where(det != 0, (s0 * t1 - s1 * t0) / det, 0.0).clamp_(min=0.0)
            alfa = torch.floor(0.5 + alfa / max_alfa * aq).clamp_(0, aq - 1) / aq * max_alfa
            lift = alfa * 255.0
            width = (1.0 + alfa) * 255.0
            beta = (t0 - alfa * s1) / s0 + lift
            beta = torch.trunc(0.5 + beta / width * bq).clamp_(0, bq) / bq * width - lift
            sse = (t2 - 2 * alfa * t1 - 2 * beta * t0 + alfa * alfa * s2
                   + 2 * alfa * beta * s1 + s0 * beta * beta)
            best[a: a + chunk] = torch.minimum(best[a: a + chunk], sse.amin(1))
    return (best / s0).clamp(min=0.0).sqrt()


def _refine_exact(case, seed):
    """Fixed point, loss and adjoint gradients of the leaves' map, in 64 bits."""
    ctx = mb.Context(0)
    img, hdr, leaves = _coded(ctx, case, seed)
    plan = ctx.refine_plan(hdr, leaves, img)
    s32, o32 = plan.params()
    plan.close()
    ctx.close()
    w, h = case["w"], case["h"]
    owner = np.full((h, w), -1, np.int64)
    src = np.zeros((h, w), np.int64)
    for k, L in enumerate(leaves):
        S, r0, c0, iso = int(L["size"]), int(L["row"]), int(L["col"]), int(L["isometry"])
        i, j = np.meshgrid(np.arange(S), np.arange(S), indexing="ij")
        m = S - 1
        u, v = ((i, j), (j, m - i), (m - j, i), (m - i, m - j), (i, m - j), (m - i, j), (j, i),
                (m - j, m - i))[iso]
        owner[r0: r0 + S, c0: c0 + S] = k
        if L["qalfa"]:
            src[r0: r0 + S, c0: c0 + S] = (int(L["dom_row"]) + 2 * u) * w + int(L["dom_col"]) + 2 * v
    f64 = dict(dtype=torch.float64, device=DEV)
    own = torch.as_tensor(owner.ravel(), device=DEV)
    q = torch.as_tensor(src.ravel(), device=DEV)
    covered = own >= 0
    own = own.clamp(min=0)
    moves = torch.as_tensor((leaves["qalfa"] != 0).astype(np.float64), **f64)[own] * covered
    s, o = torch.as_tensor(s32, **f64)[own] * moves, torch.as_tensor(o32, **f64)[own] * covered
    t = torch.as_tensor(img.ravel(), **f64)
    # The last row and column never start a domain sample.
    taps = [(q + d).clamp(max=w * h - 1) for d in (0, 1, w, w + 1)]
    x = torch.full((w * h,), 128.0, **f64)
    for _ in range(600):
        d = sum(x[at] for at in taps) / 4.0
        x = (s * d + o).clamp(0.0, 255.0)
    d = sum(x[at] for at in taps) / 4.0 * moves
    raw = s * d + o
    gate = ((raw >= 0.0) & (raw <= 255.0) & covered).to(torch.float64)
    grad, lam = 2.0 * (x - t), torch.zeros_like(x)
    for _ in range(600):
        part = gate * s * lam / 4.0
        lam = grad.clone()
        for at in taps:
            lam.index_add_(0, at, part)
    gs = torch.zeros(_most_leaves(case), **f64).index_add_(0, own, gate * lam * d)
    go = torch.zeros(_most_leaves(case), **f64).index_add_(0, own, gate * lam)
    return {"loss": float(((x - t) ** 2).sum()), "x": x.reshape(h, w), "grad_s": gs, "grad_o": go,
            "steps": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "blocks" and _level_fits(case, case["size"]) * case["n"] <= 4e9:
        rows, cols = _origins(case, seed)
        img = synthetic.gray(case["w"], case["h"], seed)
        rms = _search_rms(img, rows, cols, case["size"], case["shift"])
        return {"records": None, "rms": rms, "evals": None}
    if kind == "refine":
        return _refine_exact(case, seed)
    if kind == "colour":
        return {"ycc": None, "sub": None, "up": None, "back": None, "mse": _mse(case, seed)}
    return None


def _mse(case, seed):
    """The green plane's error after BT.601 conversion, 2x2 averaging and replication."""
    w, h = case["w"], case["h"]
    r, g, b = (p.to(torch.float64) for p in _rgb(case, seed))

    def byte(v):
        return torch.floor(v + 0.5).clamp(0.0, 255.0)

    y = byte(0.299 * r + 0.587 * g + 0.114 * b)
    cb = byte(-0.168736 * r - 0.331264 * g + 0.5 * b + 128.0).reshape(1, 1, h, w)
    cr = byte(0.5 * r - 0.418688 * g - 0.081312 * b + 128.0).reshape(1, 1, h, w)

    def half(c):
        c = torch.nn.functional.pad(c, (0, w & 1, 0, h & 1), mode="replicate")[0, 0]
        s = c[0::2, 0::2] + c[0::2, 1::2] + c[1::2, 0::2] + c[1::2, 1::2]
        s = torch.floor((s + 2.0) / 4.0)
        return s.repeat_interleave(2, 0).repeat_interleave(2, 1)[:h, :w].reshape(-1)

    back = byte(y - 0.344136 * (half(cb) - 128.0) - 0.714136 * (half(cr) - 128.0))
    return float(((g - back) ** 2).sum() / g.numel())
