"""The work that users of this package have it do, as timed cases.

Every case goes through the package's public entry points on inputs of the
kind the workloads are quoted on: fractal terrain for the total viewshed,
ellipse phantoms for the Radon operator, motion-blurred textures for the
cepstrum and the local Radon transform, activations for the surrogate's
convolutions.  A program that uses the engine keeps one SkewEngine per grid
size and calls it again and again; that handle, the input and the output buffer
are what prepare() makes.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import skewengine_gb300 as ske
from skewengine_gb300 import surrogate, synthetic

ANGLES = 180
WINDOW = 64    # cepstrum and local Radon window
KEEP = 26      # spectrum bins the local Radon filter keeps
FLAGS = {"cepstrum": ske.FLAG_CEPSTRUM_F32, "localradon": ske.FLAG_LOCAL_RADON_F32, "radon": ske.FLAG_RADON_F32}
SIDE_OF = {"e1": 256, "e2": 128, "e3": 64, "b4": 32, "d3": 64, "d2": 128, "d1": 256}  # U-Net level -> image side


def listed():
    return [
        # The smallest call: one 64 x 64 patch, where launches and the status read-back count.
        {"name": "sdem_64", "op": "sdem", "dimx": 64, "dimy": 64, "accum": "reference", "host": False},
        # Total viewshed of a 500 x 500 DEM over all 180 angles.
        {"name": "sdem_500", "op": "sdem", "dimx": 500, "dimy": 500, "accum": "reference", "host": False},
        # The headline workload: a 2000 x 2000 DEM over all 180 angles.
        {"name": "sdem_2000", "op": "sdem", "dimx": 2000, "dimy": 2000, "accum": "reference", "host": False},
        # A ragged, non-square crop of a survey, NumPy in and out, compensated sums: the whole call with its copies.
        {"name": "sdem_613x1021_host", "op": "sdem", "dimx": 613, "dimy": 1021, "accum": "kahan", "host": True},
        # A catalogue of DEMs of uneven size in one call (sides as in the batched benchmark, up to half its largest).
        {"name": "sdem_batch_8", "op": "sdem_batch", "count": 8, "lo": 256, "hi": 1000, "pick": 4, "accum": "kahan"},
        # Filtered back-projection of a 512 x 512 phantom in the reference's precision.
        {"name": "radon_512", "op": "radon", "dimx": 512, "dimy": 512, "f32": False, "host": False},
        # The float32 operator on an odd, non-square image: rows that leave their width take the back-projection.
        {"name": "radon_f32_383x509", "op": "radon", "dimx": 383, "dimy": 509, "f32": True, "host": False},
        # Blur estimation of one 512 x 512 photograph in the reference's precision.
        {"name": "cepstrum_512", "op": "cepstrum", "dimx": 512, "dimy": 512, "f32": False, "host": False},
        # Blur estimation of a burst of photographs in the float32 mode, one call.
        {"name": "cepstrum_f32_16x512", "op": "cepstrum_batch", "count": 16, "side": 512},
        # Local Radon transform of every pixel of a 512 x 512 image in the reference's precision.
        {"name": "localradon_512", "op": "localradon", "dimx": 512, "dimy": 512, "f32": False, "host": False},
        # The same transform in the float32 mode.
        {"name": "localradon_f32_512", "op": "localradon", "dimx": 512, "dimy": 512, "f32": True, "host": False},
        # A surrogate layer in training: forward, data, weight and bias gradients at the training batch of 16 tiles.
        {"name": "conv_train_e2b", "op": "conv", "layer": "e2b", "tiles": 16, "train": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi):
    """One side spread over [lo, hi] by its logarithm; the other equal (half of the time) or within a factor of two."""
    a = _log_int(rng, lo, hi)
    b = a if rng.random() < 0.5 else max(lo, min(hi, int(a * rng.uniform(0.5, 2.0))))
    return a, b


def draw(rng):
    op = rng.choice(["sdem", "sdem", "sdem_batch", "radon", "cepstrum", "cepstrum_batch", "localradon", "conv"])
    if op == "sdem":
        dimx, dimy = _sides(rng, 48, 2000)
        return {"op": op, "dimx": dimx, "dimy": dimy, "accum": rng.choice(["reference", "kahan"]),
                "host": rng.random() < 0.3}
    if op == "sdem_batch":
        return {"op": op, "count": rng.randint(2, 16), "lo": 64, "hi": _log_int(rng, 128, 800),
                "pick": rng.randrange(1 << 20), "accum": rng.choice(["reference", "kahan"])}
    if op == "cepstrum_batch":
        side = _log_int(rng, 64, 512)
        return {"op": op, "count": rng.randint(2, max(2, min(48, 8 * 512 * 512 // (side * side)))), "side": side}
    if op == "conv":
        layer = rng.choice([name for name, _, _ in surrogate.LAYERS])
        return {"op": op, "layer": layer, "tiles": _log_int(rng, 1, 32), "train": rng.random() < 0.6}
    dimx, dimy = _sides(rng, 64, {"radon": 1024, "cepstrum": 512, "localradon": 512}[op])
    return {"op": op, "dimx": dimx, "dimy": dimy, "f32": rng.random() < 0.5, "host": rng.random() < 0.2}


# ---- inputs -----------------------------------------------------------------


def _image(case, seed):
    """The input grid of a single-grid case as the workload's generator makes it."""
    dimx, dimy = case["dimx"], case["dimy"]
    if case["op"] == "sdem":
        return synthetic.fractal_dem(dimx, seed, side_y=dimy)
    if case["op"] == "radon":
        return synthetic.ellipse_phantom(dimx, seed, side_y=dimy)
    return synthetic.blurred_texture(dimx, seed, side_y=dimy)[0]


def _batch_grids(case, seed):
    sizes = np.random.default_rng(case["pick"]).integers(case["lo"], case["hi"] + 1, size=case["count"])
    rough = np.random.default_rng(case["pick"] + 1).uniform(0.6, 0.9, size=case["count"])
    return [synthetic.fractal_dem(int(s), seed + 1000 * k, roughness=float(h))
            for k, (s, h) in enumerate(zip(sizes, rough))]


def _layer(case):
    cin, cout = next((i, o) for name, i, o in surrogate.LAYERS if name == case["layer"])
    return cin, cout, SIDE_OF[case["layer"][:2]]


def _conv_inputs(case, seed):
    """Activations after a ReLU, He-initialised weights, the gradient that comes back."""
    cin, cout, side = _layer(case)
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((case["tiles"], side, side, cin), generator=g, device="cuda").clamp_min_(0).to(torch.bfloat16)
    w = torch.zeros((cout, surrogate.kpad(cin)), device="cuda")
    w[:, : 9 * cin] = torch.randn((cout, 9 * cin), generator=g, device="cuda") * math.sqrt(2.0 / (9 * cin))
    b = 0.1 * torch.randn(cout, generator=g, device="cuda")
    dy = None
    if case["train"]:
        dy = (1e-2 * torch.randn((case["tiles"], side, side, cout), generator=g, device="cuda")).to(torch.bfloat16)
    return x, w, b, dy


def prepare(case, seed):
    op = case["op"]
    if op == "conv":
        x, w, b, dy = _conv_inputs(case, seed)
        if case["train"]:
            for t in (x, w, b):
                t.requires_grad_(True)
        else:
            w = w.to(torch.bfloat16)  # inference keeps the weights in the kernels' type
        return {"case": case, "x": x, "w": w, "b": b, "dy": dy}
    if op == "sdem_batch":
        grids = [torch.from_numpy(g).cuda() for g in _batch_grids(case, seed)]
        side = max(g.shape[0] for g in grids)
        return {"case": case, "grids": grids, "outs": [torch.empty_like(g) for g in grids],
                "engine": ske.SkewEngine(side, side)}
    if op == "cepstrum_batch":
        side = case["side"]
        imgs = np.stack([synthetic.blurred_texture(side, seed + 1000 * k)[0] for k in range(case["count"])])
        x = torch.from_numpy(imgs).cuda()
        return {"case": case, "grids": x, "outs": torch.empty_like(x), "engine": ske.SkewEngine(side, side)}
    img = _image(case, seed)
    if case["host"]:
        x, out = img, np.empty_like(img)
    else:
        x = torch.from_numpy(img).cuda()
        out = torch.empty_like(x)
    flags = FLAGS[op] if case.get("f32") else 0
    return {"case": case, "x": x, "out": out, "flags": flags, "engine": ske.SkewEngine(case["dimx"], case["dimy"])}


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "conv":
        x, w, b = state["x"], state["w"], state["b"]
        if not case["train"]:
            with torch.no_grad():
                return {"y": surrogate.conv3x3(x, w, b, True)}
        y = surrogate.conv_op(x, w, b, True)
        dx, dw, db = torch.autograd.grad(y, (x, w, b), state["dy"])
        return {"y": y.detach(), "dx": dx, "dw": dw, "db": db}
    if op == "sdem_batch":
        return ske.run_batch("sdem", state["grids"], outs=state["outs"], engine=state["engine"], accum=case["accum"])
    if op == "cepstrum_batch":
        return ske.run_batch("cepstrum", state["grids"], outs=state["outs"], engine=state["engine"],
                             flags=ske.FLAG_CEPSTRUM_F32)
    return state["engine"].run(op, state["x"], out=state["out"], accum=case.get("accum", "reference"),
                               flags=state["flags"])


# ---- work -------------------------------------------------------------------


def _row_lengths(dimx, dimy, a):
    s = _sector(dimx, dimy, a)
    return np.maximum(s["last"] - s["first"], 0).astype(np.float64)


def _grid_work(op, dimx, dimy):
    """Bytes and operations of one grid: input read once, output written once; per
    line-of-sight step a subtraction, a division and a comparison; per skewed
    cell two 64-point transforms of what the operator reads; per sector two
    transforms of its rows."""
    n = dimx * dimy
    flops = 0.0
    for a in range(ANGLES):
        if op == "sdem":
            row = _row_lengths(dimx, dimy, a)
            flops += 3.0 * float(np.sum(row * (row - 1)))
            continue
        s = _sector(dimx, dimy, a)
        if op == "radon":
            h2 = 1 << max(0, (s["H"] - 1).bit_length())
            flops += n + 2 * 5.0 * h2 * math.log2(max(h2, 2)) + 2 * n
        elif op == "cepstrum":
            flops += n * (2.5 * 64 * 6 + 2.5 * 32 * 5 + 32)
        else:
            flops += n * (2 * 2.5 * 64 * 6)
    return {"bytes": 8.0 * n, "flops": flops}


def work(case):
    op = case["op"]
    if op == "conv":
        cin, cout, side = _layer(case)
        pix = case["tiles"] * side * side
        one = 2.0 * 9 * cin * cout * pix
        if not case["train"]:
            return {"bytes": 2.0 * pix * (cin + cout) + 18.0 * cin * cout, "flops": one}
        return {"bytes": 4.0 * pix * (cin + cout) + 72.0 * cin * cout, "flops": 3 * one}
    if op == "sdem_batch":
        sizes = np.random.default_rng(case["pick"]).integers(case["lo"], case["hi"] + 1, size=case["count"])
        parts = [_grid_work("sdem", int(s), int(s)) for s in sizes]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if op == "cepstrum_batch":
        one = _grid_work("cepstrum", case["side"], case["side"])
        return {k: v * case["count"] for k, v in one.items()}
    return _grid_work(op, case["dimx"], case["dimy"])


# ---- the same values in 64 bits -----------------------------------------------


def _sector(dimx, dimy, a):
    """Orientation, shear and valid row ranges of one angle."""
    fa = int(math.degrees(math.atan2(dimy, dimx)))
    tr, mi = fa < a < 180 - fa, a > 90
    kind = (2 if mi else 1) if tr else (3 if mi else 0)
    na = (a, 90 - a, a - 90, 180 - a)[kind]
    di, do = (dimy, dimx) if tr else (dimx, dimy)
    slope = math.tan(math.radians(na))
    off = int(slope * (di - 1))
    H = do + off + 1 if na else do
    drift = slope * np.arange(di)
    target = drift.astype(np.int64)
    dl = max(dimx, dimy)
    r = np.arange(H + 2)
    last = np.where((r >= off) & (r < H), dl, 0)
    first = np.where((r >= do) & (r < H), dl, 0)
    for j, t in enumerate(target):
        for q in (t, t + 1):
            if j > last[q]:
                last[q] = j + 1
        for q in (t + do - 1, t + do):
            if q < H + 2 and j < first[q]:
                first[q] = j
    return {"kind": kind, "H": H, "di": di, "do": do, "dl": dl, "scale": 1 / math.cos(math.radians(na)),
            "target": target, "weight": drift - target, "first": first[:H], "last": last[:H]}


def _orient(x, kind):
    if kind == 0:
        return x
    if kind == 1:
        return x.t().flip(0, 1)
    if kind == 2:
        return x.t().flip(1)
    return x.flip(1)


def _unorient(y, kind):
    if kind == 0:
        return y
    if kind == 1:
        return y.flip(0, 1).t()
    if kind == 2:
        return y.flip(1).t()
    return y.flip(1)


def _viewshed_rows(S, length, povh):
    """Per observer of every row the ring areas of its closed visible runs, one direction; S (R, L), NaN past length."""
    R, L = S.shape
    out = torch.zeros_like(S)
    chunk = max(1, (64 << 20) // (L * L))
    d = torch.arange(L, device=S.device, dtype=torch.float64)
    dist = d[None, :] - d[:, None]
    ahead = dist > 0
    ring = torch.where(ahead, 2 * dist + 1, torch.zeros_like(dist))
    for r0 in range(0, R, chunk):
        z = S[r0:r0 + chunk]
        live = ahead[None] & (d[None, None, :] < length[r0:r0 + chunk, None, None])
        slope = (z[:, None, :] - (z + povh)[:, :, None]) / dist.clamp_min(1)[None]
        slope = torch.where(live, slope, torch.full_like(slope, -math.inf))
        top = torch.cummax(slope, 2).values
        before = torch.cat([torch.full_like(top[..., :1], -2000.0), top[..., :-1].clamp_min(-2000.0)], 2)
        seen = live & (slope > before)
        acc = torch.cumsum(torch.where(seen, ring[None], torch.zeros_like(slope)), 2)
        hidden = torch.where(live & ~seen, acc + 1, torch.zeros_like(acc))  # acc never falls: the last one is the largest
        out[r0:r0 + chunk] = hidden.amax(2)
    return out


def _local_radon_rows(V, scale, di):
    R, C = V.shape
    pre = torch.nn.functional.pad(torch.cumsum(V, 1), (1, 0))
    c = torch.arange(C, device=V.device)
    W = pre[:, (c + WINDOW // 2 + 1).clamp_max(C)] - pre[:, (c - WINDOW // 2).clamp_min(0)]
    m = torch.arange(WINDOW, device=V.device, dtype=torch.float64)
    gauss = torch.exp(-((m - WINDOW // 2) ** 2) / (2 * (WINDOW / 5 / scale) ** 2))
    k = torch.arange(KEEP, device=V.device, dtype=torch.float64)
    taper = torch.sin(k / (0.4 * WINDOW - 1) * math.pi / 2)
    X = torch.cos(2 * math.pi / WINDOW * torch.outer(m, k)) * gauss[:, None] * taper / 8
    ang = 2 * math.pi / WINDOW * torch.outer(k, m[:WINDOW // 2])
    P = torch.nn.functional.pad(W, (0, 0, WINDOW // 2, WINDOW // 2 - 1))
    out = torch.zeros_like(V)
    for r0 in range(0, R, 256):
        r1 = min(R, r0 + 256)
        win = P[r0:r1 + WINDOW - 1].unfold(0, WINDOW, 1)  # (rows, C, 64)
        Y = win.reshape(-1, WINDOW) @ X
        p = ((Y @ torch.cos(ang)) / 8) ** 2 + ((Y @ torch.sin(ang)) / 8) ** 2
        up = p[:, 5:] > p[:, 4:-1]
        at = up.to(torch.int8).argmax(1) + 4
        val = torch.where(up.any(1), p.gather(1, at[:, None])[:, 0], torch.zeros_like(p[:, 0]))
        out[r0:r1] = val.reshape(r1 - r0, C)
    return out


def _cepstrum_rows(V):
    R, C = V.shape
    P = torch.nn.functional.pad(V, (WINDOW // 2, WINDOW // 2 - 1))
    out = torch.zeros_like(V)
    for r0 in range(0, R, 256):
        win = P[r0:r0 + 256].unfold(1, WINDOW, 1)
        X = torch.fft.rfft(win, dim=2)[..., :WINDOW // 2] / 8
        lg = torch.log(X.real ** 2 + X.imag ** 2)
        s = (-torch.fft.rfft(lg, dim=2).real[..., :16] / math.sqrt(32)).clamp_min(0).reshape(-1, 16)
        up = s[:, 5:] > s[:, 4:-1]
        at = up.to(torch.int8).argmax(1) + 5
        k = torch.arange(16, device=V.device)
        pick = (k == at[:, None] - 1) | (k > at[:, None])
        val = torch.where(up.any(1), (s * pick).amax(1), torch.zeros_like(s[:, 0]))
        out[r0:r0 + 256] = 10000 * val.reshape(-1, C)
    return out


def _grid64(op, img, povh=float(ske.DEFAULT_POVH)):
    dimy, dimx = img.shape
    x = torch.from_numpy(img).cuda().double()
    total = torch.zeros_like(x)
    acc = {}
    for a in range(ANGLES):
        s = _sector(dimx, dimy, a)
        H, di, do, dl = s["H"], s["di"], s["do"], s["dl"]
        src = _orient(x, s["kind"])
        t = torch.from_numpy(s["target"]).cuda()
        w = torch.from_numpy(s["weight"]).cuda()
        rows = torch.arange(do, device="cuda")[:, None] + t[None, :]
        cell = rows * di + torch.arange(di, device="cuda")[None, :]
        flat = torch.zeros((H + dl // di + 2) * di + dl, dtype=torch.float64, device="cuda")
        flat.index_add_(0, cell.reshape(-1), ((1 - w) * src).reshape(-1))
        flat.index_add_(0, (cell + di).reshape(-1), (w * src).reshape(-1))
        f, l = torch.from_numpy(s["first"]).cuda(), torch.from_numpy(s["last"]).cuda()
        c = torch.arange(dl, device="cuda")
        at = torch.arange(H, device="cuda")[:, None] * di + c[None, :]
        ok = (c[None, :] >= f[:, None]) & (c[None, :] < l[:, None])
        V = torch.where(ok, flat[at], torch.zeros((), dtype=torch.float64, device="cuda"))
        if op == "radon":
            h2 = 1 << max(0, (H - 1).bit_length())
            ramp = torch.arange(h2, device="cuda", dtype=torch.float64) / H
            ramp[H // 2 + 1:] = 0
            q = torch.fft.ifft(torch.fft.fft(V.sum(1), n=h2) * ramp).real[:H]
            res = torch.where(ok, q[:, None], torch.zeros_like(V))
            out = torch.zeros_like(flat).index_add_(0, at.reshape(-1), res.reshape(-1))
        else:
            if op == "sdem":
                n = (l - f).clamp_min(0)
                L = int(n.max())
                k = torch.arange(L, device="cuda")
                cells = (f[:, None] + k[None, :]).clamp_max(dl - 1)
                inside = k[None, :] < n[:, None]
                row = torch.where(inside, V.gather(1, cells), torch.full((H, L), math.nan, device="cuda",
                                                                       dtype=torch.float64))
                back = (n[:, None] - 1 - k[None, :]).clamp_min(0)
                cv = _viewshed_rows(row, n, povh) + _viewshed_rows(row.gather(1, back), n, povh).gather(1, back)
                at = (torch.arange(H, device="cuda")[:, None] * di + cells)
                res, ok = cv * s["scale"] ** 2, inside
            elif op == "localradon":
                res = _local_radon_rows(V, s["scale"], di)
            else:
                res = _cepstrum_rows(V)
            # A cell that several rows cover keeps the last row's value.
            owner = torch.full(flat.shape, -1, dtype=torch.int64, device="cuda")
            rid = torch.arange(H, device="cuda")[:, None].expand_as(at)
            owner.scatter_reduce_(0, at[ok], rid[ok], "amax")
            mine = ok & (owner[at] == rid)
            out = torch.zeros_like(flat)
            out[at[mine]] = res[mine]
        lo, hi = out[cell], out[cell + di]
        have = acc.get(s["kind"])
        if op == "cepstrum":
            v = torch.maximum(lo, hi)
            v = v if have is None else torch.maximum(v, have)
            acc[s["kind"]] = a + 1000 * torch.floor(v / 1000)
        else:
            v = (1 - w) * lo + w * hi
            acc[s["kind"]] = v if have is None else have + v
    for kind in sorted(acc):
        y = _unorient(acc[kind], kind)
        total = torch.maximum(total, y) if op == "cepstrum" else total + y
    return total


def _conv64(case, seed):
    x, w, b, dy = _conv_inputs(case, seed)
    cin, cout, _ = _layer(case)
    w4 = w.to(torch.bfloat16).double()[:, : 9 * cin].reshape(cout, 3, 3, cin).permute(0, 3, 1, 2).contiguous()
    x4 = x.double().permute(0, 3, 1, 2).contiguous()
    taps = torch.nn.functional.pad(x4, (1, 1, 1, 1))
    h = x4.shape[2]
    views = [(i, j, taps[:, :, i:i + h, j:j + h]) for i in range(3) for j in range(3)]
    y = b.double()[None, :, None, None] + sum(torch.einsum("nihw,oi->nohw", v, w4[:, :, i, j]) for i, j, v in views)
    y = y.clamp_min(0)
    got = {"y": y.permute(0, 2, 3, 1)}
    if not case["train"]:
        return got
    g = dy.double().permute(0, 3, 1, 2) * (y > 0)
    back = torch.nn.functional.pad(g, (1, 1, 1, 1))
    dx = sum(torch.einsum("nohw,oi->nihw", back[:, :, 2 - i:2 - i + h, 2 - j:2 - j + h], w4[:, :, i, j])
             for i in range(3) for j in range(3))
    dw = torch.zeros(w.shape, dtype=torch.float64, device="cuda")
    dw[:, : 9 * cin] = torch.stack([torch.einsum("nohw,nihw->oi", g, v) for _, _, v in views], 1).reshape(cout, 9 * cin)
    got.update(dx=dx.permute(0, 2, 3, 1), dw=dw, db=g.sum((0, 2, 3)))
    return got


def exact(case, seed):
    """The case's values in 64 bits; None where that takes too long (a viewshed of more than 640 cells a side, whose
    every pair of cells of every row would be formed)."""
    op = case["op"]
    if op == "conv":
        return _conv64(case, seed)
    if op == "cepstrum_batch":
        if case["count"] * case["side"] ** 2 > 16 * 512 * 512:
            return None
        return torch.stack([_grid64("cepstrum", synthetic.blurred_texture(case["side"], seed + 1000 * k)[0])
                            for k in range(case["count"])])
    if op == "sdem_batch":
        grids = _batch_grids(case, seed)
        if sum(float(g.shape[0]) ** 3 for g in grids) > 640.0 ** 3:
            return None
        return [_grid64("sdem", g) for g in grids]
    if op == "sdem" and max(case["dimx"], case["dimy"]) > 640:
        return None
    return _grid64(op, _image(case, seed))
