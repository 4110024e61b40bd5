"""Performance cases of the BM3D library: the calls a user's program makes.

Every case denoises planes (or trains the pilot that stands in for the basic
estimate) through the package's public calls, on inputs made on the GPU from a
seed: piecewise-smooth planes in [0, 1] (discs and rectangles with linear
gradients, one sinusoidal texture) plus Gaussian noise, as the benchmark and
the tests use them.

* ``listed()``  the fixed cases;
* ``draw(rng)`` one more case of the same ranges;
* ``prepare(case, seed)`` inputs, outputs and handles; ``run(state)`` one pass;
* ``work(case)`` the bytes and floating-point operations of a pass;
* ``exact(case, seed)`` the result in float64 by plain torch.
"""
import math

import numpy as np
import torch

import isp_mw_b200 as isp

# Luma / chroma norms of the opponent colour transform: the parameter sigma is
# the noise level divided by these (single planes use the luma norm).
NORM = (1.0 / math.sqrt(3.0), math.sqrt(0.5), math.sqrt(0.375))

PILOT_C = 48  # channels of the pilot network


def listed():
    return [
        # a thumbnail: the whole filter on one tiny plane, where launches and latency count
        dict(name="luma_64", kind="full", profile="fast", height=64, width=64, pad=0, sigma=25.0),
        # one 512 x 512 plane, the usual test image
        dict(name="luma_512", kind="full", profile="fast", height=512, width=512, pad=0, sigma=25.0),
        # one HD luma plane of a video, one call per frame
        dict(name="luma_1080", kind="full", profile="fast", height=1080, width=1920, pad=0, sigma=25.0),
        # a shot of four HD planes at the benchmark's noise levels, one graph replay
        dict(name="sweep_1080", kind="batch", profile="fast", sizes="1080x1920*4",
             sigmas="5,10,25,50"),
        # a folder of photos of any size and noise level in one batch
        dict(name="ragged_16", kind="batch", profile="fast",
             sizes="257x1999,1033x610,300x301,1471x877,640x480,1999x1333,263x517,768x1024,"
                   "911x1203,1080x1920,333x2048,1777x259,1200x800,480x720,1025x1023,599x1501",
             sigmas="31,7,50,12,25,18,40,9,22,15,5,36,28,45,10,20"),
        # one 4K YUV 4:4:4 frame, chroma filtered with luma's groups
        dict(name="yuv_2160", kind="yuv", profile="fast", height=2160, width=3840, pad=0, sigma=15.0),
        # one 8-bit RGB photo through the integer entry
        dict(name="rgb8_720", kind="rgb", profile="fast", height=720, width=1280, bits=8, sigma=20.0),
        # the quality profiles, on odd sizes inside a larger buffer: groups of 32, wide search
        dict(name="np_odd", kind="full", profile="np", height=717, width=1283, pad=29, sigma=25.0),
        dict(name="vn_540", kind="full", profile="vn", height=540, width=960, pad=0, sigma=40.0),
        # double-precision planes, stage by stage, as a quality reference
        dict(name="f64_lc_480", kind="stages64", profile="lc", height=480, width=640, pad=3, sigma=15.0),
        # an HD plane with the learned pilot in place of the basic stage
        dict(name="pilot_1080", kind="pilot", profile="fast", height=1080, width=1920, pad=0, sigma=25.0),
        # one training step of the pilot on a batch of crops
        dict(name="train_32", kind="train", count=32, height=128, width=128, sigma=25.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["full", "full", "full", "batch", "yuv", "rgb", "stages64", "pilot", "train"])
    sigma = round(rng.uniform(5.0, 50.0), 1)
    if kind == "full":
        profile = rng.choice(["fast", "fast", "lc", "np", "high", "vn"])
        top = {"fast": 2160, "lc": 1440, "np": 960, "high": 640, "vn": 640}[profile]
        return dict(kind=kind, profile=profile, height=_log_int(rng, 48, top),
                    width=_log_int(rng, 48, top), pad=rng.choice([0, 0, 1, 7, 64]), sigma=sigma)
    if kind == "batch":
        n = rng.randint(2, 12)
        sizes = ["%dx%d" % (_log_int(rng, 64, 1400), _log_int(rng, 64, 1400)) for _ in range(n)]
        return dict(kind=kind, profile=rng.choice(["fast", "fast", "lc"]), sizes=",".join(sizes),
                    sigmas=",".join("%.1f" % rng.uniform(5.0, 50.0) for _ in range(n)))
    if kind == "yuv":
        return dict(kind=kind, profile=rng.choice(["fast", "lc"]), height=_log_int(rng, 64, 1440),
                    width=_log_int(rng, 64, 1440), pad=rng.choice([0, 0, 5]), sigma=sigma)
    if kind == "rgb":
        return dict(kind=kind, profile="fast", height=_log_int(rng, 64, 1440),
                    width=_log_int(rng, 64, 1440), bits=rng.choice([8, 10, 16]), sigma=sigma)
    if kind == "stages64":
        return dict(kind=kind, profile=rng.choice(["fast", "lc"]), height=_log_int(rng, 48, 500),
                    width=_log_int(rng, 48, 640), pad=rng.choice([0, 3]), sigma=sigma)
    if kind == "pilot":
        return dict(kind=kind, profile="fast", height=_log_int(rng, 64, 1200),
                    width=_log_int(rng, 64, 1900), pad=rng.choice([0, 3]), sigma=sigma)
    return dict(kind=kind, count=_log_int(rng, 1, 32), height=rng.randint(24, 128),
                width=rng.randint(24, 128), sigma=sigma)


# ---- inputs -----------------------------------------------------------------

def _clean(height, width, rng, dev="cuda"):
    """Piecewise-smooth plane in [0, 1]: 40 shapes with linear gradients and a texture."""
    img = torch.full((height, width), float(rng.uniform(0.2, 0.8)), device=dev)
    yy = torch.arange(height, device=dev, dtype=torch.float32)[:, None]
    xx = torch.arange(width, device=dev, dtype=torch.float32)[None, :]
    scale = float(max(height, width))
    for _ in range(40):
        disc = rng.random() < 0.5
        r = rng.uniform(0.05, 0.35) * scale / 2
        cy, cx = rng.uniform(0, height), rng.uniform(0, width)
        hh, hw = (r, r) if disc else (r * rng.uniform(0.3, 1.0), r * rng.uniform(0.3, 1.0))
        base = rng.uniform(0.0, 1.0)
        gy, gx = rng.uniform(-0.6, 0.6, 2) / scale
        y0, y1 = max(0, int(cy - hh)), min(height, int(cy + hh) + 1)
        x0, x1 = max(0, int(cx - hw)), min(width, int(cx + hw) + 1)
        if y1 <= y0 or x1 <= x0:
            continue
        y, x = yy[y0:y1] - cy, xx[:, x0:x1] - cx
        val = base + gy * y + gx * x
        part = img[y0:y1, x0:x1]
        if disc:
            part.copy_(torch.where(y * y + x * x <= r * r, val, part))
        else:
            part.copy_(val)
    f, theta = rng.uniform(0.02, 0.2), rng.uniform(0, math.pi)
    phase = rng.uniform(0, 2 * math.pi)
    img += 0.1 * torch.sin(2 * math.pi * f * (xx * math.cos(theta) + yy * math.sin(theta)) + phase)
    return img.clamp_(0.0, 1.0)


def _noisy(height, width, sigma, seed, index=0, pad=0):
    """One noisy plane, a view of `width` columns in rows of width + pad."""
    rng = np.random.default_rng([int(seed), index])
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 1009 + index)
    clean = _clean(height, width, rng)
    plane = torch.zeros(height, width + pad, device="cuda")[:, :width]
    plane.copy_(clean + torch.randn(height, width, device="cuda", generator=gen) * (sigma / 255.0))
    return plane


def _like(plane):
    """An output plane with the row pitch of `plane`."""
    return torch.zeros(plane.shape[0], plane.stride(0), dtype=plane.dtype,
                       device=plane.device)[:, :plane.shape[1]]


def _params(profile, sigmas):
    sp = [s / n for s, n in zip(sigmas, NORM)]
    return (isp.stage_params_default(profile, False, sp),
            isp.stage_params_default(profile, True, sp))


def _batch_list(case):
    sizes = []
    for part in case["sizes"].split(","):
        size, _, times = part.partition("*")
        h, w = (int(v) for v in size.split("x"))
        sizes += [(h, w)] * int(times or 1)
    return sizes, [float(v) for v in case["sigmas"].split(",")]


def _yuv_sigmas(case):  # chroma of a YUV frame carries less noise than luma
    s = case["sigma"]
    return [s, s * 2 / 3, s * 2 / 3]


def _pilot_params(seed):
    """He-normal weights, the last layer's a tenth (the network starts near the identity)."""
    rng = np.random.default_rng([int(seed), 77])
    parts = []
    for cin, cout in _pilot_layers():
        scale = math.sqrt(2.0 / (9 * cin)) * (0.1 if cout == 1 else 1.0)
        parts.append(rng.standard_normal(cout * cin * 9) * scale)
        parts.append(np.zeros(cout))
    return np.concatenate(parts).astype(np.float32)


def _pilot_layers():
    return [(2, PILOT_C)] + [(PILOT_C, PILOT_C)] * 6 + [(PILOT_C, 1)]


def prepare(case, seed):
    ctx = isp.default_context()
    kind = case["kind"]
    st = dict(kind=kind, ctx=ctx)
    if kind == "train":
        n, h, w = case["count"], case["height"], case["width"]
        rng = np.random.default_rng([int(seed), 3])
        sig = torch.tensor(rng.uniform(5.0, 50.0, n) / 255.0, dtype=torch.float32, device="cuda")
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        clean = torch.stack([_clean(h, w, rng) for _ in range(n)])
        st["noisy"] = clean + torch.randn(n, h, w, device="cuda", generator=gen) * sig.view(-1, 1, 1)
        st["target"], st["sigma"] = clean, sig
        st["pilot"] = isp.Pilot(ctx, seed=0)
        st["pilot"].set_params(_pilot_params(seed))
        return st
    if kind == "batch":
        sizes, sigmas = _batch_list(case)
        src = [_noisy(h, w, s, seed, i) for i, ((h, w), s) in enumerate(zip(sizes, sigmas))]
        dst = [torch.zeros_like(p) for p in src]
        pairs = [_params(case["profile"], [s] * 3) for s in sigmas]
        st["dst"], st["src"] = dst, src
        st["batch"] = isp.Batch(ctx, [p[0] for p in pairs], [p[1] for p in pairs], dst, src)
        return st
    h, w = case["height"], case["width"]
    if kind == "yuv":
        sig = _yuv_sigmas(case)
        st["src"] = [_noisy(h, w, s, seed, c, case["pad"]) for c, s in enumerate(sig)]
        st["dst"] = [_like(p) for p in st["src"]]
        st["basic"], st["final"] = _params(case["profile"], sig)
        return st
    if kind == "rgb":
        top = (1 << case["bits"]) - 1
        planes = [_noisy(h, w, case["sigma"], seed, c) for c in range(3)]
        st["src"] = [(p * top).round_().clamp_(0, top).to(torch.int32) for p in planes]
        st["dst"] = [torch.zeros_like(p) for p in st["src"]]
        st["top"] = top
        # on an RGB frame the parameter is the noise level itself: the library
        # applies the colour transform's norms
        sp = [case["sigma"]] * 3
        st["basic"] = isp.stage_params_default(case["profile"], False, sp)
        st["final"] = isp.stage_params_default(case["profile"], True, sp)
        return st
    src = _noisy(h, w, case["sigma"], seed, 0, case["pad"])
    if kind == "stages64":
        wide = torch.zeros(h, w + case["pad"], dtype=torch.float64, device="cuda")[:, :w]
        wide.copy_(src)
        src = wide
        st["estimate"] = _like(src)
    st["src"], st["dst"] = src, _like(src)
    st["basic"], st["final"] = _params(case["profile"], [case["sigma"]] * 3)
    if kind == "pilot":
        st["pilot"] = isp.Pilot(ctx, seed=0)
        st["pilot"].set_params(_pilot_params(seed))
    return st


def run(st):
    kind, ctx = st["kind"], st["ctx"]
    if kind == "full":
        ctx.full(st["basic"], st["final"], st["dst"], st["src"])
        return st["dst"]
    if kind == "batch":
        st["batch"].run()
        return st["dst"]
    if kind == "yuv":
        ctx.full3(st["basic"], st["final"], st["dst"], st["src"])
        return st["dst"]
    if kind == "rgb":
        ctx.frame(st["basic"], st["final"], st["dst"], st["src"], 0, st["top"])
        return st["dst"]
    if kind == "stages64":
        ctx.stage(st["basic"], False, st["estimate"], st["src"])
        ctx.stage(st["final"], True, st["dst"], st["src"], st["estimate"])
        return [st["estimate"], st["dst"]]
    if kind == "pilot":
        st["pilot"].full(st["final"], st["dst"], st["src"])
        return st["dst"]
    loss = st["pilot"].train_step(st["noisy"], st["target"], st["sigma"], 1e-4)
    return {"loss": loss, "grad": st["pilot"].grad()}


# ---- work -------------------------------------------------------------------

def _stage_flops(profile, wiener, h, w, planes=1):
    """Matching (3 operations per pixel pair), separable fast transforms (2.5
    log2 L per sample and axis), shrinkage and aggregation; full groups."""
    p = isp.stage_params_default(profile, wiener, (10.0, 10.0, 10.0))
    bs, gs = p.block_size, p.group_size
    if h < bs or w < bs:
        return 0
    refs = math.ceil((h - bs) / p.block_step + 1) * math.ceil((w - bs) / p.block_step + 1)
    cand = min(2 * p.bm_range + 1, h - bs + 1) * min(2 * p.bm_range + 1, w - bs + 1)
    axis = 2.5 * (2 * math.log2(bs) + math.log2(gs))
    group = gs * bs * bs * (axis * (3 if wiener else 2) + (5 if wiener else 1) + 3)
    return refs * (3 * bs * bs * cand + planes * group)


def _both(profile, h, w, planes=1):
    return _stage_flops(profile, False, h, w, planes) + _stage_flops(profile, True, h, w, planes)


def work(case):
    kind = case["kind"]
    if kind == "train":
        px = case["count"] * case["height"] * case["width"]
        macs = sum(9 * a * b for a, b in _pilot_layers())
        params = macs + sum(b for _, b in _pilot_layers())
        # forward, data gradient and weight gradient (no data gradient at layer 1)
        return {"bytes": 8 * px + 4 * params * 7,
                "flops": px * (6 * macs - 2 * 9 * 2 * PILOT_C)}
    if kind == "batch":
        sizes, _ = _batch_list(case)
        return {"bytes": sum(8 * h * w for h, w in sizes),
                "flops": sum(_both(case["profile"], h, w) for h, w in sizes)}
    h, w = case["height"], case["width"]
    px = h * w
    if kind in ("yuv", "rgb"):
        return {"bytes": 24 * px, "flops": _both(case["profile"], h, w, 3)}
    if kind == "stages64":
        return {"bytes": 24 * px, "flops": _both(case["profile"], h, w)}
    if kind == "pilot":
        macs = sum(9 * a * b for a, b in _pilot_layers())
        return {"bytes": 8 * px, "flops": 2 * px * macs + _stage_flops(case["profile"], True, h, w)}
    return {"bytes": 8 * px, "flops": _both(case["profile"], h, w)}


# ---- exact results ----------------------------------------------------------

def _dct(n, dev):
    k = torch.arange(n, dtype=torch.float64, device=dev)
    m = torch.cos(math.pi * (2 * k[None, :] + 1) * k[:, None] / (2 * n)) * math.sqrt(2.0 / n)
    m[0] /= math.sqrt(2.0)
    return m


def _positions(last, step):
    pos = list(range(0, last + 1, step))
    return pos if pos[-1] == last else pos + [last]


def _stage_exact(p, wiener, src, ref, match):
    """One stage in float64: planes src filtered (guided by ref when Wiener)
    with the groups matched on `match`."""
    dev, (h, w) = match.device, match.shape
    bs, gs, rng = p.block_size, p.group_size, p.bm_range
    bottom, right = h - bs, w - bs
    th = p.thMSE * NORM[0] * bs * bs / 255.0 ** 2
    ys = torch.tensor(_positions(bottom, p.block_step), device=dev)
    xs = torch.tensor(_positions(right, p.block_step), device=dev)
    refs = torch.cartesian_prod(ys, xs)
    off = torch.arange(-rng, rng + 1, device=dev)
    offs = torch.cartesian_prod(off, off)
    blocks = match.unfold(0, bs, 1).unfold(1, bs, 1)  # every block, a view
    side = torch.arange(bs, device=dev)
    num = [torch.zeros(h * w, dtype=torch.float64, device=dev) for _ in src]
    den = [torch.zeros(h * w, dtype=torch.float64, device=dev) for _ in src]
    d2 = _dct(bs, dev)
    chunk = max(1, (1 << 27) // (offs.shape[0] * bs * bs * 8))
    for at in range(0, refs.shape[0], chunk):
        r = refs[at:at + chunk]
        # the window's blocks in raster order, then block (0, 0) once more
        pos = torch.cat([r[:, None, :] + offs, torch.zeros_like(r)[:, None, :]], 1)
        inside = ((pos >= 0).all(-1) & (pos[..., 0] <= bottom) & (pos[..., 1] <= right))
        inside[:, :-1] &= (offs != 0).any(-1)
        pos = torch.where(inside[..., None], pos, torch.zeros_like(pos))
        dist = (blocks[pos[..., 0], pos[..., 1]] -
                blocks[r[:, 0], r[:, 1]][:, None]).square().sum((-1, -2))
        ok = inside & (dist <= th) & (dist != 0)
        dist = torch.where(ok, dist, torch.inf)
        order = torch.sort(dist, dim=1, stable=True).indices[:, :gs - 1]
        count = 1 + ok.sum(1).clamp(max=gs - 1)
        member = torch.cat([r[:, None, :], torch.gather(pos, 1, order[..., None].expand(-1, -1, 2))], 1)
        for n in torch.unique(count).tolist():
            g = member[count == n][:, :n]
            pix = (g[..., 0, None, None] + side[:, None]) * w + g[..., 1, None, None] + side
            dz = _dct(n, dev)
            # the library's unnormalised coefficients carry sqrt(2) per zero index
            zero = [torch.tensor([2.0] + [1.0] * (m - 1), dtype=torch.float64, device=dev)
                    for m in (n, bs, bs)]
            zeros = zero[0][:, None, None] * zero[1][:, None] * zero[2]

            def fwd(plane):
                return torch.einsum("ka,iy,jx,rayx->rkij", dz, d2, d2, plane.reshape(-1)[pix])

            for c, plane in enumerate(src):
                sigma = p.sigma[c] / 255.0 * NORM[c]
                coef = fwd(plane)
                if wiener:
                    e = fwd(ref[c]).square() * zeros
                    wgt = e / (e + sigma * sigma)
                    coef = coef * wgt
                    total = wgt.square().sum((1, 2, 3))
                    weight = torch.where(total > 0, 1 / total, torch.ones_like(total))
                else:
                    keep = coef.abs() > sigma * p.lambda_
                    coef = coef * keep
                    weight = 1.0 / keep.sum((1, 2, 3)).clamp(min=1).double()
                out = torch.einsum("ka,iy,jx,rkij->rayx", dz, d2, d2, coef)
                wt = weight[:, None, None, None].expand_as(out)
                num[c].index_add_(0, pix.reshape(-1), (out * wt).reshape(-1))
                den[c].index_add_(0, pix.reshape(-1), wt.reshape(-1))
    return [(a / b).reshape(h, w) for a, b in zip(num, den)]


def _pilot_exact(params, noisy, sigma):
    """The pilot network in float64 (planes [n, h, w], sigma [n])."""
    x = torch.stack([noisy, sigma.view(-1, 1, 1).expand_as(noisy)], 1)
    at = 0
    for i, (cin, cout) in enumerate(_pilot_layers()):
        weight = params[at:at + cout * cin * 9].view(cout, cin, 3, 3)
        at += cout * cin * 9
        x = torch.nn.functional.conv2d(x, weight, params[at:at + cout], padding=1)
        at += cout
        x = torch.relu(x) if i < 7 else x
    return noisy + x[:, 0]


def _costly(case):
    """Whether the float64 evaluation would take long."""
    flops = work(case)["flops"]
    return flops > (2e12 if case["kind"] in ("pilot", "train") else 1e11)


def exact(case, seed):
    kind = case["kind"]
    if kind == "rgb" or _costly(case):
        return None
    st = prepare(case, seed)
    if kind == "train":
        params = torch.from_numpy(_pilot_params(seed)).cuda().double().requires_grad_(True)
        sigma = st["sigma"].double()
        err = (_pilot_exact(params, st["noisy"].double(), sigma) - st["target"].double()).square()
        loss = (err * ((25.0 / 255.0) / sigma).square().view(-1, 1, 1)).mean()
        loss.backward()
        return {"loss": float(loss), "grad": params.grad.cpu().numpy()}
    if kind == "batch":
        _, sigmas = _batch_list(case)
        out = []
        for plane, s in zip(st["src"], sigmas):
            b, f = _params(case["profile"], [s] * 3)
            x = plane.double()
            est = _stage_exact(b, False, [x], None, x)
            out.append(_stage_exact(f, True, [x], est, est[0])[0])
        return out
    planes = [p.double() for p in (st["src"] if kind == "yuv" else [st["src"]])]
    if kind == "pilot":
        params = torch.from_numpy(_pilot_params(seed)).cuda().double()
        sigma = torch.tensor([case["sigma"] / 255.0], dtype=torch.float64, device="cuda")
        est = [_pilot_exact(params, planes[0][None], sigma)[0]]
    else:
        est = _stage_exact(st["basic"], False, planes, None, planes[0])
    out = _stage_exact(st["final"], True, planes, est, est[0])
    if kind == "stages64":
        return [est[0], out[0]]
    return out if kind == "yuv" else out[0]
