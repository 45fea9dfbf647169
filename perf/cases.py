"""The workloads whose speed is measured: what a user of rc_gb300 has it do, through the public entry points.

Every case is an observation of an antenna array (layout, hours, channels) and one operation of an imaging run on it. Inputs are made from the seed alone, on
the GPU, with torch and numpy. `exact` restates each operation in 64 bits with torch."""
import ctypes
import math

import numpy as np
import torch

OVER = 8
LIGHT = 299792458.0
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # one time sample of a 96-station array gridded at once, plan and all, by a caller that may not allocate: the smallest call, all latency
        dict(name="snapshot", kind="oneshot", layout="core", radius=2000.0, ants=96, times=1, chans=1, grid=1024, planes=4, s_min=8, s_max=24, odd=False),
        # the 64-antenna 3 km array without a w-term: one 8 x 8 kernel, grid and degrid
        dict(name="no_w_pair", kind="pair", layout="disk", radius=1500.0, ants=64, times=256, chans=1, grid=2048, planes=1, s_min=8, s_max=8, odd=False),
        # w-projection of a 256-antenna observation: the gridding half of a major cycle
        dict(name="wproj_grid", kind="grid", layout="core", radius=10000.0, ants=256, times=128, chans=1, grid=4096, planes=32, s_min=8, s_max=64, odd=False),
        # and its other half, the model's visibilities
        dict(name="wproj_degrid", kind="degrid", layout="core", radius=10000.0, ants=256, times=128, chans=1, grid=4096, planes=32, s_min=8, s_max=64, odd=False),
        # one gradient of least-squares imaging: image to visibilities and back through autograd
        dict(name="lsq_gradient", kind="lsq", layout="disk", radius=1500.0, ants=64, times=512, chans=1, grid=2048, planes=16, s_min=8, s_max=64, odd=False),
        # channels and facets with grids of three sizes in one batched launch per direction
        dict(name="batch_pair", kind="batch", layout="disk", radius=1500.0, ants=64, times=48, chans=12, grid=1024, planes=24, s_min=8, s_max=96, odd=False),
        # a 40 km array with large grids and supports up to 128, grid and degrid
        dict(name="wide_pair", kind="pair", layout="core", radius=40000.0, ants=512, times=16, chans=2, grid=8192, planes=64, s_min=8, s_max=128, odd=False),
        # the double-precision pair, for a user who wants complex128
        dict(name="fp64_pair", kind="pair64", layout="disk", radius=1500.0, ants=64, times=192, chans=1, grid=2048, planes=16, s_min=8, s_max=64, odd=False),
        # the drop-in kernels on host buffers, w-bin by w-bin, as the reference's host program calls them
        dict(name="drop_in", kind="abi", layout="core", radius=5000.0, ants=128, times=24, chans=1, grid=1024, planes=4, s_min=16, s_max=32, odd=False),
        # the transforms either side of the gridder: model image to grid, grid to dirty image
        dict(name="image_transforms", kind="image", grid=4096),
        # the CLEAN minor loop of a major cycle
        dict(name="clean", kind="clean", layout="core", radius=10000.0, ants=128, times=64, grid=2048, iterations=200),
        # what a new observation costs before the first grid: w-kernels and the plan
        dict(name="setup", kind="setup", layout="core", radius=10000.0, ants=192, times=64, chans=1, grid=4096, planes=32, s_min=8, s_max=64, odd=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _edge(rng, lo, hi):
    """An image edge: mostly a size that transforms like, sometimes any even one."""
    if rng.random() < 0.3:
        return 2 * _log(rng, lo // 2, hi // 2)
    return rng.choice([m << k for m in (1, 3, 5, 7, 9, 15) for k in range(4, 12) if lo <= m << k <= hi])


def draw(rng):
    kind = rng.choice(["oneshot", "pair", "grid", "degrid", "lsq", "batch", "pair64", "abi", "image", "clean", "setup"])
    if kind == "image":
        return dict(kind=kind, grid=_edge(rng, 256, 4096))
    layout = rng.choice(["disk", "core"])
    if kind == "clean":
        return dict(kind=kind, layout=layout, radius=round(rng.uniform(1000.0, 20000.0), 1), ants=_log(rng, 16, 200), times=_log(rng, 4, 64),
                    grid=_edge(rng, 256, 2048), iterations=_log(rng, 50, 200))
    radius = round(math.exp(rng.uniform(math.log(1000.0), math.log(40000.0))), 1)
    c = dict(kind=kind, layout=layout, radius=radius, chans=1, s_min=8, odd=rng.random() < 0.25)
    if kind == "oneshot":
        c.update(ants=_log(rng, 32, 256), times=rng.randint(1, 3), grid=2 * _log(rng, 128, 1024), planes=rng.randint(1, 16), s_max=rng.randint(8, 32))
    elif kind == "abi":
        c.update(ants=_log(rng, 32, 128), times=rng.randint(2, 24), grid=2 * _log(rng, 128, 512), planes=rng.randint(1, 6), s_min=rng.choice([8, 16]),
                 s_max=rng.choice([16, 32, 64]), odd=False)
    elif kind == "batch":
        c.update(ants=_log(rng, 24, 64), times=_log(rng, 8, 48), chans=rng.randint(3, 12), grid=2 * _log(rng, 128, 512), planes=rng.randint(1, 32),
                 s_max=rng.randint(16, 96))
    elif kind in ("lsq", "pair64"):
        c.update(ants=_log(rng, 24, 96), times=_log(rng, 16, 128), grid=_edge(rng, 512, 2048), planes=rng.randint(1, 24), s_max=rng.randint(8, 64))
    else:
        c.update(ants=_log(rng, 32, 256), times=_log(rng, 8, 32 if kind == "pair" else 64), grid=_edge(rng, 512, 4608), planes=_log(rng, 1, 48), s_max=rng.randint(8, 110))
    if c["planes"] == 1:
        c["s_max"] = c["s_min"]
    return c


# ---------------------------------------------------------------- observations
def _antennas(rng, layout, n, radius):
    a = rng.uniform(0, 2 * np.pi, n)
    r = radius * np.sqrt(rng.uniform(0, 1, n)) if layout == "disk" else np.exp(rng.uniform(np.log(radius / 200.0), np.log(radius), n))
    return np.stack([r * np.cos(a), r * np.sin(a)], 1)


def _tracks(ant, n_t, dec=-45.0, lat=-30.0):
    """(baselines * times, 3) metres: earth rotation over hour angles of +-4 h."""
    i, j = np.triu_indices(len(ant), 1)
    d = torch.as_tensor(ant[j] - ant[i], device=DEV)
    la, de = math.radians(lat), math.radians(dec)
    x, y, z = (-math.sin(la) * d[:, 1])[:, None], d[:, 0][:, None], (math.cos(la) * d[:, 1])[:, None]
    h = torch.as_tensor(np.linspace(-4.0, 4.0, n_t) if n_t > 1 else np.array([0.7]), device=DEV) * (math.pi / 12)
    s, c = torch.sin(h)[None, :], torch.cos(h)[None, :]
    u = s * x + c * y
    v = -math.sin(de) * c * x + math.sin(de) * s * y + math.cos(de) * z
    w = math.cos(de) * c * x - math.cos(de) * s * y + math.sin(de) * z
    return torch.stack([u, v, w], -1).reshape(-1, 3)


def _supports(lo, hi, n, s_min, s_max, odd):
    """Support of each uniform w-bin, growing as the root of |w|, and the bins' centres."""
    e = np.linspace(lo, hi, n + 1)
    top = max(abs(lo), abs(hi), 1e-300)
    sup = []
    for a, b in zip(e[:-1], e[1:]):
        inner = 0.0 if a <= 0 <= b else min(abs(a), abs(b))
        s = int(2 * math.ceil((s_min + (s_max - s_min) * math.sqrt(inner / top)) / 2))
        sup.append(min(max(s, s_min), s_max) - (1 if odd else 0))
    return np.array(sup, np.int32), 0.5 * (e[:-1] + e[1:])


def _taper(x, beta):
    return np.i0(beta * np.sqrt(np.clip(1 - x * x, 0, None))) / np.i0(beta)


def _kernels(w, sup, field):
    """Oversampled w-kernels [plane][8 ov + ou][sy][sx] in 64 bits, end to end: the transform of a tapered phase screen over the field of view."""
    m = int(sup.max())
    m += m & 1
    n, r = OVER * m, m // 2
    k = torch.arange(-r, r, dtype=torch.float64, device=DEV)
    lm = k * (field / 2) / r
    t = torch.as_tensor(_taper(np.arange(-r, r) / r, 6.0), device=DEV)
    root = torch.sqrt(torch.clamp(1 - lm[:, None] ** 2 - lm[None, :] ** 2, min=0))
    out = []
    for wp, s in zip(w, sup):
        s = int(s)
        arena = torch.zeros(n, n, dtype=torch.complex128, device=DEV)
        arena[n // 2 - r:n // 2 + r, n // 2 - r:n // 2 + r] = torch.polar(t[:, None] * t[None, :], -2 * math.pi * float(wp) * (1 - root))
        f = torch.fft.fftshift(torch.fft.ifft2(torch.fft.ifftshift(arena), norm="forward")).reshape(m, OVER, m, OVER)  # [x][ou][y][ov]
        total = f.real.sum((0, 2))
        c = r - s // 2
        out.append((f[c:c + s, :, c:c + s, :] / total[None, :, None, :]).permute(3, 1, 2, 0).reshape(-1))
    return torch.cat(out)


def _members(c):
    """(grid size, share of the band) of each grid of a case: one, or a batch's channels with every fourth one a facet of twice, then four times the size."""
    if c["kind"] != "batch":
        return [(c["grid"], 1.0)]
    return [(c["grid"] * (1, 1, 2, 4)[k % 4], 1.0 + 0.05 * k) for k in range(c["chans"])]


def observe(c, seed):
    """uvw of each member in wavelengths, the pixel scale, the w-planes and their supports."""
    rng = np.random.default_rng([seed, 17])
    m = _tracks(_antennas(rng, c["layout"], c["ants"], c["radius"]), c["times"])
    chans = [1.0] if c["kind"] == "batch" else [1.0 + 0.01 * k for k in range(c["chans"])]
    uvw, sizes = [], []
    for g, f in _members(c):
        x = torch.stack([m * (150e6 * f * k / LIGHT) for k in chans], 1).reshape(-1, 3) if len(chans) > 1 else m * (150e6 * f / LIGHT)
        uvw.append(x.contiguous())
        sizes.append(g)
    scale = min(0.9 * (g / 2) / float((x[:, 0] ** 2 + x[:, 1] ** 2).max().sqrt()) for x, g in zip(uvw, sizes))
    hi = max(float(x[:, 2].abs().max()) for x in uvw) * 1.0001
    lo = -hi
    if c["planes"] > 1:
        sup, w = _supports(lo, hi, c["planes"], c["s_min"], c["s_max"], c["odd"])
    else:
        sup, w, lo, hi = np.array([c["s_min"] - (1 if c["odd"] else 0)], np.int32), np.zeros(1), -math.inf, math.inf
    off = np.concatenate([[0], np.cumsum(64 * sup.astype(np.int64) ** 2)])[:-1]
    return dict(uvw=uvw, sizes=sizes, scale=scale, sup=sup, w=w, off=off, range=(lo, hi), margin=int(sup.max()))


def _sky(rng, field, n=20):
    l, m = rng.uniform(-0.3 * field, 0.3 * field, (2, n))
    return l, m, np.exp(rng.uniform(np.log(0.1), np.log(10.0), n))


def _visibilities(uvw, sky, gen):
    """The sky's point sources with noise of 0.01, complex128."""
    out = torch.randn(uvw.shape[0], dtype=torch.complex128, device=DEV, generator=gen) * 0.01
    for l, m, f in zip(*sky):
        out += torch.polar(torch.full_like(uvw[:, 0], f), -2 * math.pi * (uvw @ torch.tensor([l, m, math.sqrt(1 - l * l - m * m) - 1], dtype=torch.float64, device=DEV)))
    return out


def _gen(seed, k=0):
    return torch.Generator(device=DEV).manual_seed(1000 * seed + k)


def _image(n, seed):
    """A sky image of 20 Gaussian blobs in the inner half."""
    rng = np.random.default_rng([seed, 29])
    x = torch.arange(n, dtype=torch.float64, device=DEV)
    img = torch.zeros(n, n, dtype=torch.float64, device=DEV)
    for _ in range(20):
        cy, cx = rng.uniform(0.25 * n, 0.75 * n, 2)
        s, a = rng.uniform(1, 5), math.exp(rng.uniform(math.log(0.1), math.log(10)))
        img += a * torch.exp(-(x - cy) ** 2 / (2 * s * s))[:, None] * torch.exp(-(x - cx) ** 2 / (2 * s * s))[None, :]
    return img.float()


def _correction(n):
    return torch.as_tensor(_taper((np.arange(n) - n // 2) / (n / 2), 4.0), device=DEV).float()


def _to_grid(img, taper=None):
    x = img.double()
    if taper is not None:
        t = taper.double()
        x = x / (t[:, None] * t[None, :])
    return torch.fft.fftshift(torch.fft.fft2(torch.fft.ifftshift(x)))


def _to_image(grid, taper):
    t = taper.double()
    return torch.fft.fftshift(torch.fft.ifft2(torch.fft.ifftshift(grid.to(torch.complex128)), norm="forward")).real / (t[:, None] * t[None, :])


def _inputs(c, seed):
    """Everything that a case on visibilities is given, but the plan."""
    o = observe(c, seed)
    field = o["scale"]
    sky = _sky(np.random.default_rng([seed, 23]), min(field, 0.3))
    wide = c["kind"] in ("pair64", "abi")
    g = _kernels(o["w"], o["sup"], min(field, 0.9))
    o["gcf"] = g if wide else g.to(torch.complex64)
    if c["kind"] != "setup":
        o["vis"] = [_visibilities(x, sky, _gen(seed, k)).to(torch.complex128 if wide else torch.complex64) for k, x in enumerate(o["uvw"])]
    if c["kind"] in ("degrid", "pair", "batch", "pair64", "abi"):
        o["model"] = [_to_grid(_image(n, seed + k)).to(torch.complex128 if wide else torch.complex64) for k, n in enumerate(o["sizes"])]
    if c["kind"] == "lsq":
        o["image"], o["taper"] = _image(c["grid"], seed) * 0.5, _correction(c["grid"])
    return o


def _clean_inputs(c, seed):
    """A dirty image of 30 point sources, the PSF of the array's uv coverage and both their sizes."""
    n = c["grid"]
    full = 2 * n
    uvw = _tracks(_antennas(np.random.default_rng([seed, 17]), c["layout"], c["ants"], c["radius"]), c["times"])
    uv = torch.round(uvw[:, :2] * (0.9 * n / float((uvw[:, 0] ** 2 + uvw[:, 1] ** 2).max().sqrt()))).long() + full // 2
    cover = torch.zeros(full * full, dtype=torch.float64, device=DEV)
    cover.index_add_(0, torch.cat([uv[:, 1] * full + uv[:, 0], (full - uv[:, 1]) * full + full - uv[:, 0]]), torch.ones(2 * len(uv), dtype=torch.float64, device=DEV))
    cover = torch.sqrt(cover).reshape(full, full)
    psf = torch.fft.fftshift(torch.fft.ifft2(torch.fft.ifftshift(cover))).real
    psf = psf / psf[n, n]
    rng = np.random.default_rng([seed, 31])
    sky = torch.zeros(full, full, dtype=torch.float64, device=DEV)
    for _ in range(30):
        y, x = rng.integers(n // 8, n - n // 8, 2)
        sky[n // 2 + y, n // 2 + x] += math.exp(rng.uniform(math.log(0.05), math.log(5.0)))
    dirty = torch.fft.ifft2(torch.fft.fft2(sky) * torch.fft.fft2(torch.fft.ifftshift(psf))).real
    dirty = dirty[n // 2:n // 2 + n, n // 2:n // 2 + n] + 0.002 * torch.randn(n, n, dtype=torch.float64, device=DEV, generator=_gen(seed))
    h = n // 2
    return dirty.float().contiguous(), psf[n - h:n + h, n - h:n + h].float().contiguous(), h


# ---------------------------------------------------------------- prepare and run
def _plan_args(o, k=0):
    n = o["sizes"][k]
    return dict(scale=o["scale"], grid_size=n, grid_shape=(n, n), supports=o["sup"], gcf_offsets=o["off"], margin=o["margin"], w_range=o["range"])


def prepare(case, seed):
    from rc_gb300 import engine, lib

    kind = case["kind"]
    if kind == "image":
        n = case["grid"]
        return dict(kind=kind, n=n, image=_image(n, seed), taper=_correction(n), grid=torch.randn(n, n, dtype=torch.complex64, device=DEV, generator=_gen(seed)))
    if kind == "clean":
        dirty, psf, h = _clean_inputs(case, seed)
        n, b = case["grid"], ctypes.c_int64()
        lib.check(lib.load().gb_hogbom_work_bytes(n, n, ctypes.byref(b)))
        return dict(kind=kind, n=n, dirty=dirty, psf=psf, h=h, iterations=case["iterations"], work=torch.empty(b.value, dtype=torch.uint8, device=DEV))
    o = _inputs(case, seed)
    s = dict(kind=kind, **o)
    if kind == "setup":
        s["support"] = o["margin"] + (o["margin"] & 1)
        return s
    if kind == "abi":
        return _host_state(s)
    if kind == "oneshot":
        g = lib.Geometry()
        n = o["sizes"][0]
        g.scale, g.grid_size, g.margin, g.ext_x, g.ext_y, g.pitch, g.n_planes = o["scale"], n, o["margin"], n, n, n, len(o["sup"])
        s["hold"] = (np.ascontiguousarray(o["sup"], np.int32), np.ascontiguousarray(o["off"], np.int64))
        g.supports = s["hold"][0].ctypes.data_as(ctypes.POINTER(ctypes.c_int32))
        g.gcf_offsets = s["hold"][1].ctypes.data_as(ctypes.POINTER(ctypes.c_int64))
        g.w_low, g.w_high = o["range"]
        s["geo"] = g
    elif kind == "batch":
        s["batch"] = engine.Batch([dict(uvw=x, **_plan_args(o, k)) for k, x in enumerate(o["uvw"])])
    else:
        s["plan"] = engine.Plan(o["uvw"][0], **_plan_args(o))
    if kind in ("oneshot", "grid", "pair", "batch", "pair64"):
        s["out"] = [torch.zeros(n, n, dtype=torch.complex128 if kind == "pair64" else torch.complex64, device=DEV) for n in o["sizes"]]
    if kind in ("degrid", "pair", "batch", "pair64"):
        s["pred"] = [torch.empty_like(v) for v in o["vis"]]
    return s


def _bins(o):
    """The records of each w-bin, as the reference's binner hands them to the kernels."""
    x = o["uvw"][0]
    p = _index(x, o, 0)[0]
    rec = torch.cat([x, torch.view_as_real(o["vis"][0])], 1)
    return [(k, rec[p == k].cpu().numpy()) for k in range(len(o["sup"])) if bool((p == k).any())]


def _abi_size(s):
    return next(k for k in (8, 16, 32, 64) if s <= k)


def _abi_kernels(o):
    """The drop-in kernels take sizes 8, 16, 32 and 64: each plane's kernel in the middle of the next such size."""
    out = []
    for s, a in zip(o["sup"], o["off"]):
        k, s = _abi_size(int(s)), int(s)
        g = torch.zeros(64, k, k, dtype=torch.complex128, device=DEV)
        c = k // 2 - s // 2
        g[:, c:c + s, c:c + s] = o["gcf"][a:a + 64 * s * s].reshape(64, s, s)
        out.append(g.cpu().numpy())
    return out


def _host_state(s):
    n = s["sizes"][0]
    s["bins"] = _bins(s)
    s["host_gcf"] = _abi_kernels(s)
    s["host_model"] = np.ascontiguousarray(s["model"][0].cpu().numpy())
    s["host_grid"] = np.zeros((n, n), np.complex128)
    s["host_out"] = np.zeros((sum(len(r) for _, r in s["bins"]), 5))
    return s


def _run_oneshot(s):
    from rc_gb300 import lib

    g, n = s["out"][0], s["uvw"][0].shape[0]
    g.zero_()
    lib.check(lib.load().gb_grid_f32_noalloc(ctypes.byref(s["geo"]), n, s["uvw"][0].data_ptr(), 3, None, s["vis"][0].data_ptr(), s["gcf"].data_ptr(), g.data_ptr(),
                                             torch.cuda.current_stream().cuda_stream), "gb_grid_f32_noalloc")
    return g


def _run_abi(s):
    from rc_gb300 import compat, lib

    n, args = s["sizes"][0], (s["scale"], s["sizes"][0], max(_abi_size(int(x)) for x in s["sup"]))
    b = compat.grid_buf(s["host_grid"])
    lib.check(lib.load().kern_init(ctypes.byref(b)), "kern_init")
    for k, r in s["bins"]:
        lib.check(compat.call_scatter("kern_scatter_gpu1", *args, r, s["host_gcf"][k], s["host_grid"]), "kern_scatter_gpu1")
    at = 0
    for k, r in s["bins"]:
        out = s["host_out"][at:at + len(r)]
        lib.check(compat.call_degrid("kern_degrid_gpu1", *args, s["host_gcf"][k], s["host_model"], r, out), "kern_degrid_gpu1")
        at += len(r)
    return {"grid": s["host_grid"], "vis": s["host_out"]}


def _run_clean(s):
    from rc_gb300 import lib

    n = s["n"]
    res, model = s["dirty"].clone(), torch.zeros_like(s["dirty"])
    lib.check(lib.load().gb_hogbom_f32(res.data_ptr(), n, n, s["psf"].data_ptr(), 2 * s["h"], 2 * s["h"], s["h"], s["h"], 0.1, 0.0, s["iterations"], model.data_ptr(),
                                       s["work"].data_ptr(), s["work"].numel(), torch.cuda.current_stream().cuda_stream), "gb_hogbom_f32")
    return {"residual": res, "model": model}


def run(state):
    from rc_gb300 import autograd, engine, gcf

    s, kind = state, state["kind"]
    if kind == "oneshot":
        return _run_oneshot(s)
    if kind == "abi":
        return _run_abi(s)
    if kind == "clean":
        return _run_clean(s)
    if kind == "image":
        return {"grid": autograd.ImageToGrid.apply(s["image"], s["taper"]), "image": autograd.grid_to_image(s["grid"], s["taper"])}
    if kind == "setup":
        n = s["support"]
        g64, g32, _ = gcf.generate(s["w"], s["sup"], n, min(s["scale"], 0.9) / 2, taper=_taper(np.arange(-(n // 2), n // 2) / (n // 2), 6.0))
        plan = engine.Plan(s["uvw"][0], **_plan_args(s))
        return {"gcf64": g64, "gcf32": g32, "index": plan.export_index()}
    if kind == "lsq":
        image = s["image"].detach().requires_grad_(True)
        pred = autograd.forward_model(image, s["taper"], s["plan"], s["gcf"])
        r = pred - s["vis"][0]
        loss = 0.5 * (r.real.square().sum() + r.imag.square().sum())
        loss.backward()
        return {"pred": pred.detach(), "loss": loss.detach(), "grad": image.grad}
    out = {}
    if kind == "batch":
        for g in s["out"]:
            g.zero_()
        out["grid"] = s["batch"].grid(s["vis"], s["gcf"], s["out"])
        out["vis"] = s["batch"].degrid(s["gcf"], s["model"], s["pred"])
        return out
    p, wide = s["plan"], kind == "pair64"
    if kind in ("grid", "pair", "pair64"):
        s["out"][0].zero_()
        out["grid"] = (p.grid64 if wide else p.grid)(s["vis"][0], s["gcf"], s["out"][0])
    if kind in ("degrid", "pair", "pair64"):
        out["vis"] = (p.degrid64 if wide else p.degrid)(s["gcf"], s["model"][0], s["pred"][0])
    return out


# ---------------------------------------------------------------- the work, and the answers in 64 bits
def _index(uvw, o, k, abi=False):
    """Plane, corner column and row, phase of each visibility; plane -1 for one that is out of bounds."""
    n, (lo, hi), np_ = o["sizes"][k], o["range"], len(o["sup"])
    p = torch.zeros(len(uvw), dtype=torch.long, device=uvw.device)
    if np_ > 1:
        w = uvw[:, 2]
        p = torch.clamp(torch.floor((w - lo) / (hi - lo) * np_), 0, np_ - 1).long()
        p = torch.where((w >= lo) & (w <= hi), p, torch.full_like(p, -1))
    sizes = [_abi_size(int(s)) for s in o["sup"]] if abi else [int(s) for s in o["sup"]]
    s = torch.tensor(sizes, dtype=torch.long, device=uvw.device)[p]
    c, over = [], []
    for a in (0, 1):
        x = uvw[:, a] * o["scale"]
        over.append(torch.clamp(torch.round(OVER * (x - torch.floor(x))), 0, OVER - 1).long())
        c.append(torch.round(x).long() + n // 2 - s // 2)
    g = torch.clamp(torch.div((max(sizes) if abi else o["margin"]) - s, 2, rounding_mode="floor"), min=0)
    ok = (c[0] >= g) & (c[0] <= n - s - 1 - g) & (c[1] >= g) & (c[1] <= n - s - 1 - g)
    return torch.where(ok, p, torch.full_like(p, -1)), c[0], c[1], over[0] + OVER * over[1]


def _parts(uvw, o, k, abi=False):
    """(which visibilities, their kernels, their pixels), a few million taps at a time."""
    p, x, y, ph = _index(uvw, o, k, abi)
    host = _abi_kernels(o) if abi else None
    n = o["sizes"][k]
    for q, (s, a) in enumerate(zip(o["sup"], o["off"])):
        s = int(s)
        g = o["gcf"][a:a + 64 * s * s].reshape(64, s, s).to(torch.complex128)
        if abi:
            s, g = _abi_size(s), torch.as_tensor(host[q], device=DEV)
        d = torch.arange(s, device=DEV)
        at = (d[:, None] * n + d[None, :]).reshape(-1)
        which = torch.nonzero(p == q)[:, 0]
        for part in torch.split(which, max(1, (1 << 24) // (s * s))):
            yield part, g.reshape(64, -1)[ph[part]], (y[part] * n + x[part])[:, None] + at[None, :]


def _exact_grid(uvw, vis, o, k=0, abi=False):
    n = o["sizes"][k]
    out = torch.zeros(n * n, 2, dtype=torch.float64, device=DEV)
    for part, g, at in _parts(uvw, o, k, abi):
        out.index_add_(0, at.reshape(-1), torch.view_as_real(vis[part].to(torch.complex128)[:, None] * g).reshape(-1, 2))
    return torch.view_as_complex(out).reshape(n, n)


def _exact_degrid(uvw, grid, o, k=0, abi=False):
    out = torch.zeros(len(uvw), dtype=torch.complex128, device=DEV)
    flat = grid.to(torch.complex128).reshape(-1)
    for part, g, at in _parts(uvw, o, k, abi):
        out[part] = (flat[at] * (g if abi else g.conj())).sum(1)
    return out


def _exact_clean(c, seed):
    dirty, psf, h = _clean_inputs(c, seed)
    n, r, p = c["grid"], dirty.double(), psf.double()
    model = torch.zeros_like(r)
    for _ in range(c["iterations"]):
        at = int(r.abs().argmax())
        y, x = divmod(at, n)
        f = 0.1 * float(r[y, x])
        model[y, x] += f
        y0, y1, x0, x1 = max(0, y - h), min(n, y + h), max(0, x - h), min(n, x + h)
        r[y0:y1, x0:x1] -= f / float(p[h, h]) * p[y0 - y + h:y1 - y + h, x0 - x + h:x1 - x + h]
    return {"residual": r, "model": model}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "clean":
        return _exact_clean(c, seed)
    if kind == "image":
        s = prepare(c, seed)
        return {"grid": _to_grid(s["image"], s["taper"]), "image": _to_image(s["grid"], s["taper"])}
    o = _inputs(c, seed)
    u = o["uvw"]
    if kind == "setup":
        g = _kernels(o["w"], o["sup"], min(o["scale"], 0.9))
        return {"gcf64": g, "gcf32": g, "index": None}
    if kind == "abi":
        recs = _bins(o)
        bins = [torch.as_tensor(r, device=DEV) for _, r in recs]
        x = torch.cat([b[:, :3] for b in bins])
        v = torch.view_as_complex(torch.cat([b[:, 3:] for b in bins]).contiguous())
        out = torch.cat([x, torch.view_as_real(v - _exact_degrid(x, o["model"][0], o, 0, True))], 1)
        return {"grid": _exact_grid(x, v, o, 0, True), "vis": out}
    if kind == "lsq":
        pred = _exact_degrid(u[0], _to_grid(o["image"], o["taper"]), o)
        r = pred - o["vis"][0]
        return {"pred": pred, "loss": 0.5 * r.abs().square().sum(), "grad": _to_image(_exact_grid(u[0], r, o), o["taper"])}
    if kind == "batch":
        return {"grid": [_exact_grid(x, o["vis"][k], o, k) for k, x in enumerate(u)], "vis": [_exact_degrid(x, o["model"][k], o, k) for k, x in enumerate(u)]}
    if kind == "oneshot":
        return _exact_grid(u[0], o["vis"][0], o)
    out = {}
    if kind != "degrid":
        out["grid"] = _exact_grid(u[0], o["vis"][0], o)
    if kind != "grid":
        out["vis"] = _exact_degrid(u[0], o["model"][0], o)
    return out


def work(case):
    """Bytes that the operation cannot do without, each input read and each output written once, and its additions and multiplications."""
    c, kind = case, case["kind"]
    n = c["grid"]
    cells = n * n
    if kind == "image":  # real and complex n x n both ways; two real transforms
        return {"bytes": 2 * 12 * cells, "flops": 2 * 2.5 * cells * math.log2(cells)}
    if kind == "clean":  # dirty image, PSF, residual and model; a subtraction over the PSF's overlap, about 9/16 of the window, in each iteration
        return {"bytes": 16 * cells, "flops": c["iterations"] * 2 * 9 / 16 * cells}
    o = observe(c, 0)
    taps = vis = 0
    for k, u in enumerate(o["uvw"]):
        p = _index(u, o, k, kind == "abi")[0]
        s = [_abi_size(int(x)) if kind == "abi" else int(x) for x in o["sup"]]
        taps += int((torch.tensor(s, device=u.device)[p[p >= 0]] ** 2).sum())
        vis += len(u)
    cells = sum(x * x for x in o["sizes"])
    gcf = 64 * int((o["sup"].astype(np.int64) ** 2).sum())
    if kind == "setup":  # uvw in, index records out, kernels out in both precisions; the planes' transforms of 8 x 8 phases of the screen
        m = int(o["sup"].max())
        return {"bytes": 24 * vis + 20 * vis + 24 * gcf, "flops": len(o["sup"]) * 5 * 64 * m * m * math.log2(64 * m * m)}
    width = 16 if kind in ("pair64", "abi") else 8
    both = 2 if kind in ("pair", "batch", "pair64", "abi", "lsq") else 1
    extra = 8 * cells if kind == "lsq" else 0
    if kind == "oneshot":
        extra = 24 * vis
    if kind == "abi":
        extra = 2 * 24 * vis + 24 * vis
    return {"bytes": width * (both * vis + gcf + both * cells) + extra, "flops": 8 * taps * both}
