"""The extraction workloads whose speed is measured.

A case is one frame (or one list of frames) and the settings it is extracted
with, through the public entry points of the library: the C ABI on frames that
are already on the GPU (a reduction pipeline that calibrated them there), the
Python calls on host frames and on FITS data blocks, the frame stream, the
batch, and the background stage alone.  Frames are synthetic star and galaxy
fields with the densities, fluxes and noise of the repository's workloads,
rendered on the GPU from the seed alone (sources are deposited as whole
numbers, so the frame does not depend on the order of the additions).

Fields of a case
  entry    device: frame in device memory, rows to the caller's page-locked
           buffer; host: numpy frame in, rows and segmentation map out; fits:
           16-bit or float FITS data block in; stream: page-locked frames
           through submit / next; batch: a list of frames of mixed sizes;
           background: the background stage without allocation
  w, h     frame size (of the largest frame of a batch)
  field    sparse, survey: uniform density; king: a star cluster; gauss: plain
           point sources on a gradient sky
  density  injected sources per pixel
  fwhm, taps  Gaussian detection mask (0 taps: mexican hat of 7 x 7)
  graph    1: captured graphs ("graph" parameter)
  weight   WEIGHT_TYPE; local: BACKPHOTO_TYPE LOCAL; naper: apertures
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gpu-sextractor_b200"))
import sexgpu  # noqa: E402

DEFAULTS = dict(entry="device", field="survey", density=0.0119, fwhm=2.5, taps=5, graph=0, weight=0, local=0, naper=1,
                back_size=64, nthresh=32, mincont=0.005, minarea=5, clean=1, bitpix=0, frames=1)


def _case(name, w, h, **kw):
    c = dict(DEFAULTS, w=w, h=h)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: a cutout around one target, taken from an image
        # in host memory, with its segmentation map
        _case("cutout_160", 160, 160, entry="host", field="gauss", density=0.0019, fwhm=2.0, taps=3),
        # a detector quadrant already on the GPU, default settings, odd size
        # (rows that are no multiple of 16 bytes)
        _case("quadrant_1023", 1023, 1021, field="gauss", density=0.0019, fwhm=2.0, taps=3),
        # the same kind of frame over and over in a survey's loop: captured graph
        _case("survey_1024_graph", 1024, 1024, field="survey", density=0.006, graph=1, fwhm=2.0, taps=3, back_size=32),
        # a camera's FITS file as it is stored (16-bit integers), as the command
        # line reads it, with the segmentation map
        _case("fits16_2048", 2048, 1489, entry="fits", bitpix=16, field="sparse", density=0.002, fwhm=3.0, taps=7),
        # host frames through the stream: the next upload overlaps this extraction
        _case("stream_2048", 2048, 2048, entry="stream", density=0.006, fwhm=2.0, taps=3),
        # a weighted mosaic tile of ragged size, LOCAL background, four apertures
        _case("weighted_local_2501", 2501, 1999, field="sparse", density=0.004, weight=3, local=1, naper=4),
        # the background stage by itself, in a calibration loop that must not allocate
        _case("background_3200", 3200, 3120, entry="background", field="sparse", density=0.002),
        # a sparse extragalactic survey frame
        _case("sparse_4096", 4096, 4096, field="sparse", density=0.0006, fwhm=3.0, taps=7, back_size=128),
        # the reference's headline frame: 4096 x 4096, 43% of the pixels in objects
        _case("crowded_4096", 4096, 4096),
        # a star cluster, deblended finely
        _case("cluster_4096", 4096, 4096, field="king", density=0.0238, nthresh=64, mincont=0.0005),
        # a mixed list of frames (a night's detectors and cutouts) as one batch
        _case("batch_mixed", 2048, 2048, entry="batch", density=0.005, frames=12, graph=1, fwhm=2.0, taps=3),
        # the largest: a mosaic with its variance map
        _case("mosaic_16384", 16384, 16384, density=0.0093, weight=1, back_size=128, fwhm=4.0, taps=7),
    ]


def draw(rng):
    entry = rng.choice(["device"] * 6 + ["host", "fits", "stream", "batch", "background"])
    # area over its logarithm, from cutouts to mosaics (the host frames to
    # 4096 x 4096, the background stage to its limit on the number of meshes)
    top = {"device": 12288, "background": 3800, "batch": 2048}.get(entry, 4096)
    low = 512 if entry == "batch" else 96
    side = math.exp(rng.uniform(math.log(low), math.log(top)))
    aspect = math.exp(rng.uniform(-0.5, 0.5))
    w, h = max(64, int(side * math.sqrt(aspect))), max(64, int(side / math.sqrt(aspect)))
    if rng.random() < 0.5:
        w = w // 16 * 16
    field = rng.choice(["sparse", "survey", "survey", "gauss", "king"])
    density = math.exp(rng.uniform(math.log(3e-4), math.log(0.012)))
    if field == "king":
        side = min(side, 4096)
        w, h = min(w, 4096), min(h, 4096)
    taps, fwhm = rng.choice([(3, 1.5), (3, 2.0), (5, 2.5), (5, 3.0), (7, 3.0), (7, 4.0), (9, 5.0), (0, 2.5)])
    fine = side <= 4096 and rng.random() < 0.25
    return _case(None, w, h, entry=entry, field=field, density=density, fwhm=fwhm, taps=taps,
                 graph=1 if entry == "batch" else int(entry in ("device", "stream") and rng.random() < 0.4),
                 # (a mask with negative taps turns the masked pixels into detections: not used with weights)
                 weight=rng.choice([0, 0, 0, 1, 2, 3, 4]) if entry in ("device", "host") and taps else 0,
                 local=int(entry in ("device", "host") and side <= 4096 and rng.random() < 0.2),
                 naper=rng.choice([1, 1, 1, 3, 6]), back_size=rng.choice([32, 64, 64, 100, 128]),
                 nthresh=64 if fine else 32, mincont=0.0005 if fine else 0.005, minarea=rng.choice([3, 5, 5, 8]),
                 clean=int(rng.random() < 0.85), bitpix=rng.choice([16, -32]) if entry == "fits" else 0,
                 frames=rng.choice([4, 9, 12]) if entry == "batch" else 1)


# ---------------------------------------------------------------------------
# frames
# ---------------------------------------------------------------------------
MARGIN = 24        # canvas border around the frame: the largest stamp's half size
QUANTUM = 256.0    # deposited counts per ADU


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _rand(n, g, lo=0.0, hi=1.0):
    return torch.rand(n, generator=g, device="cuda") * (hi - lo) + lo


def _deposit(canvas, x, y, flux, half, profile):
    """Adds stamps of (2 half + 1) squared pixels, each scaled to its flux."""
    pitch = canvas.shape[1]
    off = torch.arange(-half, half + 1, device="cuda")
    step = max(1, (1 << 24) // (2 * half + 1) ** 2)
    for k in range(0, x.numel(), step):
        s = slice(k, k + step)
        ix, iy = torch.floor(x[s] + 0.5).long(), torch.floor(y[s] + 0.5).long()
        dx = (ix.float() - x[s])[:, None, None] + off[None, None, :]
        dy = (iy.float() - y[s])[:, None, None] + off[None, :, None]
        img = profile(s, dx, dy)
        img = img * (flux[s] * QUANTUM / img.sum(dim=(1, 2)))[:, None, None]
        idx = (iy[:, None, None] + off[None, :, None] + MARGIN) * pitch + ix[:, None, None] + off[None, None, :] + MARGIN
        canvas.view(-1).index_add_(0, idx.reshape(-1), torch.round(img).to(torch.int32).reshape(-1))


def _positions(c, n, w, h, g):
    if c["field"] != "king":
        x, y = _rand(n, g, 0, w - 1), _rand(n, g, 0, h - 1)
        m = n // 40  # blended pairs, 3 to 10 pixels apart
        r, t = _rand(m, g, 3.0, 10.0), _rand(m, g, 0.0, 2 * math.pi)
        x[:m], y[:m] = x[m:2 * m] + r * torch.cos(t), y[m:2 * m] + r * torch.sin(t)
    else:  # King profile, core radius 0.073 and tidal radius 0.49 of the frame
        rc, rt = 0.0732 * min(w, h), 0.488 * min(w, h)
        cut = 1.0 / math.sqrt(1.0 + (rt / rc) ** 2)
        r = rt * torch.sqrt(_rand(40 * n, g))
        p = ((1.0 / torch.sqrt(1.0 + (r / rc) ** 2) - cut) / (1.0 - cut)) ** 2
        r = r[_rand(40 * n, g) < p][:n]
        t = _rand(r.numel(), g, 0.0, 2 * math.pi)
        x, y = w / 2 + r * torch.cos(t), h / 2 + r * torch.sin(t)
    return x.clamp(0, w - 1), y.clamp(0, h - 1)


def _frame(c, w, h, seed):
    """A w x h frame (float32, on the GPU) of the case's kind of field."""
    g = _gen(seed)
    x, y = _positions(c, max(1, round(c["density"] * w * h)), w, h, g)
    n = x.numel()
    canvas = torch.zeros(h + 2 * MARGIN, w + 2 * MARGIN, dtype=torch.int32, device="cuda")
    if c["field"] == "gauss":
        flux = 10.0 ** _rand(n, g, 2.0, 5.0)
        sigma = 3.0 / 2.3548
        _deposit(canvas, x, y, flux, 8, lambda s, dx, dy: torch.exp(-0.5 * (dx * dx + dy * dy) / sigma ** 2))
    else:
        lo = 1e2 if c["field"] in ("king", "sparse") else 1e3
        u = _rand(n, g)
        flux = (lo ** -0.75 + u * (1e6 ** -0.75 - lo ** -0.75)) ** (-1.0 / 0.75)
        star = _rand(n, g) < 0.6
        k = torch.nonzero(star).view(-1)
        alpha2 = (2.5 / (2.0 * math.sqrt(2.0 ** (1.0 / 3.0) - 1.0))) ** 2
        _deposit(canvas, x[k], y[k], flux[k], 12, lambda s, dx, dy: (1.0 + (dx * dx + dy * dy) / alpha2) ** -3.0)
        re, index = _rand(n, g, 1.0, 8.0), _rand(n, g, 0.5, 4.0)
        q, pa = _rand(n, g, 0.3, 1.0), _rand(n, g, 0.0, math.pi)
        for half, lo_re, hi_re in ((8, 0.0, 8 / 3), (16, 8 / 3, 16 / 3), (24, 16 / 3, 99.0)):
            k = torch.nonzero(~star & (re >= lo_re) & (re < hi_re)).view(-1)

            def sersic(s, dx, dy, k=k):
                p = [v[k][s][:, None, None] for v in (torch.cos(pa), torch.sin(pa), q, re, index)]
                u, v = dx * p[0] + dy * p[1], (dy * p[0] - dx * p[1]) / p[2]
                r = torch.sqrt(u * u + v * v + 0.1)
                return torch.exp(-(2.0 * p[4] - 1.0 / 3.0) * ((r / p[3]) ** (1.0 / p[4]) - 1.0))

            _deposit(canvas, x[k], y[k], flux[k], half, sersic)
    img = torch.empty(h, w, device="cuda")
    cx = _rand(5, g, -1.0, 1.0).tolist()
    u = torch.linspace(-1, 1, w, device="cuda")[None, :]
    for y0 in range(0, h, 2048):  # bands, so that the largest frame needs no frame-size temporaries
        y1 = min(h, y0 + 2048)
        src = canvas[MARGIN + y0:MARGIN + y1, MARGIN:MARGIN + w].float() / QUANTUM
        v = torch.arange(y0, y1, device="cuda")[:, None] * (2.0 / max(1, h - 1)) - 1
        noise = torch.randn(y1 - y0, w, generator=g, device="cuda")
        if c["field"] == "gauss":
            img[y0:y1] = 1025.0 + 25.0 * u + src + 10.0 * noise
        else:
            sky = 800.0 * (1.0 + 0.02 * (cx[0] * u + cx[1] * v + cx[2] * u * u + cx[3] * u * v + cx[4] * v * v))
            img[y0:y1] = torch.clamp(sky + src + noise * torch.sqrt(64.0 + src), max=60000.0)
    if c["field"] != "gauss":
        img[:, (_rand(3, g) * w).long().clamp(max=w - 1)] = 0.0  # dead columns
    return img


def _weight(c, w, h, seed):
    """The case's weight map: noise varying by 20%, 2% of the pixels masked."""
    if c["weight"] not in (1, 2, 3):
        return None
    g = _gen(seed + 7919)
    u = torch.linspace(0, 6.2832, w, device="cuda")[None, :]
    v = torch.linspace(0, 6.2832, h, device="cuda")[:, None]
    k = _rand(2, g, 1.0, 4.0).tolist()
    var = torch.sin(k[0] * u + 1.0) * torch.cos(k[1] * v + 2.0)
    var.mul_(0.2).add_(1.0).mul_(64.0)
    dead = torch.rand((h + 7) // 8, (w + 7) // 8, generator=g, device="cuda") < 0.02
    dead = dead.repeat_interleave(8, 0)[:h].repeat_interleave(8, 1)[:, :w]
    if c["weight"] == 2:
        var.sqrt_()
    elif c["weight"] == 3:
        var.reciprocal_()
    var.masked_fill_(dead, 0.0 if c["weight"] == 3 else 1e30)
    return var


def _mask(c):
    n = c["taps"] or 7
    r2 = (np.arange(n)[:, None] - n // 2) ** 2.0 + (np.arange(n)[None, :] - n // 2) ** 2.0
    s2 = (c["fwhm"] / 2.3548) ** 2
    m = np.exp(-0.5 * r2 / s2) * (1.0 if c["taps"] else 1.0 - 0.5 * r2 / s2)
    return (m / np.abs(m).sum()).astype(np.float32)


def _settings(c):
    kw = dict(conv=_mask(c), back_size=c["back_size"], deblend_nthresh=c["nthresh"], deblend_mincont=c["mincont"],
              detect_minarea=c["minarea"], clean_flag=c["clean"], weight_type=c["weight"], back_photo_type=c["local"])
    if c["naper"] > 1:
        kw["phot_apertures"] = [4.0 + 3.0 * k for k in range(c["naper"])]
    return kw


def _pinned(t):
    """A page-locked host copy as a numpy array (and the tensor that owns it)."""
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    p.copy_(t)
    return p.numpy()


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def _room(w, h):
    """Rows kept for a frame's catalogue: more than such a field gives."""
    return w * h // (80 if w * h <= 1 << 24 else 160) + 256


def _keep(table, rows):
    """A catalogue into the program's own table (zero beyond its rows)."""
    table.view(np.uint8)[:rows.nbytes] = rows.view(np.uint8)
    return table


def prepare(case, seed):
    c = case
    w, h, entry = c["w"], c["h"], c["entry"]
    s = dict(case=c, kw=_settings(c))
    if entry == "batch":
        # half detectors of full size, the rest halves and quarters
        s["frames"] = []
        for i in range(c["frames"]):
            d = (1, 1, 2, 4)[i % 4]
            f = _frame(c, w // d, h // d, seed * 64 + i).cpu().numpy()
            s["frames"].append((f, dict(s["kw"], back_size=(32, 64, 128)[i % 3])))
    else:
        img, wmap = _frame(c, w, h, seed), _weight(c, w, h, seed)
        if entry == "device":
            s["img"], s["wmap"] = img, wmap
            # the page-locked buffers that the rows come to
            rows = _room(w, h)
            pin = torch.zeros(rows * sexgpu.OBJECT_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True)
            s["rows"] = pin.numpy().view(sexgpu.OBJECT_DTYPE)
            if c["naper"] > 1:
                s["apers"] = torch.zeros(rows, c["naper"], 4, pin_memory=True).numpy()
        elif entry == "host":
            s["img"] = img.cpu().numpy()
            s["wmap"] = wmap.cpu().numpy() if wmap is not None else None
        elif entry == "fits":
            f = img.cpu().numpy()
            s["data"] = (np.rint(f) - 32768).clip(-32768, 32767).astype(">i2") if c["bitpix"] == 16 else f.astype(">f4")
        elif entry == "stream":
            s["img"] = _pinned(img)
            s["next"] = _pinned(_frame(c, w, h, seed + 104729))
        elif entry == "background":
            s["img"], s["sub"] = img, torch.empty_like(img)
            nx, ny = sexgpu.background_meshes(w, h, c["back_size"])
            s["back"], s["sigma"] = torch.empty(ny, nx, device="cuda"), torch.empty(ny, nx, device="cuda")
        del img, wmap
    if entry in ("host", "fits"):
        s["tables"] = [np.zeros(_room(w, h), sexgpu.OBJECT_DTYPE)]
    elif entry == "stream":
        s["tables"] = [np.zeros(_room(w, h), sexgpu.OBJECT_DTYPE) for _ in range(2)]
    elif entry == "batch":
        s["tables"] = [np.zeros(_room(*f.shape), sexgpu.OBJECT_DTYPE) for f, _ in s["frames"]]
    if entry != "background":
        s["ctx"] = sexgpu.Context(0)
        s["ctx"].set_param("graph", c["graph"])
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return s


def _columns(rows):
    return {f: rows[f] for f in rows.dtype.names}


def run(state):
    s = state
    c, kw, ctx = s["case"], s["kw"], s.get("ctx")
    entry, w, h = c["entry"], c["w"], c["h"]
    if entry == "device":
        wmap = s["wmap"].data_ptr() if s["wmap"] is not None else None
        ctx.extract_device(s["img"].data_ptr(), w, h, wmap_ptr=wmap, **kw)
        n, rows = C.c_int(), s["rows"]
        rc = sexgpu.lib().sexgpu_copy_results(ctx.h, rows.ctypes.data_as(C.c_void_p), len(rows), C.byref(n), None, None,
                                              None)
        if rc != sexgpu.OK:
            raise RuntimeError("sexgpu_copy_results: %s" % sexgpu.ERRORS.get(rc, rc))
        out = _columns(rows)
        if c["naper"] > 1:
            a = s["apers"]
            rc = sexgpu.lib().sexgpu_copy_apertures(ctx.h, a.ctypes.data_as(C.POINTER(C.c_float)), len(a), None, None)
            if rc != sexgpu.OK:
                raise RuntimeError("sexgpu_copy_apertures: %s" % sexgpu.ERRORS.get(rc, rc))
            out["apertures"] = a
        return out
    if entry == "host":
        rows, seg, _ = ctx.extract(s["img"], weight=s["wmap"], **kw)
        return dict(_columns(_keep(s["tables"][0], rows)), segmentation=seg)
    if entry == "fits":
        zero = dict(bzero=32768.0) if c["bitpix"] == 16 else {}
        rows, seg, _ = ctx.extract_fits(s["data"], c["bitpix"], w, h, **zero, **kw)
        return dict(_columns(_keep(s["tables"][0], rows)), segmentation=seg)
    if entry == "stream":
        # two frames in flight: the second uploads while the first is extracted
        ctx.stream_submit(s["img"])
        ctx.stream_submit(s["next"])
        a, _ = ctx.stream_next(**kw)
        b, _ = ctx.stream_next(**kw)
        return [_keep(t, rows).view(np.uint8) for t, rows in zip(s["tables"], (a, b))]
    if entry == "batch":
        return [_keep(t, rows).view(np.uint8) for t, (rows, _) in zip(s["tables"], ctx.extract_batch(s["frames"]))]
    m = s["back"].numel()
    r = sexgpu.background_noalloc(s["img"].data_ptr(), s["sub"].data_ptr(), w, h, s["back"].data_ptr(),
                                  s["sigma"].data_ptr(), m, stream=torch.cuda.current_stream().cuda_stream, **kw)
    return [s["sub"], s["back"], s["sigma"], r.backmean, r.backsig, r.dthresh, r.thresh]


def work(case):
    c = case
    n = c["w"] * c["h"]
    if c["entry"] == "batch":
        n = sum((c["w"] // d) * (c["h"] // d) for d in ((1, 1, 2, 4) * 8)[:c["frames"]])
    elif c["entry"] == "stream":
        n *= 2
    rows = min(c["density"], 1 / 250) * n
    size = abs(c["bitpix"]) // 8 if c["entry"] == "fits" else 4
    read = n * size + (4 * n if c["weight"] in (1, 2, 3) else 0)
    if c["entry"] == "background":
        return {"bytes": read + 4 * n, "flops": 20 * n}
    write = rows * sexgpu.OBJECT_DTYPE.itemsize + (4 * n if c["entry"] in ("host", "fits") else 0)
    # the filter, and a few operations a pixel for the background and the sums
    return {"bytes": read + write, "flops": n * (2 * (c["taps"] or 7) ** 2 + 40)}


def exact(case, seed):
    """A catalogue is the outcome of thresholds, merges and cuts that are
    defined on 32-bit values (the objects themselves would differ in 64 bits),
    so no output has a 64-bit value to compare with."""
    return None
