"""GPU parity: libsexgpu (through its C ABI) against the CPU oracle.

Integer outputs (segmentation map, object set, NUMBER, ISOAREA, FLAGS, pixel
counts, positions of peaks) must be identical.  Float columns derived from
exact sums or from the same arithmetic must be identical too; the two double
sums the GPU reduces in a different order (position errors, FWHM fit) are held
to a relative tolerance of 1e-9 (RTOL_REORDERED), and the magnitudes, which go
through log10 (CUDA's on the GPU, glibc's in the oracle; they may differ by an
ulp), to 2 float ulps (RTOL_LOG).
"""
import numpy as np
import pytest

import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

RTOL_REORDERED = 1e-9
REORDERED = {"poserr_mx2", "poserr_my2", "poserr_mxy", "fwhm"}
RTOL_LOG = 2.5e-7
LOGCOLS = {"mag_iso", "mag_auto", "mag_aper"}
# CLASS_STAR goes through log10 and exp in double (CUDA's on the GPU, glibc's
# in the oracle) before its single rounding to float
ATOL_CLASS = 1e-6
CLASSCOLS = {"class_star"}


def compare_catalogs(g, o):
    assert len(g) == len(o), (len(g), len(o))
    bad = {}
    for name in g.dtype.names:
        a, b = g[name], o[name]
        if name in REORDERED:
            ok = np.isclose(a, b, rtol=RTOL_REORDERED, atol=1e-12) | (np.isnan(a) & np.isnan(b))
        elif name in LOGCOLS:
            ok = np.isclose(a, b, rtol=RTOL_LOG, atol=0)
        elif name in CLASSCOLS:
            ok = np.isclose(a, b, rtol=0, atol=ATOL_CLASS)
        else:
            ok = (a == b) | (np.isnan(a) & np.isnan(b)) if a.dtype.kind == "f" else (a == b)
        if ok.ndim > 1:
            ok = ok.all(axis=tuple(range(1, ok.ndim)))
        if not ok.all():
            i = int(np.nonzero(~ok)[0][0])
            bad[name] = (int((~ok).sum()), i, a[i], b[i])
    assert not bad, bad


def test_background_bitexact(gpu_ctx):
    img = synth.frame_c0(seed=5, w=512, h=384)
    for bs in (64, 50, 32):
        sub_g, back_g, sig_g, sg = gpu_ctx.background(img, back_size=bs)
        sub_o, back_o, sig_o, so = O.background(img, back_size=bs)
        assert np.array_equal(back_g, back_o)
        assert np.array_equal(sig_g, sig_o)
        assert sg.backmean == so.backmean and sg.backsig == so.backsig and sg.dthresh == so.dthresh
        assert np.array_equal(sub_g, sub_o)


@pytest.mark.parametrize("kind", ["poisson", "constant_meshes", "bimodal", "blanks", "spikes", "mesh_255",
                                  "mesh_256", "ragged"])
def test_background_histogram_shapes(gpu_ctx, kind):
    """Mesh histograms of unusual shapes: few distinct values (many pixels
    per bin), meshes of zero spread, two modes, blank pixels, a spike on a
    flat sky, meshes of 65025 pixels (the largest of the warp-per-mesh
    histogram) and of 65536 (the CTA-per-mesh form), ragged last meshes.
    Mesh modes and sigmas and the subtracted frame, bit for bit."""
    rng = np.random.default_rng(21)
    shape, bs = (384, 512), 64
    if kind == "poisson":
        img = rng.poisson(3.0, shape).astype(np.float32)
    elif kind == "constant_meshes":
        img = rng.normal(100, 5, shape).astype(np.float32)
        img[:128, :192] = 42.0
    elif kind == "bimodal":
        img = np.where(rng.random(shape) < 0.3, rng.normal(50, 2, shape), rng.normal(80, 3, shape)).astype(np.float32)
    elif kind == "blanks":
        img = rng.normal(300, 12, shape).astype(np.float32)
        img[rng.random(shape) < 0.2] = -1e30
    elif kind == "spikes":
        img = rng.normal(0, 1, shape).astype(np.float32)
        img[rng.random(shape) < 0.05] = 5e3
    elif kind in ("mesh_255", "mesh_256"):
        shape, bs = (600, 700), int(kind[-3:])
        img = rng.normal(200, 10, shape).astype(np.float32)
    else:
        shape, bs = (389, 517), 48
        img = rng.gamma(2.0, 30.0, shape).astype(np.float32)
    sub_g, back_g, sig_g, sg = gpu_ctx.background(img, back_size=bs)
    sub_o, back_o, sig_o, so = O.background(img, back_size=bs)
    assert np.array_equal(back_g, back_o)
    assert np.array_equal(sig_g, sig_o)
    assert sg.backmean == so.backmean and sg.backsig == so.backsig
    assert np.array_equal(sub_g, sub_o)


def test_filter_bitexact(gpu_ctx, masks):
    rng = np.random.default_rng(3)
    sub = rng.normal(0, 10, (300, 257)).astype(np.float32)
    for name in ("default", "gauss_2.5_5x5", "mexhat_2.5_7x7", "gauss_5.0_9x9"):
        m = masks[name]
        assert np.array_equal(gpu_ctx.filter(sub, m), O.filter_image(sub, m))


@pytest.mark.parametrize("seed", [0, 1])
def test_extract_c0(gpu_ctx, masks, seed):
    img = synth.frame_c0(seed=seed)
    kw = dict(conv=masks["default"])
    g, gseg, gs = gpu_ctx.extract(img, **kw)
    o, oseg, os_ = O.extract(img, **kw)
    assert gs.nraw == os_.nraw and gs.nraw_pix == os_.nraw_pix
    assert gs.ndetected == os_.ndetected
    assert np.array_equal(gseg, oseg)
    compare_catalogs(g, o)


def run_both(gpu_ctx, img, **kw):
    g, gseg, gs = gpu_ctx.extract(img, **kw)
    o, oseg, os_ = O.extract(img, **kw)
    assert (gs.nraw, gs.nraw_pix, gs.ndetected, gs.nobj) == (os_.nraw, os_.nraw_pix, os_.ndetected, os_.nobj)
    assert (gs.backmean, gs.backsig, gs.dthresh, gs.thresh) == (os_.backmean, os_.backsig, os_.dthresh, os_.thresh)
    assert gs.npix_above == os_.npix_above
    assert np.array_equal(gseg, oseg)
    compare_catalogs(g, o)
    return g


@pytest.mark.parametrize("w,h", [(7, 5), (64, 64), (333, 257), (1000, 37), (37, 700)])
def test_shapes(gpu_ctx, w, h):
    img = synth.frame_c0(seed=w * 7 + h, w=w, h=h, nsrc=max(1, w * h // 400))
    run_both(gpu_ctx, img)


def _blob(img, xc, yc, sigma, flux):
    h, w = img.shape
    y, x = np.mgrid[0:h, 0:w]
    img += (flux / (2 * np.pi * sigma ** 2) * np.exp(-((x - xc) ** 2 + (y - yc) ** 2) / (2 * sigma ** 2))).astype(np.float32)


def test_object_size_tiers_and_flux_range(gpu_ctx):
    """Raw objects of every size class (a few pixels, hundreds, ~2000,
    >4096) and point sources so bright (peak 2^29 and 2^32 x the detection
    threshold) that their branch fluxes come close to, or need more than,
    64 bits of fixed-scale sum."""
    img = synth.frame_c0(seed=91, w=700, h=600, nsrc=500)
    _blob(img, 150.0, 150.0, 25.0, 4e8)       # 34,000 pixels above threshold
    _blob(img, 160.0, 175.0, 4.0, 2e6)        # a knot inside it: deblended
    _blob(img, 450.0, 150.0, 7.0, 3e6)        # ~2000 pixels
    _blob(img, 465.0, 160.0, 3.0, 1e6)
    _blob(img, 300.0, 450.0, 0.7, 6e10)       # 178 pixels, peak 2^29 x threshold
    _blob(img, 560.0, 470.0, 1.2, 8e11)       # 367 pixels, peak 2^32 x threshold
    _blob(img, 566.0, 474.0, 1.2, 5e11)
    g = run_both(gpu_ctx, img)
    assert len(g) > 100


def test_crowded_king_field_precision_settings(gpu_ctx, masks):
    """The crowded-field precision form (DEBLEND_NTHRESH 64, DEBLEND_MINCONT
    0.0005, King-profile density) at a quarter of its size."""
    img = synth.frame_c2(seed=2001, w=1024, h=1024, nsrc=25000, rc=75.0, rt=500.0)
    g = run_both(gpu_ctx, img, conv=masks["gauss_2.5_5x5"], deblend_nthresh=64, deblend_mincont=0.0005)
    assert len(g) > 1000


def test_constant_frame_has_no_objects(gpu_ctx):
    img = np.full((200, 300), 1000.0, np.float32)
    g = run_both(gpu_ctx, img)
    assert len(g) == 0


def test_bad_pixels_and_nan(gpu_ctx):
    img = synth.frame_c0(seed=21, w=400, h=300, nsrc=300)
    img[:70, :130] = -1e30          # whole meshes unusable: nearest-mesh fill
    img[200:203, 50:60] = np.nan
    run_both(gpu_ctx, img)


@pytest.mark.parametrize("opts", [
    dict(deblend_nthresh=1), dict(clean_flag=0), dict(filter_flag=0),
    dict(back_type=1, back_value=1000.0), dict(thresh_type=1, detect_thresh=40.0, analysis_thresh=40.0),
    dict(numbering=1), dict(detect_minarea=1), dict(detect_minarea=3), dict(detect_minarea=12),
    dict(deblend_mincont=0.0), dict(deblend_mincont=1.0), dict(deblend_nthresh=64, deblend_mincont=0.0005),
    dict(clean_param=2.0), dict(gain=4.0), dict(mask_type=0), dict(back_filtersize=1),
    dict(back_filtersize=5, back_filtthresh=3.0), dict(satur_level=2000.0), dict(phot_aperture=12.0),
    dict(back_photo_type=1), dict(back_photo_type=1, back_photo_thick=6, gain=2.0, satur_level=3000.0),
])
def test_options(gpu_ctx, masks, opts):
    img = synth.frame_c0(seed=3, w=512, h=400, nsrc=700)
    run_both(gpu_ctx, img, **opts)


@pytest.mark.parametrize("mask", ["gauss_2.5_5x5", "mexhat_2.5_7x7", "gauss_4.0_7x7", "tophat_5.0_5x5"])
def test_masks_crowded(gpu_ctx, masks, mask):
    img = synth.frame_c1(seed=77, w=600, h=500, nsrc=3000)
    run_both(gpu_ctx, img, conv=masks[mask])


def test_repeatable(gpu_ctx, masks):
    img = synth.frame_c1(seed=78, w=700, h=600, nsrc=4000)
    a, sa, _ = gpu_ctx.extract(img, conv=masks["gauss_2.5_5x5"])
    b, sb, _ = gpu_ctx.extract(img, conv=masks["gauss_2.5_5x5"])
    assert a.tobytes() == b.tobytes() and np.array_equal(sa, sb)


def test_full_size_c1(gpu_ctx, masks):
    """The 4096^2 paper-scale frame: the whole catalogue and segmentation map
    against the oracle (about 10 s of CPU for the oracle)."""
    img = synth.frame_c1(seed=1000)
    g = run_both(gpu_ctx, img, conv=masks["gauss_2.5_5x5"])
    assert len(g) > 50000


@pytest.mark.parametrize("wtype", [1, 2, 3, 4])
def test_weight_maps(gpu_ctx, masks, wtype):
    """WEIGHT_TYPE MAP_VAR / MAP_RMS / MAP_WEIGHT: variance 1.0 +- 20% (x64),
    2% of the pixels unusable in 8x8 blocks; per-pixel thresholds against the
    local rms, per-object thresholds, variance-weighted errors."""
    img, vm = synth.frame_c1(seed=4001, w=768, h=640, density=9e-3, var=True)
    # 4: WEIGHT_TYPE BACKGROUND, the variance is the background rms map squared (no map given)
    wmap = {1: vm, 2: np.sqrt(vm), 3: np.where(vm < 1e29, 1.0 / vm, 0.0).astype(np.float32), 4: None}[wtype]
    kw = dict(conv=masks["gauss_4.0_7x7"], back_size=128, weight_type=wtype)
    g, gseg, gs = gpu_ctx.extract(img, weight=wmap, **kw)
    o, oseg, os_ = O.extract(img, weight=wmap, **kw)
    assert gs.sigfac == os_.sigfac
    assert (gs.nraw, gs.nraw_pix, gs.ndetected, gs.nobj) == (os_.nraw, os_.nraw_pix, os_.ndetected, os_.nobj)
    assert gs.npix_above == os_.npix_above
    assert np.array_equal(gseg, oseg)
    compare_catalogs(g, o)
    assert len(g) > 100 and g["dthresh"].min() < g["dthresh"].max()


def test_weight_map_absolute_thresholds(gpu_ctx, masks):
    img, vm = synth.frame_c1(seed=4002, w=512, h=512, density=8e-3, var=True)
    kw = dict(conv=masks["gauss_2.5_5x5"], weight_type=1, thresh_type=1, detect_thresh=30.0, analysis_thresh=30.0)
    g, gseg, gs = gpu_ctx.extract(img, weight=vm, **kw)
    o, oseg, os_ = O.extract(img, weight=vm, **kw)
    assert np.array_equal(gseg, oseg)
    compare_catalogs(g, o)


@pytest.mark.parametrize("warp_max,mask,weighted", [(1, "mexhat_2.5_7x7", False), (300, "gauss_2.5_5x5", False),
                                                    (1, "gauss_4.0_7x7", True)])
def test_kron_boxes_summed_by_blocks(masks, warp_max, mask, weighted):
    """AUTO photometry with the Kron boxes queued for whole thread blocks
    (kron_warp_max 1: every box; with more than 8192 survivors the queue
    overflows and the remaining boxes are summed by their warps; 300: a mix).
    The catalogue must not change."""
    import sexgpu
    with sexgpu.Context(0) as ctx:
        ctx.set_param("kron_warp_max", warp_max)
        kw = dict(conv=masks[mask])
        if weighted:
            img, vm = synth.frame_c1(seed=4003, w=768, h=640, density=9e-3, var=True)
            kw.update(weight=vm, weight_type=1, back_size=128)
        else:
            img = synth.frame_c1(seed=79, w=1700, h=1600, density=9e-3)
        g = run_both(ctx, img, **kw)
        assert len(g) > (100 if weighted else 8192)


def test_kron_param_rejects_bad_values(gpu_ctx):
    import sexgpu
    with pytest.raises(RuntimeError):
        gpu_ctx.set_param("kron_warp_max", 0)
    with pytest.raises(RuntimeError):
        gpu_ctx.set_param("no_such_parameter", 1)


def test_class_star(masks):
    """CLASS_STAR from a (seeded, synthetic) 10-10-1 network, against the
    oracle; without a network the column is 0 and nothing else changes."""
    import sexgpu
    from conftest import synthetic_nnw
    net = synthetic_nnw(5)
    img = synth.frame_c1(seed=81, w=900, h=800, nsrc=5000)
    kw = dict(conv=masks["gauss_2.5_5x5"], seeing_fwhm=1.1, pixel_scale=0.4)
    with sexgpu.Context(0) as ctx:
        g0, _, _ = ctx.extract(img, **kw)
        assert not g0["class_star"].any()
        ctx.set_nnw(sexgpu.NNW.from_arrays(*net))
        g, gseg, gs = ctx.extract(img, **kw)
    o, oseg, os_ = O.extract(img, nnw=O.NNW.from_arrays(*net), **kw)
    assert np.array_equal(gseg, oseg)
    compare_catalogs(g, o)
    cs = g["class_star"]
    assert len(g) > 500 and cs.std() > 0.01 and np.isfinite(cs).all()
    assert np.array_equal(g0["flux_auto"], g["flux_auto"])


@pytest.mark.parametrize("w,h,bs,fs", [(512, 384, 64, 3), (333, 257, 50, 5), (1000, 37, 64, 3), (300, 300, 32, 1)])
def test_background_rms_map(gpu_ctx, w, h, bs, fs):
    """BACKGROUND_RMS of the last extraction against the oracle, bit for bit."""
    img = synth.frame_c0(seed=15, w=w, h=h, nsrc=max(20, w * h // 800))
    gpu_ctx.extract(img, back_size=bs, back_filtersize=fs)
    g = gpu_ctx.background_rms(img.shape)
    o = O.background_rms(img, back_size=bs, back_filtersize=fs)
    assert g.tobytes() == o.tobytes()


@pytest.mark.parametrize("kw", [dict(back_size=64), dict(back_size=37, back_filtersize=5),
                                dict(back_size=40, back_type=1, back_value=1234.5)])
def test_background_map(gpu_ctx, masks, kw):
    """sexgpu_background_map: the background subtracted from every pixel (the
    BACKGROUND check image) against the oracle's, bit for bit."""
    img = synth.frame_c0(seed=8, w=500, h=350, nsrc=200)
    gpu_ctx.extract(img, conv=masks["default"], **kw)
    assert gpu_ctx.background_map(img.shape).tobytes() == O.background_map(img, **kw).tobytes()


@pytest.mark.parametrize("mask_type,gain", [(2, 0.0), (0, 3.0)])
def test_several_apertures(gpu_ctx, masks, mask_type, gain):
    """PHOT_APERTURES with several diameters (the reference allows one,
    src/define.h:50, src/cuda/cudaanalyse.cu:3363): every aperture of every
    row against the oracle; the row's FLUX_APER columns are the first."""
    img = synth.frame_c1(seed=23, w=900, h=700, nsrc=6000)
    aps = [1.5, 5.0, 8.5, 14.0, 30.0]
    kw = dict(conv=masks["gauss_2.5_5x5"], phot_apertures=aps, mask_type=mask_type, gain=gain,
              mag_zeropoint=25.0)
    g, gseg, _ = gpu_ctx.extract(img, **kw)
    ga = gpu_ctx.apertures()
    o, oseg, _ = O.extract(img, **kw)
    assert np.array_equal(gseg, oseg)
    compare_catalogs(g, o)
    oa = o["aper"][:, :len(aps), :]
    assert ga.shape == oa.shape == (len(g), len(aps), 4)
    for k in (0, 1, 3):  # flux, error, magnitude error
        assert ga[:, :, k].tobytes() == oa[:, :, k].tobytes(), k
    assert np.allclose(ga[:, :, 2], oa[:, :, 2], rtol=RTOL_LOG, atol=0)
    assert np.array_equal(ga[:, 0, 0], g["flux_aper"])
    # a wider aperture holds more flux on average
    assert (np.median(ga[:, 4, 0]) > np.median(ga[:, 1, 0]))


@pytest.mark.parametrize("peaks", [2, 31, 32, 33, 319, 320, 321, 1535, 1536, 1537, 5000])
@pytest.mark.parametrize("nthresh,mincont,minarea", [(32, 0.005, 5), (64, 0.0, 1), (2, 1e-4, 3)])
def test_deblending_by_number_of_peaks(gpu_ctx, peaks, nthresh, mincont, minarea):
    """One raw object with a given number of local maxima on either side of
    the sizes at which its merge tree goes to a warp, a block in shared memory
    or a block on global memory: bumps of random heights, three pixels apart, on
    a plateau of random saddles, beside a single bump and a flat-topped one."""
    rng = np.random.default_rng(peaks)
    nx = max(2, int(np.sqrt(peaks)))
    ny = -(-peaks // nx)
    img = np.zeros((3 * ny + 20, 3 * nx + 40), np.float32)
    img[2:3 * ny + 3, 2:3 * nx + 3] = rng.uniform(10.0, 12.0, (3 * ny + 1, 3 * nx + 1))
    tops = np.exp(rng.uniform(np.log(13.0), np.log(2e4), nx * ny)).astype(np.float32)
    for k in range(peaks):
        y, x = 4 + 3 * (k // nx), 4 + 3 * (k % nx)
        img[y - 1:y + 2, x - 1:x + 2] += tops[k] * rng.uniform(0.05, 0.9, (3, 3)).astype(np.float32)
        img[y, x] = 13.0 + 2.0 * tops[k]
    img[3 * ny + 8:3 * ny + 13, 5:10] = 50.0
    img[3 * ny + 10, 7] = 90.0
    img[3 * ny + 8:3 * ny + 14, 20:27] = 40.0
    g = run_both(gpu_ctx, img, filter_flag=0, back_type=1, back_value=0.0, thresh_type=1, detect_thresh=5.0,
                 analysis_thresh=5.0, deblend_nthresh=nthresh, deblend_mincont=mincont, detect_minarea=minarea,
                 clean_flag=0)
    assert len(g) >= 3


@pytest.mark.parametrize("kind", ["halves", "eighths", "zero_mean", "wide", "growing", "tiny", "inf", "mostly_blank",
                                  "integers"])
@pytest.mark.parametrize("shape,bs", [((200, 333), 37), ((300, 516), 128), ((64, 64), 64), ((640, 700), 300),
                                      ((9, 2000), 1024)])
def test_background_sums_round_like_the_sequence(gpu_ctx, kind, shape, bs):
    """The mesh sums are cut into stretches and composed; every rounding of the
    reference's pixel-by-pixel sums has to come out: squares that tie half way
    between two doubles (values with few bits), sums that jump over binades
    inside a stretch, sums of both signs, pixels whose sum is not exact,
    infinities, blanks.  Bit for bit, with ragged meshes and meshes above 65535
    pixels."""
    rng = np.random.default_rng(len(kind) * 1000 + bs)
    n = rng.normal(0.0, 1.0, shape)
    if kind == "halves":
        img = np.round(2 * (1000.5 + 40 * n)) / 2 + 2.0 ** -13
    elif kind == "eighths":
        img = np.round(8 * (90000.0 + 3000 * n)) / 8
    elif kind == "zero_mean":
        img = 8.0 * n
    elif kind == "wide":
        img = np.exp(rng.uniform(-25, 25, shape))
    elif kind == "growing":
        img = np.exp(np.linspace(-20, 40, n.size)).reshape(shape) * (1 + 0.01 * n)
    elif kind == "tiny":
        img = 1e-42 * (1.0 + n * n) + np.where(n > 2, 1e-20, 0.0)
    elif kind == "inf":
        img = 100.0 + n
        img[shape[0] // 2, ::71] = np.inf
    elif kind == "mostly_blank":
        img = np.where(rng.random(shape) < 0.47, -1e30, 500.0 + 20 * n)
    else:
        img = np.rint(30000.0 + 200 * n)
    img = img.astype(np.float32)
    with np.errstate(all="ignore"):
        sub_o, back_o, sig_o, so = O.background(img, back_size=bs)
    sub_g, back_g, sig_g, sg = gpu_ctx.background(img, back_size=bs)
    assert np.array_equal(back_g, back_o, equal_nan=True)
    assert np.array_equal(sig_g, sig_o, equal_nan=True)
    assert np.array_equal([sg.backmean, sg.backsig], [so.backmean, so.backsig], equal_nan=True)


@pytest.mark.parametrize("w,h,bs", [(70, 1600, 2), (1600, 70, 2), (1536, 40, 2), (33, 1540, 2), (64, 64, 64), (3, 90, 2)])
def test_background_splines_long_and_short(gpu_ctx, w, h, bs):
    """Mesh grids on either side of the longest line whose spline is kept on
    chip (768 meshes), one mesh, two meshes: background and rms maps."""
    img = synth.frame_c0(seed=31, w=w, h=h, nsrc=20)
    gpu_ctx.extract(img, back_size=bs)
    assert gpu_ctx.background_map(img.shape).tobytes() == O.background_map(img, back_size=bs).tobytes()
    assert gpu_ctx.background_rms(img.shape).tobytes() == O.background_rms(img, back_size=bs).tobytes()


@pytest.mark.parametrize("w,h,minarea", [(1031, 517, 1), (64, 3000, 5), (3000, 64, 5), (2048, 2048, 5)])
def test_lists_and_catalogue_order(gpu_ctx, w, h, minarea):
    """Object pixel lists read from boxes of one pixel up to boxes cut into
    bands of rows (a frame-wide object with a deblended chain of knots, objects
    inside its box), and the completion order over many raw objects of one row:
    completion and first-pixel numbering against the oracle, CLEAN on."""
    rng = np.random.default_rng(w + h)
    img = rng.normal(0.0, 1.0, (h, w)).astype(np.float32)
    t = np.arange(max(w, h) * 2)
    x = np.clip((w - 1) * t / (t.size - 1), 0, w - 1).astype(int)
    y = np.clip((h - 1) * (0.5 + 0.45 * np.sin(9.0 * t / t.size)), 0, h - 1).astype(int)
    for d in range(-2, 3):
        img[np.clip(y + d, 0, h - 1), x] = np.maximum(img[np.clip(y + d, 0, h - 1), x], 30.0 - 4 * abs(d))
    for k in range(0, t.size, max(1, t.size // 40)):
        _blob(img, float(x[k]), float(y[k]), 1.5, float(rng.uniform(300, 9000)))
    img[h // 3, 1::7] += 40.0
    for numbering in (0, 1):
        g = run_both(gpu_ctx, img, filter_flag=0, back_type=1, back_value=0.0, thresh_type=1, detect_thresh=3.2,
                     analysis_thresh=3.2, detect_minarea=minarea, numbering=numbering, deblend_mincont=0.001)
        assert len(g) > 10


@pytest.mark.parametrize("w,h", [(1, 1), (3, 2), (63, 33), (64, 32), (65, 31), (68, 36), (132, 97), (257, 65)])
@pytest.mark.parametrize("mw,mh", [(1, 1), (3, 3), (5, 5), (7, 7), (9, 9), (11, 11), (4, 6), (2, 1), (31, 31)])
def test_filter_at_tile_edges(gpu_ctx, w, h, mw, mh):
    """Frames of one tile, of whole tiles and just beyond, with rows that are
    and are not a multiple of 16 bytes, under every specialised mask size, even
    sizes and the largest mask: bit for bit."""
    rng = np.random.default_rng(100 * w + mw)
    sub = rng.normal(0, 10, (h, w)).astype(np.float32)
    m = rng.uniform(-0.2, 1.0, (mh, mw)).astype(np.float32)
    assert np.array_equal(gpu_ctx.filter(sub, m), O.filter_image(sub, m))


@pytest.mark.parametrize("w,h", [(7, 5), (63, 33), (64, 32), (65, 31), (68, 36), (132, 97), (257, 65)])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("bs,thr", [(3, 0.3), (64, 0.1), (40, 1.5)])
def test_components_at_tile_edges(gpu_ctx, masks, w, h, weighted, bs, thr):
    """Noise cut near its mean, so that components wind through the tiles and
    over their borders, with meshes narrower than four pixels (more spline
    segments than a tile row has staged nodes) and wider than a tile; with and
    without a variance map that marks unusable pixels."""
    rng = np.random.default_rng(w * 1000 + h + bs)
    img = rng.normal(100.0, 10.0, (h, w)).astype(np.float32)
    kw = dict(back_size=bs, filter_flag=0, detect_thresh=thr, analysis_thresh=thr, detect_minarea=1,
              deblend_nthresh=4, deblend_mincont=0.5, clean_flag=0)
    if weighted:
        var = rng.uniform(50.0, 150.0, (h, w)).astype(np.float32)
        var[rng.random((h, w)) < 0.05] = 1e30
        g, gseg, gs = gpu_ctx.extract(img, weight=var, weight_type=1, **kw)
        o, oseg, os_ = O.extract(img, weight=var, weight_type=1, **kw)
        assert gs.npix_above == os_.npix_above
        assert np.array_equal(gseg, oseg)
        compare_catalogs(g, o)
    else:
        run_both(gpu_ctx, img, **kw)


@pytest.mark.parametrize("w,h,nsrc", [(64, 48, 0), (333, 257, 60), (1024, 700, 900)])
def test_results_sized_by_count(gpu_ctx, w, h, nsrc):
    """Rows and maps that are fetched after the extraction into arrays of their
    size are those of the one-call form; a limit of exactly the rows is enough,
    one less is an error."""
    import ctypes as C

    import sexgpu
    img = synth.frame_c0(seed=w + nsrc, w=w, h=h, nsrc=nsrc) if nsrc else np.full((h, w), 7.0, np.float32)
    g, gseg, gs, sub, cd = gpu_ctx.extract(img, want_maps=True)
    cfg, n = sexgpu.make_config(), C.c_int()
    rows, seg = np.zeros(len(g) + 3, sexgpu.OBJECT_DTYPE), np.zeros((h, w), np.int32)
    sub1, cd1 = np.zeros((h, w), np.float32), np.zeros((h, w), np.float32)
    f = [a.ctypes.data_as(C.POINTER(C.c_float)) for a in (img, sub1, cd1)]
    assert sexgpu.lib().sexgpu_extract(gpu_ctx.h, f[0], None, w, h, C.byref(cfg), rows.ctypes.data_as(C.c_void_p),
                                       len(rows), C.byref(n), seg.ctypes.data_as(C.c_void_p), f[1], f[2],
                                       None) == sexgpu.OK
    assert n.value == len(g) == gs.nobj
    assert np.array_equal(rows[:len(g)].view(np.uint8), g.view(np.uint8)) and not rows[len(g):].view(np.uint8).any()
    assert np.array_equal(seg, gseg) and np.array_equal(sub1, sub) and np.array_equal(cd1, cd)
    assert len(gpu_ctx.extract(img, max_objects=len(g))[0]) == len(g)
    if len(g):
        with pytest.raises(RuntimeError):
            gpu_ctx.extract(img, max_objects=len(g) - 1)


@pytest.mark.parametrize("w,h,bs", [(333, 140, 37), (520, 300, 256), (512, 130, 128), (260, 64, 64)])
@pytest.mark.parametrize("wtype", [1, 3])
@pytest.mark.parametrize("spread", [0.1, 9.0])
def test_weight_scale_of_meshes(gpu_ctx, w, h, bs, wtype, spread):
    """The mean relative variance of a mesh is its exact sum rounded once, for
    rows that are and are not a multiple of 16 bytes, meshes of more pixels than
    the double bins hold, variances over more binades than they span, and meshes
    of mostly unusable pixels."""
    rng = np.random.default_rng(w + bs + wtype)
    img = rng.normal(300.0, 10.0, (h, w)).astype(np.float32)
    wmap = np.exp(rng.normal(0.0, spread, (h, w))).clip(1e-6, 1e12).astype(np.float32)
    bad = 1e30 if wtype == 1 else 0.0
    wmap[rng.random((h, w)) < 0.1] = bad
    wmap[: h // 3, : w // 2][rng.random((h // 3, w // 2)) < 0.6] = bad
    kw = dict(back_size=bs, weight_type=wtype, filter_flag=0, detect_thresh=3.0, analysis_thresh=3.0)
    _, gseg, gs = gpu_ctx.extract(img, weight=wmap, **kw)
    _, oseg, os_ = O.extract(img, weight=wmap, **kw)
    assert gs.sigfac == os_.sigfac and gs.npix_above == os_.npix_above
    assert np.array_equal(gseg, oseg)


@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 1), (31, 1), (1, 33), (32, 32), (41, 25), (255, 3), (64, 64), (241, 17)])
@pytest.mark.parametrize("flat", [0.0, 0.3, 0.7])
def test_medians_of_mesh_maps(gpu_ctx, nx, ny, flat):
    """Medians over mesh counts on either side of whole warps and blocks and of
    the count up to which they are taken beside the row nodes, with meshes of no
    scatter (of which more than half send the rms to the positive ones), and
    rows of nodes of any length: bit for bit."""
    rng = np.random.default_rng(1000 * nx + ny)
    img = rng.normal(500.0, 10.0, (8 * ny, 8 * nx)).astype(np.float32)
    for k in np.flatnonzero(rng.random(nx * ny) < flat):
        y, x = 8 * (k // nx), 8 * (k % nx)
        img[y:y + 8, x:x + 8] = rng.integers(480, 520)
    got, want = gpu_ctx.background(img, back_size=8, back_filtersize=1), O.background(img, back_size=8, back_filtersize=1)
    assert all(np.array_equal(a, b) for a, b in zip(got[:3], want[:3]))
    assert (got[3].backmean, got[3].backsig) == (want[3].backmean, want[3].backsig)


@pytest.mark.parametrize("w,h", [(5, 37), (36, 13), (103, 81), (322, 171)])
@pytest.mark.parametrize("weight_type", [1, 2, 4])
@pytest.mark.parametrize("minarea", [1, 5, 30])
def test_objects_of_zero_variance(gpu_ctx, masks, w, h, weight_type, minarea):
    """Where the variance is 0 the threshold is, and objects may have filtered
    values of 0 only: their peak is their first pixel all the same."""
    rng = np.random.default_rng(w + minarea)
    img = np.full((h, w), 137.0, np.float32)
    img[rng.random((h, w)) < 0.02] = -1e30
    kw = dict(back_size=64, conv=masks["default"], detect_thresh=1.5, analysis_thresh=1.5, detect_minarea=minarea,
              deblend_nthresh=8, weight_type=weight_type)
    if weight_type != 4:
        kw["weight"] = np.where(rng.random((h, w)) < 0.3, 0.0, 25.0).astype(np.float32)
    g, gseg, gs = gpu_ctx.extract(img, **kw)
    o, oseg, os_ = O.extract(img, **kw)
    assert np.array_equal(gseg, oseg) and gs.nraw == os_.nraw
    compare_catalogs(g, o)


@pytest.mark.parametrize("w,h,mask", [(97, 244, "mexhat_4.0_9x9"), (322, 515, "mexhat_5.0_11x11"),
                                      (720, 198, "mexhat_5.0_11x11")])
@pytest.mark.parametrize("nthresh,mincont", [(2, 0.1), (8, 0.005), (32, 0.005), (64, 0.0001), (32, 1.0)])
def test_deblending_far_above_the_threshold(gpu_ctx, masks, w, h, mask, nthresh, mincont):
    """Under a mask with negative taps blank pixels (-1e30) leave filtered values
    90 binary orders above the threshold; thousands of them add up to branch
    fluxes of more than 127 bits in units of the threshold's last bit, which the
    MINCONT cut has to get right all the same."""
    rng = np.random.default_rng(w)
    img = rng.normal(1000.0, 10.0, (h, w)).astype(np.float32)
    img[rng.random((h, w)) < 0.025] = -1e30
    g = run_both(gpu_ctx, img, conv=masks[mask], deblend_nthresh=nthresh, deblend_mincont=mincont)
    assert g["fdpeak"].max() > 1e28


@pytest.mark.parametrize("length,bits,bright", [(60, 84, 12), (60, 88, 3), (60, 86, 25), (60, 94, 2), (200, 80, 12),
                                                (200, 80, 40), (200, 82, 60), (200, 88, 40), (700, 76, 40), (700, 78, 200),
                                                (700, 84, 3)])
def test_sums_far_above_the_threshold(gpu_ctx, length, bits, bright):
    """A bar with some pixels 2^bits above the others.  Its moments are exact sums
    (math.fsum) where no term lies more than 101 binary orders above another,
    though all together need more than the 126 bits that partial sums have and
    would fit or not with the order of the pixels; where the oracle's 127 bits
    hold them, every column is the oracle's.  Terms further apart are reported."""
    import math
    rng = np.random.default_rng(length + bits + bright)
    img = np.zeros((64, length + 60), np.float32)
    img[30:33, 30:30 + length] = rng.uniform(6, 20, (3, length))
    img[24:30, 40:46] = rng.uniform(6, 20, (6, 6))
    img[31, 30 + length - 1 - 2 * np.arange(bright)] = 2.0 ** bits * rng.uniform(6, 20, bright)
    kw = dict(filter_flag=0, back_type=1, back_value=0.0, thresh_type=1, detect_thresh=5.0, analysis_thresh=5.0)
    yy, xx = np.nonzero(img)
    v, x, y = img[yy, xx], (xx - 30).astype(np.float32), (yy - 24).astype(np.float32)
    terms = [t[t > 0].astype(np.float64) for t in (v, v * x, v * y, v * x * x, v * y * y, v * x * y)]
    total, mx, my = (math.fsum(t) for t in terms[:3])
    rv = float(np.float32(total))
    span = max(int(np.ptp(np.frexp(t)[1])) for t in terms)
    need = max(math.fsum(t) / 2.0 ** (np.frexp(t)[1].min() - 24) for t in terms)
    for _ in range(3):
        if span > 101:
            with pytest.raises(RuntimeError, match="exact sum out of range"):
                gpu_ctx.extract(img, **kw)
            continue
        g, _, _ = gpu_ctx.extract(img, **kw)
        assert len(g) == 1
        assert (g["fdflux"][0], g["dflux"][0], g["flux"][0]) == (np.float32(total),) * 3
        assert (g["mx"][0], g["my"][0]) == (mx / rv + 30, my / rv + 24)
        if need < 2.0 ** 126:
            compare_catalogs(g, O.extract(img, **kw)[0])
