"""Failure paths on the GPU, made without faulting or hanging the device.

Each device loop of the extraction (union-find walks and link retries of the
connected components and of the deblending, CLEAN's master chains) carries
an iteration cap; running out sets a device status word that the host reads,
and the entry point returns SEXGPU_ERR_LOOP.  The "loop_cap" execution
parameter lowers every cap so that a normal frame runs out of it (the
reference's own loops are unbounded: src/cuda/cudadetection.cu:610,
src/cuda/cudadeblend.cu:686).  Zero thresholds (src/back.c:196) and exact sums
beyond their range are reported the same way.  After each error the same
context extracts the next frame exactly as the oracle does.
"""
import numpy as np
import pytest

import synth
from oracle import oracle as O
from test_gpu_parity import compare_catalogs

pytestmark = pytest.mark.gpu


def _check_recovers(ctx, masks, seed):
    img = synth.frame_c0(seed=seed, w=512, h=400, nsrc=400)
    g, gseg, _ = ctx.extract(img, conv=masks["default"])
    o, oseg, _ = O.extract(img, conv=masks["default"])
    assert np.array_equal(gseg, oseg)
    compare_catalogs(g, o)


@pytest.mark.parametrize("cap", [1, 2])
def test_loop_cap_reports_and_context_recovers(gpu_ctx, masks, cap):
    img = synth.frame_c1(seed=71, w=640, h=512, nsrc=3000)
    gpu_ctx.set_param("loop_cap", cap)
    try:
        with pytest.raises(RuntimeError, match="device loop cap reached"):
            gpu_ctx.extract(img, conv=masks["gauss_2.5_5x5"])
    finally:
        gpu_ctx.set_param("loop_cap", 0)
    _check_recovers(gpu_ctx, masks, 72)


def test_loop_cap_rejects_negative(gpu_ctx):
    with pytest.raises(RuntimeError, match="bad argument"):
        gpu_ctx.set_param("loop_cap", -1)


def test_zero_threshold_reported(gpu_ctx, masks):
    """An absolute DETECT_THRESH of 0 gives a zero detection threshold,
    which the reference rejects (src/back.c:196)."""
    img = synth.frame_c0(seed=73, w=256, h=256, nsrc=50)
    with pytest.raises(RuntimeError, match="zero or negative threshold"):
        gpu_ctx.extract(img, conv=masks["default"], thresh_type=1, detect_thresh=0.0, analysis_thresh=0.0)
    _check_recovers(gpu_ctx, masks, 74)


def test_exact_sum_out_of_range_reported(gpu_ctx, masks):
    """One object whose pixels span more than 100 binary orders of magnitude
    (1e-28 ... 1e6 against an absolute threshold of 1e-30): its exact sums
    cannot hold the range, the entry point says so, and nothing is written
    outside the sums (the terms out of range are dropped, counted in the
    status)."""
    img = np.zeros((128, 160), np.float32)
    img[60:63, 70:73] = np.array([[1e-28, 1e-27, 1e-26], [1e-25, 1e6, 1e-24], [1e-23, 1e-22, 1e-21]], np.float32)
    with pytest.raises(RuntimeError, match="exact sum out of range"):
        gpu_ctx.extract(img, filter_flag=0, back_type=1, back_value=0.0, thresh_type=1, detect_thresh=1e-30,
                        analysis_thresh=1e-30)
    _check_recovers(gpu_ctx, masks, 75)


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("first", ["frame", "error", "background"])
def test_first_frames_of_a_context(masks, first, graph):
    """A context's first reads of the frame scalars go to pageable memory, later
    ones to a page of its own: counts, thresholds and errors are the same over
    its first frames, whichever call comes first."""
    import sexgpu
    img = synth.frame_c0(seed=76, w=200, h=150, nsrc=60)
    kw = dict(conv=masks["default"])
    o, oseg, os_ = O.extract(img, **kw)
    with sexgpu.Context(0) as ctx:
        ctx.set_param("graph", graph)
        if first == "error":
            with pytest.raises(RuntimeError, match="zero or negative threshold"):
                ctx.extract(img, thresh_type=1, detect_thresh=0.0, analysis_thresh=0.0, **kw)
        elif first == "background":
            for _ in range(5):
                got, want = ctx.background(img), O.background(img)
                assert np.array_equal(got[0], want[0]) and got[3].backsig == want[3].backsig
        for _ in range(4):
            g, gseg, gs = ctx.extract(img, **kw)
            assert np.array_equal(gseg, oseg)
            compare_catalogs(g, o)
            assert (gs.backmean, gs.dthresh, gs.nobj, gs.nraw, gs.npix_above) == \
                (os_.backmean, os_.dthresh, os_.nobj, os_.nraw, os_.npix_above)
        with pytest.raises(RuntimeError, match="zero or negative threshold"):
            ctx.extract(img, thresh_type=1, detect_thresh=0.0, analysis_thresh=0.0, **kw)


def _tile_frame(kind):
    """Objects each inside one 64 x 32 tile of the labelling (every label is one
    step from its root) and far apart (nothing to CLEAN).  single: cones, one
    peak each; ramps: pairs of peaks at the ends of long slopes, so that pixels
    are many steps from their peak; steps: rows of peaks, each higher than the
    one before and joined to it at a lower level, all other pixels next to a
    peak, so that only the walks over the joins are long."""
    img = np.zeros((96, 192), np.float32)
    for t in range(9):
        y, x = 16 + 32 * (t // 3), 64 * (t % 3) + 8
        if kind == "single":
            dy, dx = np.mgrid[-8:9, -8:9]
            img[y - 8:y + 9, x + 12:x + 29] = 400.0 * np.exp(-0.02 * (dx * dx + dy * dy) - 0.001 * dx - 0.002 * dy) + t
        elif kind == "ramps":
            slope = 10.0 + 20.0 * np.abs(np.arange(41) - 20.0 - 0.25 * t)
            img[y, x:x + 41] = slope
            img[y + 1, x:x + 41] = 0.5 * slope
        else:
            img[y - 1:y + 2, x - 1:x + 24] = 6.0 + 0.01 * np.arange(25)
            for k in range(8):
                img[y, x + 3 * k] = 100.0 * 2.0 ** k
                if k < 7:
                    img[y, x + 3 * k + 1:x + 3 * k + 3] = 90.0 * 0.7 ** k
    return img


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("cap", [1, 2])
@pytest.mark.parametrize("kind", ["ramps", "steps"])
def test_loop_cap_of_the_deblending(kind, cap, graph):
    """Only the deblending's walks run out: frames of single peaks pass under the
    cap, frames of joined peaks end with the error, in the plain form and in a
    replayed graph whose later stages run on zeroed counts, and the context
    then extracts either as the oracle does."""
    import sexgpu
    kw = dict(filter_flag=0, back_type=1, back_value=0.0, thresh_type=1, detect_thresh=5.0, analysis_thresh=5.0,
              deblend_nthresh=64, deblend_mincont=0.0)
    single, joined = _tile_frame("single"), _tile_frame(kind)

    def check(img):
        g, gseg, _ = ctx.extract(img, **kw)
        o, oseg, _ = O.extract(img, **kw)
        assert np.array_equal(gseg, oseg) and len(g) >= 9
        compare_catalogs(g, o)

    with sexgpu.Context(0) as ctx:
        ctx.set_param("graph", graph)
        ctx.set_param("loop_cap", cap)
        for turn in range(2):
            for _ in range(3):
                check(single)
            assert ctx.graph_stats()[0] == graph
            with pytest.raises(RuntimeError, match="device loop cap reached"):
                ctx.extract(joined, **kw)
        check(single)
        ctx.set_param("loop_cap", 0)
        for _ in range(3):
            check(joined)
        check(single)
