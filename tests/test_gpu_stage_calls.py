"""Calls that are no extraction leave the background of the last one alone.

sexgpu_background_map and sexgpu_background_rms give the maps "of the last
extraction".  sexgpu_filter and sexgpu_background on the same context, on
frames narrower, as wide and wider than the extraction's (so that any buffer
they shared would be overwritten, or outgrown and freed), must not change
them, in the plain form or after a captured graph.
"""
import numpy as np
import pytest

import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

W, H, BS = 500, 300, 32


def _filter(ctx, w, h):
    rng = np.random.default_rng(w)
    sub, m = rng.normal(0.0, 10.0, (h, w)).astype(np.float32), np.ones((5, 5), np.float32)
    assert np.array_equal(ctx.filter(sub, m), O.filter_image(sub, m))


def _background(ctx, w, h):
    img = synth.frame_c0(seed=w, w=w, h=h, nsrc=30)
    got, want = ctx.background(img, back_size=24), O.background(img, back_size=24)
    assert all(np.array_equal(a, b) for a, b in zip(got[:3], want[:3]))


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("absolute", [False, True])
@pytest.mark.parametrize("call", [_filter, _background])
def test_maps_are_those_of_the_last_extraction(call, absolute, graph):
    import sexgpu
    kw = dict(back_size=BS, back_type=1, back_value=1000.0) if absolute else dict(back_size=BS)
    img = synth.frame_c0(seed=41, w=W, h=H, nsrc=150)
    back, rms = O.background_map(img, **kw), O.background_rms(img, **kw)
    with sexgpu.Context(0) as ctx:
        ctx.set_param("graph", graph)
        for w, h in ((W, H), (W // 3, H), (20, 15), (W - 1, H // 2), (3 * W, H + 100), (4000, 64)):
            for _ in range(3 if graph else 1):
                ctx.extract(img, **kw)
            call(ctx, w, h)
            assert ctx.background_map(img.shape).tobytes() == back.tobytes(), (w, h)
            assert ctx.background_rms(img.shape).tobytes() == rms.tobytes(), (w, h)
            # once more without an extraction between them
            call(ctx, 2 * w, h)
            assert ctx.background_map(img.shape).tobytes() == back.tobytes(), (2 * w, h)
            assert ctx.background_rms(img.shape).tobytes() == rms.tobytes(), (2 * w, h)
