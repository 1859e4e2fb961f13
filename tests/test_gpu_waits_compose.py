"""A frame whose marching kernels gave up is not composed: the composition
reads materials and lights by the indices that those kernels leave with each
pixel, so it has to leave too. With no polls at all render_frame, on a context
that never rendered, and frame in a mode without GI (whose shading passes then
are the only ones) report the wait that ran out, the device film keeps the last
frame that was composed, and the context goes on as a fresh one would."""
import ctypes

import numpy as np
import pytest

import interflect_b200 as ifx
from conftest import scene_src

pytestmark = pytest.mark.gpu
W, H = 96, 72


def placed(ctx, scene):
    ctx.upload(scene)
    ctx.generate(3000)
    ctx.build(8)
    ctx.light_surfels()
    ctx.solve(16)
    ctx.grid_build()


def test_no_frame_is_composed_after_a_wait_ran_out():
    scene = ifx.parse(scene_src("product"))
    with ifx.Context(0) as ctx:
        placed(ctx, scene)
        ctx.set_wait_limit(0)
        with pytest.raises(ifx.WaitTimeout, match="bounded wait expired"):
            ctx.render_frame(W, H)
        for mode in ("direct", "normals"):
            with pytest.raises(ifx.WaitTimeout, match="bounded wait expired"):
                ctx.frame(W, H, mode=mode)
        ctx.set_wait_limit(None)
        lin, s8, ev = ctx.render_frame(W, H)
        # Another view, out of polls: the film is still the last one composed.
        ctx.set_wait_limit(0)
        cam = ifx.camera((3.0, 2.0, 6.0), (0.0, 0.9, 0.0))
        left, n = np.zeros_like(lin), ctypes.c_uint64()
        r = ifx.lib().ifx_render_frame(ctx._h, ctypes.byref(cam), ifx.MODES["beauty"], W, H, scene.cfg.exposure,
                                       left.ctypes.data_as(ctypes.c_void_p), None, ctypes.byref(n))
        assert r == ifx.IFX_ERR_TIMEOUT
        assert left.tobytes() == lin.tobytes()
        ctx.set_wait_limit(None)
        got = ctx.render_frame(W, H, cam=cam)
    with ifx.Context(0) as fresh:
        placed(fresh, scene)
        want = fresh.render_frame(W, H), fresh.render_frame(W, H, cam=cam)
    assert (lin.tobytes(), s8.tobytes(), ev) == (want[0][0].tobytes(), want[0][1].tobytes(), want[0][2])
    assert (got[0].tobytes(), got[1].tobytes(), got[2]) == (want[1][0].tobytes(), want[1][1].tobytes(), want[1][2])
