"""An upload that fails half way leaves the context without a scene: no call
goes on with the last one, whose program may be gone from the device, and the
next upload that succeeds is all that it needs."""
import pytest

import interflect_b200 as ifx
from conftest import scene_src
from test_gpu_upload_memory import FullDevice, frame

pytestmark = pytest.mark.gpu


def many_objects():
    """A scene whose program takes 5 MB."""
    s = "render { width: 64, height: 64, surfels: 500, bounces: 4, exposure: 1.0 }\n"
    s += "camera { pos: [0, 1, 5], look: [0, 0, 0], up: [0, 1, 0], fov: 45 }\n"
    s += 'material "a" { albedo: [0.5, 0.5, 0.5], roughness: 0.5 }\n'
    s += "light { verts: [[-1, 9, -1], [1, 9, -1], [1, 9, 1], [-1, 9, 1]], emit: [5, 5, 5] }\n"
    for i in range(30000):
        s += f'sphere {{ center: [{i % 31}, {i // 31 % 31}, {i // 961}], radius: 0.2, mat: "a" }}\n'
    return s


def test_a_failed_upload_leaves_no_scene():
    scene, big = ifx.parse(scene_src("product")), ifx.parse(many_objects())
    with ifx.Context(0) as ctx:
        ctx.upload(scene)
        want = frame(ctx)
        with FullDevice(2 << 20):
            with pytest.raises(ifx.DeviceError, match="out of memory"):
                ctx.upload(big)
        for call in (lambda: ctx.frame(80, 60), lambda: ctx.render_frame(80, 60), lambda: ctx.generate(3000),
                     lambda: ctx.build(8), ctx.light_surfels, lambda: ctx.render_reference(8, 8, spp=1)):
            with pytest.raises(ifx.DeviceError, match="no scene uploaded"):
                call()
        with pytest.raises(ifx.DeviceError, match="no transfer"):
            ctx.solve(4)
        ctx.upload(scene)
        assert frame(ctx) == want
