"""An upload that finds no memory for the object grid (18 MB of lists for a
scene of more than 32 objects) goes on without one, as the grid never changes a
result: the context then renders the new scene, not the new objects with what
the last scene chose (a three-node tree has kernels of its own)."""
import ctypes

import pytest

import interflect_b200 as ifx
from interflect_b200.scenes import gen_scenes

pytestmark = pytest.mark.gpu


class FullDevice:
    """The device's memory taken in ever smaller pieces, but for `left` bytes."""

    def __init__(self, left):
        self.left = left

    def __enter__(self):
        self.cu = ctypes.CDLL("libcuda.so.1")
        self.held = []
        spare = self.take(self.left)
        size = 1 << 37
        while size >= 1 << 21:
            p = self.take(size)
            if p is None:
                size //= 2
            else:
                self.held.append(p)
        assert spare is not None and self.held
        self.free(spare)
        return self

    def take(self, size):
        p = ctypes.c_uint64()
        return p if self.cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(size)) == 0 else None

    def free(self, p):
        assert self.cu.cuMemFree_v2(p) == 0

    def __exit__(self, *_):
        for p in self.held:
            self.free(p)


def frame(ctx):
    ctx.generate(3000)
    f = ctx.frame(80, 60)
    t = f["transfer"]
    return f["linear"].tobytes(), f["srgb"].tobytes(), t.links, t.evals, f["shade_evals"]


def test_a_scene_without_memory_for_its_grid_is_uploaded_without_one():
    three_nodes, deep = ifx.parse(gen_scenes.c2(False)), ifx.parse(gen_scenes.c3())
    assert (three_nodes.info.bvh_nodes, deep.info.bvh_nodes > 3) == (3, True)
    with ifx.Context(0) as fresh:
        fresh.upload(deep)
        want = frame(fresh)
    with ifx.Context(0) as ctx:
        ctx.upload(three_nodes)
        frame(ctx)
        with FullDevice(8 << 20):  # enough for a scene's arrays, not for its lists
            ctx.upload(deep)
        assert frame(ctx) == want
        ctx.upload(deep)  # with its grid
        assert frame(ctx) == want
