"""The packed frame where its solve changes: clusters of few members (summed by
threads) and of many (by warps), and more scenes than the 256 whose stop flags
a CTA keeps. Every scene is bit-identical to its own unbatched frame."""
import pytest

import interflect_b200 as ifx
from conftest import scene_src

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,surfels,res", [(3, 400, 8), (3, 4000, 2), (2, 4000, 4), (258, 60, 3)])
def test_every_scene_equals_its_unbatched_frame(count, surfels, res):
    src = [ifx.parse(scene_src(name)) for name in ("cornell", "product", "stress")]
    ctxs, want = [], []
    try:
        ms = ifx.MultiScene(0)
        for i in range(count):
            ctx = ifx.Context(0)
            ctxs.append(ctx)
            ctx.upload(src[i % 3])
            ctx.generate(surfels + i % 7)
            ctx.set_light_emission(ctx.light_emission() * (0.5 + 0.1 * (i % 11)))
            ctx.build(res)
            ctx.light_surfels()
            st = ctx.solve(3 + i % 5)
            ctx.grid_build()
            lin, srgb, _ = ctx.render_frame(24 + i % 3, 16)
            want.append((st.iterations, lin.tobytes(), srgb.tobytes()))
            ms.add(ctx, 24 + i % 3, 16, 3 + i % 5)
        ms.build(autotune=False)
        ms.run()
        for i in range(count):
            lin, srgb, st = ms.download(i)
            assert (st.iterations, lin.tobytes(), srgb.tobytes()) == want[i], i
        ms.close()
    finally:
        for ctx in ctxs:
            ctx.close()
