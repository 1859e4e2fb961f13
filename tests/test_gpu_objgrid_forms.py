"""The object grid in each of its forms changes no result: masks (up to 32
stored objects), lists of 12-bit objects with keys (up to 4,094) and of 16-bit
objects without (up to 32,768), on both sides of each line; cells with more
objects than a list holds; cameras inside the fine level, inside the coarse one
(eight times the scene's extent) and outside both. With the grid and without,
surfels, transfer, solve, frame and path-traced film are equal to the bit, and
so are all counts."""
import numpy as np
import pytest

import interflect_b200 as ifx
from test_objgrid_check import KINDS

pytestmark = pytest.mark.gpu
HEAD = """
render { width: 48, height: 36, surfels: 700, bounces: 6, exposure: 1.0 }
camera { pos: [0, 0.4, 3.5], look: [0, 0, 0], up: [0, 1, 0], fov: 55 }
material "a" { albedo: [0.5, 0.5, 0.5], roughness: 0.5 }
material "b" { albedo: [0.2, 0.5, 0.8], roughness: 0.2 }
plane { normal: [0, 1, 0], height: -1.4, mat: "a" }
light { verts: [[-1, 2, -1], [1, 2, -1], [1, 2, 1], [-1, 2, 1]], emit: [5, 5, 5] }
"""


def objects(count, half, low, high):
    """A plane and count - 1 spheres, boxes and tori of sizes [low, high] in [-half, half]^3."""
    rng = np.random.default_rng(count)
    out = []
    for i in range(count - 1):
        c = "[%.5g, %.5g, %.5g]" % tuple(rng.uniform(-half, half, 3))
        r, m = rng.uniform(low, high), "ab"[i % 2]
        out.append(['sphere { center: %s, radius: %.5g, mat: "%s" }' % (c, r, m),
                    'box { center: %s, size: [%.5g, %.5g, %.5g], mat: "%s" }' % (c, r, 2 * r, 1.5 * r, m),
                    'torus { center: %s, major: %.5g, minor: %.5g, mat: "%s" }' % (c, r, 0.3 * r, m)][i % 3])
    return HEAD + "\n".join(out) + "\n"


SCENES = {"kinds": lambda: KINDS, "32": lambda: objects(32, 1.2, 0.1, 0.4), "33": lambda: objects(33, 1.2, 0.1, 0.4),
          "crowded": lambda: objects(200, 0.5, 0.1, 0.5), "4094": lambda: objects(4094, 1.3, 0.01, 0.06),
          "4095": lambda: objects(4095, 1.3, 0.01, 0.06), "crowded 4500": lambda: objects(4500, 0.7, 0.05, 0.2),
          "32768": lambda: objects(32768, 1.3, 0.005, 0.03)}


def outputs(text, away, on):
    scene = ifx.parse(text)
    cam = ifx.camera((0.3 * away, 0.2 * away + 0.2, away), (0, 0, 0), fov=55 * 3.5 / away)
    with ifx.Context(0) as ctx:
        ctx.set_leaf_grid(on)
        ctx.upload(scene)
        n = ctx.generate(700)
        f = ctx.frame(48, 36, cluster_res=4, cam=cam)
        t, d, s = ctx.transfer(), ctx.row_diag(), ctx.surfels()
        lin, srgb, evals = ctx.render_frame(48, 36, cam=cam)[:3]
        ref = ctx.render_reference(24, 18, spp=2, cam=cam)
        counts = (n, f["transfer"].links, f["transfer"].evals, f["shade_evals"], evals, f["solve"].iterations)
        return counts, dict(frame=f["linear"], view=lin, srgb=srgb, film=np.asarray(ref[0]), idx=t["idx"], w=t["w"],
                            row_evals=d["row_evals"], **s)


@pytest.mark.parametrize("away", [3.5, 12.0, 28.0])
@pytest.mark.parametrize("name", SCENES)
def test_the_grid_changes_nothing(name, away):
    text = SCENES[name]()
    counts, with_grid = outputs(text, away, True)
    plain_counts, plain = outputs(text, away, False)
    assert counts == plain_counts and counts[0] > 100
    for k in plain:
        assert np.asarray(with_grid[k]).tobytes() == np.asarray(plain[k]).tobytes(), k
    assert with_grid["frame"].std() > 0
