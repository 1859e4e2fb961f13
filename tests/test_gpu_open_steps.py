"""Cone-shadow marches far outside the object grid. Steps are taken without a
query only where the rounding of a coordinate is known to be far below the
grid's margin, which is so inside the grid alone: between two tilted planes,
three million units away, a coordinate is good to a quarter, two steps. The transfer between surfels that a caller places there is the
traversal's, weight for weight and count for count."""
import numpy as np
import pytest

import interflect_b200 as ifx

pytestmark = pytest.mark.gpu
SCENE = """
render { width: 64, height: 64, surfels: 500, bounces: 4, exposure: 1.0 }
camera { pos: [0, 1, 5], look: [0, 0, 0], up: [0, 1, 0], fov: 45 }
material "a" { albedo: [0.5, 0.5, 0.5], roughness: 0.5 }
plane { normal: [0.6, 0.8, 0], height: -0.7, mat: "a" }
plane { normal: [-0.6, -0.8, 0], height: -0.7, mat: "a" }
sphere { center: [0, 0, 0], radius: 0.4, mat: "a" }
box { center: [0.7, 0, 0.3], size: [0.3, 0.3, 0.3], mat: "a" }
light { verts: [[-0.1, 0.6, -0.1], [0.1, 0.6, -0.1], [0.1, 0.6, 0.1], [-0.1, 0.6, 0.1]], emit: [5, 5, 5] }
"""


@pytest.mark.parametrize("away", [0.0, 3.0, 3e6])
def test_the_transfer_far_from_the_scene_is_the_traversals(away):
    rng = np.random.default_rng(5)
    n = 6000
    up = np.array([0.6, 0.8, 0.0])
    along, across = np.array([0.8, -0.6, 0.0]), np.array([0.0, 0.0, 1.0])
    # Surfels near one plane and, as the target that their marches approach, one near the other.
    p = (away * along + rng.uniform(-0.02, 0.02, (n, 1)) * along + rng.uniform(-0.02, 0.02, (n, 1)) * across
         + rng.uniform(0.1, 0.69, (n, 1)) * up)
    p[0] = away * along - 0.69 * up
    normal = np.tile(-up, (n, 1))
    normal[0] = up
    area = np.full(n, 1e-6)
    area[0] = 0.004
    got = {}
    for on in (True, False):
        with ifx.Context(0) as ctx:
            ctx.set_leaf_grid(on)
            ctx.upload(ifx.parse(SCENE))
            ctx.upload_surfels(p, normal, np.full((n, 3), 0.5), area)
            info = ctx.build(8)
            t, d = ctx.transfer(), ctx.row_diag()
            assert info.candidates >= n // 2
            got[on] = (info.candidates, info.links, info.evals, t["w"].tobytes(), t["idx"].tobytes(),
                       d["row_evals"].tobytes(), d["row_sum"].tobytes())
    assert got[True] == got[False]
