"""Scenes without an object grid (a cone has no exact distance, and the linear
scan has no leaves) take kernels of their own: of three-node trees, of others,
and without the BVH, each also with counting kernels. Against the oracle: every
link and count exact, weights, radiosities, pixels and the path-traced film
within 1e-4 (the parity bar; expected bit-identical)."""
import pytest

import interflect_b200 as ifx
from pyoracle import Oracle
from test_gpu_edges import NCPU, rel_err, run_pipeline
from test_gpu_objgrid_forms import objects
from test_objgrid_check import KINDS

pytestmark = pytest.mark.gpu
CONE = '\ncone { a: [0.3, -0.9, 0.4], b: [0.2, 0.3, 0.5], radius: 0.35, radius_top: 0.1, mat: "a" }\n'
THREE = "\n".join(line for line in KINDS.splitlines() if not line.startswith(("capsule", "cylinder", "torus", "plane"))
                  and "round" not in line)
SCENES = {"three nodes": lambda: THREE + CONE, "kinds": lambda: KINDS + CONE,
          "120 objects": lambda: objects(120, 1.2, 0.1, 0.4) + CONE, "no cone": lambda: KINDS}


@pytest.mark.parametrize("name,bvh", [("three nodes", True), ("three nodes", False), ("kinds", True), ("kinds", False),
                                      ("120 objects", True), ("120 objects", False), ("no cone", False)])
def test_every_stage_equals_the_oracles(name, bvh):
    src = SCENES[name]()
    scene = ifx.parse(src)
    scene.set_use_bvh(bvh)
    assert (scene.info.bvh_nodes == 3) == (name == "three nodes")
    o = Oracle(src, threads=NCPU)
    o.set_use_bvh(bvh)
    with ifx.Context(0) as ctx:
        k, _ = run_pipeline(ctx, o, scene, 1500, 6, 5, 56, 40)
        assert k > 300
        film, _ = o.render(20, 14, "reference", spp=2)
        assert rel_err(ctx.render_reference(20, 14, 2)[0], film).max() <= 1e-4
        plain = ctx.frame(56, 40, cluster_res=6, max_bounces=5)
        ctx.set_work_counting(True)
        counted = ctx.frame(56, 40, cluster_res=6, max_bounces=5)
    assert plain["linear"].tobytes() == counted["linear"].tobytes()
    assert plain["transfer"] == counted["transfer"] and plain["shade_evals"] == counted["shade_evals"]
