"""The object grid's rules (csrc/objgrid.h) on the CPU: tests/cpp/objgrid_check
forms the cells' lists over the oracle's objects and requires every answer the
rules accept, at points throughout the scene, at its surfaces and along
marches, to be the oracle's traversal's, distance bits and material. The
scenes cover every admitted primitive kind, hard and smooth subtractions,
planes, overlapping and touching objects and trees of one to hundreds of
nodes; each at a coarse grid (long lists) and a fine one."""
import os
import subprocess

import pytest

from conftest import ROOT

SRCS = ["scene.cpp", "gi.cpp", "render.cpp", "diff.cpp"]
KINDS = """
render { width: 64, height: 64, surfels: 500, bounces: 4, exposure: 1.0 }
camera { pos: [0, 1, 5], look: [0, 0, 0], up: [0, 1, 0], fov: 45 }
material "a" { albedo: [0.5, 0.5, 0.5], roughness: 0.5 }
material "b" { albedo: [0.2, 0.5, 0.8], roughness: 0.5 }
plane { normal: [0, 1, 0], height: -1, mat: "a" }
box { center: [-1, -0.5, 0], size: [1, 1, 1], mat: "b" }
box { center: [0, -0.5, 0], size: [1, 1, 1], round: 0.2, mat: "a" }
box { center: [1.2, -0.4, 0.4], size: [0.6, 1.2, 0.6], rotate_y: 30, mat: "b" }
sphere { center: [0.1, 0.3, 0.1], radius: 0.5, mat: "b", subtract_sphere: [[0.1, 0.6, 0.1], 0.4] }
sphere { center: [-1.2, 0.5, 0.6], radius: 0.5, mat: "a", subtract_cylinder: [[-2, 0.5, 0.6], [0, 0.5, 0.6], 0.2], smooth: 0.1 }
torus { center: [0.9, 0.4, -0.9], major: 0.5, minor: 0.2, mat: "a" }
capsule { a: [-0.5, -0.8, 1.1], b: [0.6, 0.2, 1.3], radius: 0.2, mat: "b" }
cylinder { a: [-1.3, -1.0, -1.2], b: [-0.9, 0.4, -1.0], radius: 0.25, mat: "a" }
light { verts: [[-1, 2, -1], [1, 2, -1], [1, 2, 1], [-1, 2, 1]], emit: [5, 5, 5] }
"""
SCENES = ["interflect_b200/scenes/c1_cornell.rad", "interflect_b200/scenes/c2_product.rad",
          "interflect_b200/scenes/c3_stress.rad", "tests/golden/scenes/product.rad",
          "tests/golden/scenes/stress.rad", "tests/golden/scenes/minimal.rad", "kinds"]


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("objgrid") / "objgrid_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "oracle"), "-o", out,
                    os.path.join(ROOT, "tests", "cpp", "objgrid_check.cpp")] +
                   [os.path.join(ROOT, "oracle", s) for s in SRCS] + ["-lpthread"], check=True)
    return out


@pytest.mark.parametrize("cells", ["9", "64"])
@pytest.mark.parametrize("scene", SCENES)
def test_accepted_answers_equal_the_reference_traversal(exe, tmp_path, scene, cells):
    path = os.path.join(ROOT, scene)
    if scene == "kinds":
        path = str(tmp_path / "kinds.rad")
        with open(path, "w") as f:
            f.write(KINDS)
    r = subprocess.run([exe, path, cells], capture_output=True, text=True, timeout=600)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "every accepted answer equals the reference traversal" in r.stdout
