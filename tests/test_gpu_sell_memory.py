"""A transfer whose sliced copy finds no memory is solved from its CSR rows. One
row of 65,600 links among 70,000 of 400: padded to their longest, the slices of
such a matrix would pass 2^32 entries, but sorted by length they take little
more than the links. Without memory for them the results are the same."""
import numpy as np
import pytest

import interflect_b200 as ifx
from conftest import scene_src
from test_gpu_upload_memory import FullDevice

pytestmark = pytest.mark.gpu


def test_a_transfer_without_memory_for_its_copy_is_solved():
    n = 70000
    rng = np.random.default_rng(5)
    scene = ifx.parse(scene_src("cornell"))
    lo, hi = np.array(scene.info.bounds_lo, np.float32), np.array(scene.info.bounds_hi, np.float32)
    nrm = np.eye(3, dtype=np.float32)[rng.integers(0, 3, n)]
    p, albedo = lo + rng.random((n, 3), np.float32) * (hi - lo), rng.random((n, 3), np.float32)
    e, area = rng.random((n, 3), np.float32), 0.5 + rng.random(n, np.float32)
    length = np.full(n, 400)
    length[n // 3] = 65600
    starts = np.zeros(n + 1, np.uint32)
    starts[1:] = np.cumsum(length)
    links = int(starts[-1])
    w = rng.random(links, np.float32) * (0.8 / 400)
    w[starts[n // 3]:starts[n // 3 + 1]] *= 400 / 65600
    out = []
    with ifx.Context(0) as ctx, ifx.Context(0) as full:
        for c in (ctx, full):
            c.upload(scene)
            c.upload_surfels(p, nrm, albedo, area)
            c.set_emission(e)
            nc = c.build_clusters(8)
        idx = rng.integers(0, nc, links).astype(np.uint32)
        ctx.upload_transfer(starts, idx, w)
        with FullDevice(320 << 20):  # 225 MB of rows, 243 MB of slices
            full.upload_transfer(starts, idx, w)
            out.append(full.solve(3))
        rows = full.surfels()
        out.append(ctx.solve(3))
        full.set_emission(e)
        full.upload_transfer(starts, idx, w)  # with its copy
        out.append(full.solve(3))
        slices, again = ctx.surfels(), full.surfels()
    for k in ("rad", "irr"):
        assert rows[k].tobytes() == slices[k].tobytes() == again[k].tobytes()
    assert out[0] == out[1] == out[2] and out[0].iterations == 3
