"""Surfels read back, few of them and many, and while the device has no memory
left for the arrays packed to the caller's layout: the same values as with it."""
import numpy as np
import pytest

import interflect_b200 as ifx
from conftest import scene_src
from test_gpu_upload_memory import FullDevice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1024, 1025])
def test_few_surfels_are_read_back(n):
    rng = np.random.default_rng(n)
    p, nrm, albedo, e = (rng.random((n, 3), np.float32) for _ in range(4))
    area = rng.random(n, np.float32)
    with ifx.Context(0) as ctx:
        ctx.upload(ifx.parse(scene_src("cornell")))
        ctx.upload_surfels(p, nrm, albedo, area)
        ctx.set_emission(e)
        s = ctx.surfels()
    for k, v in dict(p=p, n=nrm, albedo=albedo, area=area, direct=e, rad=e, irr=np.zeros_like(e)).items():
        assert s[k].tobytes() == v.tobytes(), k


@pytest.mark.parametrize("n", [60001, 49 * 2048])
def test_surfels_are_read_back_without_memory(n):
    rng = np.random.default_rng(n)
    p, nrm, albedo, e = (rng.random((n, 3), np.float32) for _ in range(4))
    area = rng.random(n, np.float32)
    with ifx.Context(0) as ctx, ifx.Context(0) as full:
        for c in (ctx, full):
            c.upload(ifx.parse(scene_src("cornell")))
            c.upload_surfels(p, nrm, albedo, area)
            c.set_emission(e)
        want = ctx.surfels()
        with FullDevice(1 << 20):
            got = full.surfels()
        again = full.surfels()
    assert want["p"].tobytes() == p.tobytes() and want["area"].tobytes() == area.tobytes()
    assert want["direct"].tobytes() == e.tobytes()
    for k in want:
        assert got[k].tobytes() == want[k].tobytes() == again[k].tobytes(), k
