"""Surfels read back while the device has no memory left for the arrays packed
to the caller's layout: the same values as with memory."""
import numpy as np
import pytest

import interflect_b200 as ifx
from conftest import scene_src
from test_gpu_upload_memory import FullDevice

pytestmark = pytest.mark.gpu


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
