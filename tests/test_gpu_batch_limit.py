"""The batched solve at the number of clusters where its row kernel changes.
k_spmm_shared holds 16 right-hand sides of all clusters, 192 bytes each, beside
256 bytes a warp in 200 KiB: with the 32 warps of the default launch shape up
to 1,024 clusters. On both sides every right-hand side equals its own solve to
the bit."""
import numpy as np
import pytest

import interflect_b200 as ifx
from conftest import scene_src
from test_gpu_sell_wide import placed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [1023, 1024, 1025, 1056, 1057])
@pytest.mark.parametrize("rhs", [1, 15, 16, 17])
def test_each_right_hand_side_equals_its_own_solve(nc, rhs):
    n, rng = 5003, np.random.default_rng(nc + rhs)
    scene = ifx.parse(scene_src("cornell"))
    p, nrm = placed(scene, 9, nc, n, rng)
    starts = np.zeros(n + 1, np.uint32)
    starts[1:] = np.cumsum(rng.choice([0, 1, 15, 16, 17, 33, 70], n))
    w = rng.random(int(starts[-1]), np.float32) * np.float32(0.02)
    E = rng.random((rhs, n, 3), np.float32) ** 4
    with ifx.Context(0) as ctx:
        ctx.upload(scene)
        ctx.upload_surfels(p, nrm, rng.random((n, 3), np.float32), 0.5 + rng.random(n, np.float32))
        assert ctx.build_clusters(9) == nc
        ctx.upload_transfer(starts, rng.integers(0, nc, starts[-1]), w)
        rad, irr, it, out = ctx.solve_batched(E, 9)
        for r in {0, rhs // 2, rhs - 1}:
            ctx.set_emission(E[r])
            st = ctx.solve(9)
            s = ctx.surfels()
            assert (st.iterations, np.float32(st.residual)) == (it[r], out[r])
            assert s["rad"].tobytes() == rad[r].tobytes() and s["irr"].tobytes() == irr[r].tobytes()
