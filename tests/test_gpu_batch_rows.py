"""The batched solve's row kernels: up to 16 right-hand sides from shared
memory where the clusters fit it (at most 1,060), else from global memory. Every right-hand side must equal its
own solve to the bit, whichever runs."""
import numpy as np
import pytest

import interflect_b200 as ifx
from conftest import scene_src

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res,low,high", [(4, 1, 530), (9, 531, 1060), (16, 1061, 100000)])
@pytest.mark.parametrize("rhs", [1, 16, 17, 33])
def test_each_right_hand_side_equals_its_own_solve(res, low, high, rhs):
    with ifx.Context(0) as ctx:
        ctx.upload(ifx.parse(scene_src("cornell")))
        n = ctx.generate(4001)
        nc = ctx.build(res).clusters
        assert low <= nc <= high, nc
        E = np.random.default_rng(rhs).random((rhs, n, 3), np.float32) ** 4
        rad, irr, it, out = ctx.solve_batched(E, 9)
        for r in {0, rhs // 2, rhs - 1}:
            ctx.set_emission(E[r])
            st = ctx.solve(9)
            s = ctx.surfels()
            assert (st.iterations, np.float32(st.residual)) == (it[r], out[r])
            assert s["rad"].tobytes() == rad[r].tobytes() and s["irr"].tobytes() == irr[r].tobytes()
