"""The batched solve where its row kernel changes. k_spmm_shared holds 16
right-hand sides of all clusters, 192 bytes each, beside 256 bytes a warp in
200 KiB: with the 32 warps of the default launch shape up to 1,024 clusters. It
takes matrices of 32 links a row in the mean or 2^19 in all, and of 60 a row
where rows times right-hand sides pass 1,250,000. On both sides of each line
every right-hand side equals its own solve to the bit."""
import numpy as np
import pytest

import interflect_b200 as ifx
from conftest import scene_src
from test_gpu_sell_wide import placed

pytestmark = pytest.mark.gpu


def check(n, nc, length, rhs, bounces):
    rng = np.random.default_rng(n + nc + rhs)
    scene = ifx.parse(scene_src("cornell"))
    p, nrm = placed(scene, 9, nc, n, rng)
    starts = np.zeros(n + 1, np.uint32)
    starts[1:] = np.cumsum(length)
    w = rng.random(int(starts[-1]), np.float32) * np.float32(0.02)
    E = rng.random((rhs, n, 3), np.float32) ** 4
    with ifx.Context(0) as ctx:
        ctx.upload(scene)
        ctx.upload_surfels(p, nrm, rng.random((n, 3), np.float32), 0.5 + rng.random(n, np.float32))
        assert ctx.build_clusters(9) == nc
        ctx.upload_transfer(starts, rng.integers(0, nc, starts[-1]), w)
        rad, irr, it, out = ctx.solve_batched(E, bounces)
        for r in {0, rhs // 2, rhs - 1}:
            ctx.set_emission(E[r])
            st = ctx.solve(bounces)
            s = ctx.surfels()
            assert (st.iterations, np.float32(st.residual)) == (it[r], out[r])
            assert s["rad"].tobytes() == rad[r].tobytes() and s["irr"].tobytes() == irr[r].tobytes()


def lengths(n, links, most, seed):
    """n row lengths of 0 to about 2 * most that add up to `links`."""
    length = np.random.default_rng(seed).integers(0, 2 * most + 1, n)
    i = 0
    while need := links - int(length.sum()):
        length[i] += max(-int(length[i]), min(need, 9))
        i += 1
    return length


@pytest.mark.parametrize("nc", [1023, 1024, 1025, 1056, 1057])
@pytest.mark.parametrize("rhs", [1, 15, 16, 17])
def test_at_the_number_of_clusters(nc, rhs):
    length = np.random.default_rng(nc).choice([0, 1, 15, 16, 17, 33, 150, 200], 5003)
    assert length.sum() >= 32 * 5003
    check(5003, nc, length, rhs, 9)


@pytest.mark.parametrize("n,rhs,links", [(3001, 16, 32 * 3001), (3001, 16, 32 * 3001 - 1), (40001, 3, 1 << 19),
                                         (40001, 3, (1 << 19) - 1), (78125, 16, 32 * 78125), (78126, 16, 32 * 78126),
                                         (78126, 16, 60 * 78126), (78126, 16, 60 * 78126 - 1)])
def test_at_the_number_of_links(n, rhs, links):
    check(n, 300, lengths(n, links, links // n, n), rhs, 3)
