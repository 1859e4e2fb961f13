"""The context's solve over its sliced copy where its kernels change: 65,536
rows (from there one wave of CTAs takes several rows a thread), 1,024 and 4,096
clusters (whose radiosities it gathers from shared memory below them). Against
the f32 sums formed by numpy in member and CSR order, equal to the bit."""
import numpy as np
import pytest

import interflect_b200 as ifx
from conftest import scene_src
from test_gpu_solve_rows import row_sums

pytestmark = pytest.mark.gpu


def placed(scene, res, count, n, rng):
    """n surfels in `count` clusters: every (cell, normal) pair of the first `count` has at least one."""
    lo, hi = np.array(scene.info.bounds_lo, np.float64), np.array(scene.info.bounds_hi, np.float64)
    at = np.concatenate([np.arange(count), rng.integers(0, count, n - count)])
    rng.shuffle(at)
    cell, axis = at // 6, at % 6
    ijk = np.stack([cell % res, cell // res % res, cell // (res * res)], 1)
    nrm = np.zeros((n, 3), np.float32)
    nrm[np.arange(n), axis // 2] = 1.0 - 2.0 * (axis % 2)
    p = lo + (ijk + rng.uniform(0.3, 0.7, (n, 3))) / res * (hi - lo)
    return p.astype(np.float32), nrm


@pytest.mark.parametrize("n,nc", [(65535, 1024), (65536, 1024), (65535, 1025), (65536, 1025), (65573, 4096), (65573, 4097),
                                  (230001, 3000), (400003, 700)])
def test_rows_equal_the_ordered_sums(n, nc):
    check(n, nc, np.random.default_rng(n).choice([0, 1, 3, 4, 5, 8, 9, 12, 31, 32, 33, 65], n))


@pytest.mark.parametrize("n,nc,links", [(8000, 1000, 63000), (8000, 1000, 62999), (70001, 2500, 350005)])
def test_rows_of_few_links(n, nc, links):
    """A CTA of 128 rows copies the radiosities where it has as many links as there are clusters."""
    length = np.random.default_rng(n).multinomial(links, np.full(n, 1 / n))
    check(n, nc, length)


def check(n, nc, length):
    rng = np.random.default_rng(n + nc)
    scene = ifx.parse(scene_src("cornell"))
    p, nrm = placed(scene, 9, nc, n, rng)
    albedo, e, area = rng.random((n, 3), np.float32), rng.random((n, 3), np.float32), 0.5 + rng.random(n, np.float32)
    starts = np.zeros(n + 1, np.uint32)
    starts[1:] = np.cumsum(length)
    idx = rng.integers(0, nc, starts[-1])
    w = rng.random(int(starts[-1]), np.float32) * np.float32(0.02)
    with ifx.Context(0) as ctx:
        ctx.upload(scene)
        ctx.upload_surfels(p, nrm, albedo, area)
        assert ctx.build_clusters(9) == nc
        c = ctx.clusters(nc)
        ctx.upload_transfer(starts, idx, w)
        ctx.set_emission(e)
        st = ctx.solve(2)
        s = ctx.surfels()
    offsets, members = c["offsets"].astype(np.int64), c["members"]
    rad, count = e, np.diff(offsets)
    for _ in range(2):
        before = rad
        acc, prod = np.zeros((nc, 3), np.float32), rad[members] * area[members, None]
        for j in range(int(count.max())):
            k = np.nonzero(count > j)[0]
            acc[k] = acc[k] + prod[offsets[k] + j]
        irr = row_sums(starts.astype(np.int64), idx, w, acc / np.maximum(c["area"], np.float32(1e-12))[:, None])
        rad = e + albedo * irr
    assert st.iterations == 2 and np.float32(st.residual) == np.abs(rad - before).max()
    assert s["irr"].tobytes() == irr.tobytes() and s["rad"].tobytes() == rad.tobytes()
