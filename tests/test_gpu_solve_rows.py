"""The device-buffer solve's row kernels against the same f32 sums formed by
numpy in CSR order: from 49,152 rows on links are read eight at a time from
aligned places. Rows of 0, 1, 31, 32, 33, 64, 65 and other lengths, at every alignment, and
row counts around the switch and off a warp's multiple. Products and sums
round the same way, so the results are equal to the bit."""
import numpy as np
import pytest

import interflect_b200 as ifx

pytestmark = pytest.mark.gpu


def row_sums(starts, idx, w, crad):
    n = len(starts) - 1
    length = np.diff(starts)
    irr = np.zeros((n, 3), np.float32)
    for j in range(int(length.max(initial=0))):
        r = np.nonzero(length > j)[0]
        k = starts[r] + j
        irr[r] = irr[r] + crad[idx[k]] * w[k, None]
    return irr


@pytest.mark.parametrize("n,nc", [(1000, 300), (49151, 300), (49152, 300), (49152 + 37, 4096), (70001, 4097)])
def test_rows_equal_the_ordered_sums(n, nc):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + nc)
    length = rng.choice([0, 1, 2, 5, 31, 32, 33, 63, 64, 65, 97], n)
    starts = np.zeros(n + 1, np.int64)
    starts[1:] = np.cumsum(length)
    idx = rng.integers(0, nc, starts[-1])
    w = (rng.random(starts[-1], np.float32) * 0.02).astype(np.float32)
    area = (0.5 + rng.random(n)).astype(np.float32)
    albedo, direct = rng.random((n, 3), np.float32), rng.random((n, 3), np.float32)
    cid = np.concatenate([np.arange(nc), rng.integers(0, nc, n - nc)]) if n >= nc else rng.integers(0, nc, n)
    members = np.argsort(cid, kind="stable")
    offsets = np.searchsorted(cid[members], np.arange(nc + 1))
    carea = np.maximum(np.array([area[members[a:b]].sum() for a, b in zip(offsets[:-1], offsets[1:])], np.float32), 1e-3)

    def bounce(rad):
        # Cluster means: members summed in member order.
        acc = np.zeros((nc, 3), np.float32)
        count = np.diff(offsets)
        prod = rad[members] * area[members, None]
        for j in range(int(count.max())):
            c = np.nonzero(count > j)[0]
            acc[c] = acc[c] + prod[offsets[c] + j]
        irr = row_sums(starts, idx, w, acc / carea[:, None])
        return irr, direct + albedo * irr

    def f4(xyz, last=None):
        a = np.zeros((len(xyz), 4), np.float32)
        a[:, :3] = xyz
        if last is not None:
            a[:, 3] = last
        return torch.from_numpy(a).cuda()

    def u32(a):
        return torch.from_numpy(np.ascontiguousarray(a, np.uint32).view(np.int32)).cuda()

    d = dict(p=f4(np.zeros((n, 3), np.float32), area), direct=f4(direct), albedo=f4(albedo),
             irr=f4(np.zeros((n, 3), np.float32)), rad=f4(direct), cp=f4(np.zeros((nc, 3), np.float32), carea),
             ranges=u32(np.stack([offsets[:-1], offsets[1:]], 1).reshape(-1)), members=u32(members),
             starts=u32(starts), idx=u32(idx), w=torch.from_numpy(w).cuda())
    st = ifx.solve_noalloc(0, torch.cuda.current_stream().cuda_stream, n, nc, *(v.data_ptr() for v in d.values()), 2)
    irr, rad = direct, direct
    for _ in range(2):
        before = rad
        irr, rad = bounce(rad)
    assert st.iterations == 2
    assert np.float32(st.residual) == np.abs(rad - before).max()
    assert d["irr"].cpu().numpy()[:, :3].tobytes() == irr.tobytes()
    assert d["rad"].cpu().numpy()[:, :3].tobytes() == rad.tobytes()
