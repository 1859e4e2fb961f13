"""The device-buffer solve on both sides of the line from which rows are walked
in 256-bit loads: 49,152 rows with a mean of 64 links. One link less and the
16-byte walk runs; the kernel that holds both decides by the links themselves.
Row lengths from 0 to 300, at every alignment, the last row ending at any place
of a 32-byte block; against the f32 sums formed by numpy in CSR order, equal to
the bit."""
import numpy as np
import pytest

import interflect_b200 as ifx
from test_gpu_solve_rows import row_sums

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,missing", [(49152, 1), (49152, 0), (49152, -1), (49152 + 37, -5), (70001, 3), (70001, -2),
                                       (49151, 0)])
def test_rows_equal_the_ordered_sums(n, missing):
    torch = pytest.importorskip("torch")
    rng, nc = np.random.default_rng(n - missing), 500
    length = rng.choice([0, 1, 7, 8, 9, 31, 64, 65, 97, 129, 300], n)
    # Rows in turn give or take links until the mean is 64, `missing` links short.
    need, i = 64 * n - missing - int(length.sum()), 0
    while need:
        step = max(-int(length[i]), min(need, 40))
        length[i] += step
        need -= step
        i += 1
    starts = np.zeros(n + 1, np.int64)
    starts[1:] = np.cumsum(length)
    assert starts[-1] == 64 * n - missing
    idx = rng.integers(0, nc, starts[-1])
    w = (rng.random(starts[-1], np.float32) * 0.01).astype(np.float32)
    albedo, direct = rng.random((n, 3), np.float32), rng.random((n, 3), np.float32)
    # One member of area 1 a cluster: its mean is the member's radiosity.
    members = rng.permutation(n)[:nc]

    def four(xyz, last=0.0):
        a = np.full((len(xyz), 4), last, np.float32)
        a[:, :3] = xyz
        return torch.from_numpy(a).cuda()

    def u32(a):
        return torch.from_numpy(np.ascontiguousarray(a, np.uint32).view(np.int32)).cuda()

    zero = np.zeros((n, 3), np.float32)
    d = dict(p=four(zero, 1.0), direct=four(direct), albedo=four(albedo), irr=four(zero), rad=four(direct),
             cp=four(zero[:nc], 1.0), ranges=u32(np.stack([np.arange(nc), np.arange(nc) + 1], 1).reshape(-1)),
             members=u32(members), starts=u32(starts), idx=u32(idx), w=torch.from_numpy(w).cuda())
    st = ifx.solve_noalloc(0, torch.cuda.current_stream().cuda_stream, n, nc, *(v.data_ptr() for v in d.values()), 2)
    rad = direct
    for _ in range(2):
        before = rad
        irr = row_sums(starts, idx, w, rad[members])
        rad = direct + albedo * irr
    assert st.iterations == 2 and np.float32(st.residual) == np.abs(rad - before).max()
    assert d["irr"].cpu().numpy()[:, :3].tobytes() == irr.tobytes()
    assert d["rad"].cpu().numpy()[:, :3].tobytes() == rad.tobytes()
