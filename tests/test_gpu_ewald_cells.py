"""The periodic correction is looked up as a bucket's lists are applied, from
the table point found when each node was accepted (csrc/forces_grouped.cu).  A
box shifted by half its size on an axis has the same differences at other
images, so with coordinates and masses on which float32 arithmetic is exact the
same table points must be found and the forces agree.

Tolerance: 4096 float32 terms summed in another order, each rounded to 2^-24 of
a partial sum no larger than the largest force: a random walk of 64 such steps,
4e-6 of it; 2e-5 is five of those."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
N = 4096   # masses 1 / 4096: exact products and centres of mass


def _forces(p, quad, bpl):
    from cnb import _lib
    from cnb.core.octree import OctreeManager
    codes, _ = orc.compute_codes(p[:, 0], p[:, 1], p[:, 2], 1)
    perm = orc.argsort_stable(codes)
    P = [torch.from_numpy(np.ascontiguousarray(p[perm][:, k])).cuda() for k in range(3)]
    st = int(torch.cuda.current_stream().cuda_stream)
    tm = OctreeManager(N, node_table=True, bucket=32 * bpl, quad=quad)
    tm.build(P, torch.full((N,), 1.0 / N, device="cuda"), torch.from_numpy(codes[perm]).cuda())
    table = torch.empty((65 ** 3, 24), device="cuda")
    _lib.call("cnb_ewald_table", table.data_ptr(), 64, st)
    f = torch.empty((N, 3), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("cnb_forces_grouped_ewald", *(q.data_ptr() for q in P), tm.node_table.data_ptr(),
              tm.workspace.data_ptr(), f.data_ptr(), N, 0.0, None, bpl, 4, 1.0, 0.01, table.data_ptr(), 64,
              tm.quad.data_ptr() if quad else None, None, None, None, status.data_ptr(), st)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    out = np.empty((N, 3))
    out[perm] = f.cpu().numpy()
    # bodies of buckets whose centre is exactly half a box from some source on some axis: the
    # image is then a tie, taken either way
    nb = int(tm.workspace[0].item())
    tie = np.zeros(N, bool)
    for lo, count, _, _ in tm.workspace[4:4 + 4 * nb].view(nb, 4).cpu().numpy():
        b = p[perm[lo:lo + count]].astype(np.float64)
        c = 0.5 * (b.min(0) + b.max(0))
        tie[perm[lo:lo + count]] = (np.abs(p.astype(np.float64) - c) == 0.5).any()
    return out, tie


@pytest.mark.parametrize("quad,bpl", [(False, 1), (False, 2), (True, 2)])
@pytest.mark.parametrize("shift", [(0.5, 0.0, 0.0), (0.5, 0.5, 0.5)])
def test_forces_do_not_depend_on_the_images(shift, quad, bpl):
    rng = np.random.default_rng(11)
    p = rng.integers(0, 1 << 20, (N, 3)) / float(1 << 20)
    f, tie = _forces(p.astype(np.float32), quad, bpl)
    g, tie2 = _forces(((p + np.array(shift)) % 1.0).astype(np.float32), quad, bpl)
    ok = ~(tie | tie2)
    assert ok.sum() > N // 2
    assert np.abs(f[ok] - g[ok]).max() <= 2e-5 * np.abs(f).max()
