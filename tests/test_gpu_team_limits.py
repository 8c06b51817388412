"""Both sides of each limit between the team sizes of the bucket traversal
(csrc/forces_grouped.cu, team_warps): at theta = 0 every body meets every leaf
exactly once, whatever the team, and no node is dropped."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

LIMITS = {("bucket", 2): (20480, 57344), ("bucket", 1): (10240, 20480), ("periodic", 2): (49152, 131072),
          ("periodic", 1): (24576, 65536), ("ewald", 2): (20480, 57344), ("ewald", 1): (10240, 20480),
          ("quad", 2): (14336, 40960), ("quad", 1): (7168, 18432)}


@pytest.mark.parametrize("law,bpl,n", [(law, bpl, n + more) for (law, bpl), ns in LIMITS.items() for n in ns
                                       for more in (0, 1)] + [("ewald", 1, 45056)])
def test_every_leaf_once(law, bpl, n):
    from cnb import _lib
    from cnb.core.octree import OctreeManager
    p = np.random.default_rng(n + bpl).random((n, 3)).astype(np.float32)
    codes, _ = orc.compute_codes(p[:, 0], p[:, 1], p[:, 2], 1)
    perm = orc.argsort_stable(codes)
    P = [torch.from_numpy(np.ascontiguousarray(p[perm][:, k])).cuda() for k in range(3)]
    tm = OctreeManager(n, node_table=True, bucket=32 * bpl, quad=law == "quad")
    tm.build(P, torch.full((n,), 1.0 / n, device="cuda"), torch.from_numpy(codes[perm]).cuda())
    f = torch.full((n, 3), float("nan"), device="cuda")
    stats = torch.zeros(4, dtype=torch.int64, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = int(torch.cuda.current_stream().cuda_stream)
    head = [q.data_ptr() for q in P] + [tm.node_table.data_ptr(), tm.workspace.data_ptr(), f.data_ptr(), n, 0.0, None]
    if law in ("ewald", "quad"):
        table = torch.empty((9 ** 3, 24), device="cuda")
        _lib.call("cnb_ewald_table", table.data_ptr(), 8, st)
        _lib.call("cnb_forces_grouped_ewald", *head, bpl, 4, 1.0, 0.02, table.data_ptr(), 8,
                  tm.quad.data_ptr() if law == "quad" else None, None, None, stats.data_ptr(),
                  status.data_ptr(), st)
    else:
        mac = _lib.MAC_PERIODIC if law == "periodic" else _lib.MAC_REF_X_BUCKET
        _lib.call("cnb_forces_grouped", *head, mac, bpl, 4, 1.0, 0.02, 1.0, 0.0, stats.data_ptr(),
                  status.data_ptr(), st)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert int(stats[0]) == n * n
    assert bool(torch.isfinite(f).all())
