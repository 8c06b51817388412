"""The grouped traversal with a team of warps per bucket (csrc/forces_grouped.cu):
every law and bucket width on both sides of each team size's limit.

theta = 0 opens every node, so each body meets every leaf exactly once (the
count is n^2, whatever the order) and the stack is as full as it gets.  Forces
of the minimum-image laws are then a direct sum: float32 terms with about eight
roundings each, added in float32, so their error is a random walk of n
roundings, (8 + sqrt(n)) 2^-24 of the summed magnitudes.

At theta > 0 a box alone (teams) is compared with the same box inside a batch
too large for teams: the same buckets and nodes, another order of at most 3000
terms.  The magnitudes of a unit box's forces add up to less than 10 (2 pi for
a sphere of radius one half, doubled near the softening), so both sums are
within (8 + sqrt(3000)) 2^-24 * 10 = 4e-5 of the exact one, 8e-5 of each other;
the two forms of a quadrupole or table term share their roundings."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

# coordinates k / M with odd M: no two differ by half a box, where the image is a tie
M = 1000003


def _tree(n, bpl, quad):
    from cnb.core.octree import OctreeManager
    rng = np.random.default_rng(n + bpl)
    p = (rng.integers(0, M, (n, 3)) / M).astype(np.float32)
    codes, _ = orc.compute_codes(p[:, 0], p[:, 1], p[:, 2], 1)
    perm = orc.argsort_stable(codes)
    pos = [torch.from_numpy(np.ascontiguousarray(p[perm, k])).cuda() for k in range(3)]
    mass = torch.full((n,), 1.0 / n, device="cuda")
    tm = OctreeManager(n, node_table=True, bucket=32 * bpl, quad=quad)
    tm.build(pos, mass, torch.from_numpy(codes[perm]).cuda())
    return pos, mass, tm


SIZES = {"bucket": (1, 2, 65, 8193, 24577, 49153, 57345, 114688), "periodic": (1, 65, 12289, 49153, 65537),
         "ewald": (1, 2, 65, 8193, 24577, 32769, 65537, 98304), "quad": (1, 65, 6145, 12289, 20481, 49153, 98304)}
# 32-body buckets: nothing above their last limit (one warp's stack may drop nodes at theta = 0)
LAST = {"bucket": 57344, "periodic": 65537, "ewald": 40960, "quad": 32768}


@pytest.mark.parametrize("bpl", [1, 2])
@pytest.mark.parametrize("law,n", [(law, n) for law in SIZES for n in SIZES[law]])
def test_every_leaf_once(law, n, bpl):
    from cnb import _lib
    from cnb.controller import direct_sum
    if bpl == 1:
        n = min(n, LAST[law])
    pos, mass, tm = _tree(n, bpl, law == "quad")
    soft = 0.02
    f = torch.full((n, 3), 7.0, device="cuda")
    stats = torch.zeros(4, dtype=torch.int64, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = int(torch.cuda.current_stream().cuda_stream)
    head = [q.data_ptr() for q in pos] + [tm.node_table.data_ptr(), tm.workspace.data_ptr(), f.data_ptr(), n, 0.0, None]
    if law in ("ewald", "quad"):
        table = torch.empty((9 ** 3, 24), device="cuda")
        _lib.call("cnb_ewald_table", table.data_ptr(), 8, st)
        _lib.call("cnb_forces_grouped_ewald", *head, bpl, 4, 1.0, soft, table.data_ptr(), 8,
                  tm.quad.data_ptr() if law == "quad" else None, None, None, stats.data_ptr(),
                  status.data_ptr(), st)
    else:
        mac = _lib.MAC_PERIODIC if law == "periodic" else _lib.MAC_REF_X_BUCKET
        _lib.call("cnb_forces_grouped", *head, mac, bpl, 4, 1.0, soft, 1.0, 0.0, stats.data_ptr(),
                  status.data_ptr(), st)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert int(stats[0].item()) == n * n
    assert bool(torch.isfinite(f).all())
    if law in ("ewald", "quad"):
        return
    t = torch.from_numpy(np.random.default_rng(1).choice(n, min(n, 64), replace=False)).cuda()
    want = direct_sum(pos, mass, t, 1.0, soft)
    x = torch.stack(pos, 1).double()
    d = x[None] - x[t][:, None]
    d -= torch.round(d)
    size = (d.abs() * ((d * d).sum(2, keepdim=True) + soft * soft) ** -1.5).sum(1) / n
    assert bool(((f[t].double() - want).abs() <= (8 + n ** 0.5) * 2.0 ** -24 * size + 1e-12).all())


@pytest.mark.parametrize("bpl", [1, 2])
@pytest.mark.parametrize("mac", ["ref_x_bucket", "ewald"])
@pytest.mark.parametrize("grid", [16, 24, 32])
def test_same_forces_as_one_warp_a_bucket(grid, mac, bpl):
    from cnb.core.batched import BatchedBoxes
    mine = [dict(n_grid=grid, seed=5, a_start=0.05, theta=0.5), dict(n_grid=16, seed=4, a_start=0.05, theta=0.5)]
    others = [dict(n_grid=32, seed=6 + k, a_start=0.05, theta=0.6) for k in range(4)]
    force = []
    for boxes in (mine, mine + others):
        bb = BatchedBoxes(boxes, mac=mac, bodies_per_lane=bpl)
        bb.sort_and_build()
        inter = torch.zeros(bb.n, dtype=torch.int32, device="cuda")
        bb.stats.zero_()
        bb.compute_forces(bucket_inter=inter if mac == "ewald" else None)
        bb.check()
        if mac == "ewald":
            bk = bb.buckets()
            assert int((inter[:bk.shape[0]].long() * bk[:, 1].long()).sum()) == int(bb.stats[0])
        force.append(bb.force[bb.box_slice(0)].double())
    assert bool(((force[0] - force[1]).abs() <= 8e-5).all())
