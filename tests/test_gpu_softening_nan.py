"""A softening that is not a number is reported by every force path: NaN forces
and CNB_FLAG_NONFINITE, on small systems (groups of bodies, teams of warps) and
on larger ones (a warp per bucket), in both precisions of the per-body walk and
where the softening is a box's own."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _tree(n, quad=False):
    from cnb.core.octree import OctreeManager
    p = np.random.default_rng(n).random((n, 3)).astype(np.float32)
    codes, _ = orc.compute_codes(p[:, 0], p[:, 1], p[:, 2], 1)
    perm = orc.argsort_stable(codes)
    P = [torch.from_numpy(np.ascontiguousarray(p[perm][:, k])).cuda() for k in range(3)]
    tm = OctreeManager(n, node_table=True, bucket=64, quad=quad)
    tm.build(P, torch.full((n,), 1.0 / n, device="cuda"), torch.from_numpy(codes[perm]).cuda())
    f = torch.zeros((n, 3), device="cuda")
    return P, tm, f, torch.zeros(1, dtype=torch.int32, device="cuda"), int(torch.cuda.current_stream().cuda_stream)


def _reported(f, status):
    from cnb import _lib
    torch.cuda.synchronize()
    assert int(status.item()) & _lib.FLAG_NONFINITE
    assert bool(torch.isnan(f).all())


@pytest.mark.parametrize("law,n", [("ref_x", 4000), ("ref_x", 120011), ("ref_x_bucket", 4000),
                                   ("ref_x_bucket", 120011), ("periodic", 4000), ("ewald", 4000),
                                   ("ewald", 120011), ("quad", 4000), ("quad", 120011)])
def test_grouped(law, n):
    from cnb import _lib
    P, tm, f, status, st = _tree(n, law == "quad")
    head = [q.data_ptr() for q in P] + [tm.node_table.data_ptr(), tm.workspace.data_ptr(), f.data_ptr(), n, 0.6, None]
    nan = float("nan")
    if law in ("ewald", "quad"):
        table = torch.empty((9 ** 3, 24), device="cuda")
        _lib.call("cnb_ewald_table", table.data_ptr(), 8, st)
        _lib.call("cnb_forces_grouped_ewald", *head, 2, 4, 1.0, nan, table.data_ptr(), 8,
                  tm.quad.data_ptr() if law == "quad" else None, None, None, None, status.data_ptr(), st)
    else:
        mac = {"ref_x": _lib.MAC_REF_X, "ref_x_bucket": _lib.MAC_REF_X_BUCKET, "periodic": _lib.MAC_PERIODIC}[law]
        _lib.call("cnb_forces_grouped", *head, mac, 2, 4, 1.0, nan, 1.0, 0.0, None, status.data_ptr(), st)
    _reported(f, status)


@pytest.mark.parametrize("precision", [0, 1])
def test_per_body(precision):
    from cnb import _lib
    n = 4000
    P, tm, f, status, st = _tree(n)
    _lib.call("cnb_compute_forces_table", *(q.data_ptr() for q in P), tm.node_table.data_ptr(), f.data_ptr(), 0.6,
              1.0, float("nan"), 1.0, tm.root_idx.data_ptr(), 0, n, n, precision, status.data_ptr(), st)
    _reported(f, status)


@pytest.mark.parametrize("mac", ["ref_x", "ewald"])
def test_boxes(mac):
    from cnb import _lib
    from cnb.core.batched import BatchedBoxes
    bb = BatchedBoxes([dict(n_grid=16, seed=k, a_start=0.05, theta=0.5) for k in (1, 2)], mac=mac)
    bb.sort_and_build()
    bb.box_params[1, 1] = float("nan")
    bb.compute_forces()
    with pytest.raises(_lib.CnbError):
        bb.check()
    torch.cuda.synchronize()
    assert bool(torch.isfinite(bb.force[bb.box_slice(0)]).all())
    assert bool(torch.isnan(bb.force[bb.box_slice(1)]).all())
