"""Small systems whose trees are as deep as the keys allow: a cusp around a
corner of the box, every body in a key cell of its own, 64 levels.  Every node
that a walk opens leaves a sibling behind on each level, so the traversals'
stacks fill at the angles where they are widest; none may drop a node."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
SOFT = 1e-3


def _cusp(n, seed):
    rng = np.random.default_rng(seed)
    p = np.abs(rng.normal(size=(2 * n, 3))) ** 3 * 2.0 ** (-16 * rng.random((2 * n, 1))) * 0.3
    p = (p % 1.0).astype(np.float32)
    p[p >= 1] = 0
    codes, _ = orc.compute_codes(p[:, 0], p[:, 1], p[:, 2], 1)
    first = np.sort(np.unique(codes, return_index=True)[1])[:n]
    p, codes = p[first], codes[first]
    assert codes.size == n
    perm = orc.argsort_stable(codes)
    return [np.ascontiguousarray(p[perm][:, k]) for k in range(3)], codes[perm]


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# groups of 2 and of 4 targets; buckets, for which the main pass's region goes by theta
@pytest.mark.parametrize("n,bpl", [(10240, 2), (24576, 2), (24577, 2), (59145, 2), (120000, 1), (120000, 2)])
@pytest.mark.parametrize("theta", [0.1, 0.2, 0.3, 0.5])
def test_exact_decisions(n, bpl, theta):
    """The accepted (body, node) pairs are the oracle's, count for count; float32
    sums of at most n = 6e4 terms rounded to 2^-24: a random walk of sqrt(n)
    roundings is 1.5e-5 of the summed magnitudes, which are at most a few
    times the largest force in a cusp: 1e-4 (groups only: the buckets' lists take
    the cut of two heavy nodes here, at d^2 = 1e-7 to 5e-14, in float32).  Buckets
    that the main pass gives up, of itself or for the test, get the same forces
    from the second."""
    from cnb import _lib
    from cnb.core.octree import OctreeManager
    pos, codes = _cusp(n, 1)
    mass = np.full(n, 1.0 / n, np.float32)
    ch, par = orc.build_tree(codes)
    nm, nc, lo, hi = orc.compute_multipoles(*pos, mass, ch, par)
    want, dropped, _, acc = orc.compute_forces(*pos, ch, nm, nc, lo, hi, theta, 1.0, SOFT, 1.0,
                                               orc.find_root(par), return_accepted=True)
    assert dropped == 0
    P = [_cuda(a) for a in pos]
    tm = OctreeManager(n, node_table=True, bucket=32 * bpl)
    tm.build(P, _cuda(mass), _cuda(codes))
    out = []
    for every in (0, 3):
        f = torch.full((n, 3), float("nan"), device="cuda")
        stats = torch.zeros(4, dtype=torch.int64, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        _lib.call("cnb_exact_test_spill", every)
        try:
            _lib.call("cnb_forces_grouped", *(q.data_ptr() for q in P), tm.node_table.data_ptr(),
                      tm.workspace.data_ptr(), f.data_ptr(), n, theta, None, _lib.MAC_REF_X, bpl, 2, 1.0, SOFT,
                      1.0, 0.0, stats.data_ptr(), status.data_ptr(),
                      int(torch.cuda.current_stream().cuda_stream))
        finally:
            _lib.call("cnb_exact_test_spill", 0)
        torch.cuda.synchronize()
        assert int(status.item()) == 0
        assert int(stats[0]) == acc
        out.append(f.cpu().numpy())
    assert np.isfinite(out[0]).all()
    if n <= (_lib.EXACT_WALK_BODIES_SMALL_ANGLE if theta < 0.4 else _lib.EXACT_WALK_BODIES):
        assert np.abs(out[0] - want).max() <= 1e-4 * np.abs(want).max()
    np.testing.assert_array_equal(out[0].view(np.uint32), out[1].view(np.uint32))


@pytest.mark.parametrize("n,bpl", [(20000, 2), (59145, 2), (120000, 1), (120000, 2)])
def test_a_deep_tree_costs_what_its_pairs_cost(n, bpl):
    """Per accepted pair a cusp takes at most four times as long as the same
    number of bodies spread evenly (about as long when nothing goes wrong; a
    walk that crawls through a full stack takes tens of times as long)."""
    from cnb import _lib
    from cnb.core.octree import OctreeManager
    theta = 0.3
    p = np.random.default_rng(1).random((n, 3)).astype(np.float32)
    codes, _ = orc.compute_codes(p[:, 0], p[:, 1], p[:, 2], 1)
    perm = orc.argsort_stable(codes)
    even = [p[perm][:, k] for k in range(3)], codes[perm]
    cost = []
    for pos, codes in (even, _cusp(n, 1)):
        P = [_cuda(a) for a in pos]
        tm = OctreeManager(n, node_table=True, bucket=32 * bpl)
        tm.build(P, torch.full((n,), 1.0 / n, device="cuda"), _cuda(codes))
        f = torch.empty((n, 3), device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        best = float("inf")
        for _ in range(4):
            stats = torch.zeros(4, dtype=torch.int64, device="cuda")
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            _lib.call("cnb_forces_grouped", *(q.data_ptr() for q in P), tm.node_table.data_ptr(),
                      tm.workspace.data_ptr(), f.data_ptr(), n, theta, None, _lib.MAC_REF_X, bpl, 2, 1.0, SOFT,
                      1.0, 0.0, stats.data_ptr(), status.data_ptr(),
                      int(torch.cuda.current_stream().cuda_stream))
            e[1].record()
            e[1].synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        assert int(status.item()) == 0
        cost.append(best / int(stats[0]))
    assert cost[1] <= 4 * cost[0]


# per law and bucket width a size for teams of eight, four and two warps
TEAMS = {("bucket", 2): (20000, 40000, 70000), ("bucket", 1): (8000, 20000, 40000),
         ("periodic", 2): (20000, 70000, 140000), ("periodic", 1): (12000, 40000, 70000),
         ("ewald", 2): (20000, 50000, 70000), ("ewald", 1): (8000, 20000, 40000),
         ("quad", 2): (12000, 40000, 70000), ("quad", 1): (6000, 18000, 30000)}


@pytest.mark.parametrize("theta", [0.0, 0.1, 0.2])
@pytest.mark.parametrize("law,bpl,n", [(law, bpl, n) for law, bpl in TEAMS for n in TEAMS[law, bpl]])
def test_teams_drop_nothing(law, bpl, n, theta):
    """No node is dropped (the status says so); at theta = 0 every body meets
    every leaf exactly once."""
    from cnb import _lib
    from cnb.core.octree import OctreeManager
    pos, codes = _cusp(n, 3)
    P = [_cuda(a) for a in pos]
    tm = OctreeManager(n, node_table=True, bucket=32 * bpl, quad=law == "quad")
    tm.build(P, torch.full((n,), 1.0 / n, device="cuda"), _cuda(codes))
    f = torch.full((n, 3), float("nan"), device="cuda")
    stats = torch.zeros(4, dtype=torch.int64, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = int(torch.cuda.current_stream().cuda_stream)
    head = [q.data_ptr() for q in P] + [tm.node_table.data_ptr(), tm.workspace.data_ptr(), f.data_ptr(), n,
                                        theta, None]
    if law in ("ewald", "quad"):
        table = torch.empty((9 ** 3, 24), device="cuda")
        _lib.call("cnb_ewald_table", table.data_ptr(), 8, st)
        _lib.call("cnb_forces_grouped_ewald", *head, bpl, 4, 1.0, SOFT, table.data_ptr(), 8,
                  tm.quad.data_ptr() if law == "quad" else None, None, None, stats.data_ptr(),
                  status.data_ptr(), st)
    else:
        mac = _lib.MAC_PERIODIC if law == "periodic" else _lib.MAC_REF_X_BUCKET
        _lib.call("cnb_forces_grouped", *head, mac, bpl, 4, 1.0, SOFT, 1.0, 0.0, stats.data_ptr(),
                  status.data_ptr(), st)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert bool(torch.isfinite(f).all())
    if theta == 0.0:
        assert int(stats[0]) == n * n
