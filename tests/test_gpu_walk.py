"""The walk by groups of consecutive targets (csrc/forces_ref.cu): every group
size, both precisions, both tree layouts, ragged ranges, and the grouped
traversal's use of it on small systems, against the CPU oracle.

Tolerances: float64 sums of float32 inputs rounded once to float32, 1e-6 of the
largest force; float32 sums of at most a few thousand terms, each rounded to
2^-24: their random-walk error is below 1e-5 of the largest force (a body whose
float32 test lands on the other side of the reference's changes by one node's
multipole error, so float32 is compared between group sizes, which share their
decisions, not with the oracle)."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _tree(n, seed, scatter=False):
    rng = np.random.default_rng(seed)
    g = int(np.ceil(n ** (1 / 3)))
    cell = rng.permutation(g ** 3)[:n]
    q = np.stack([cell // (g * g), cell // g % g, cell % g], 1) / g
    p = ((q + rng.normal(0, 0.6 / g, q.shape)) % 1.0).astype(np.float32)
    p[p >= 1] = 0
    codes, _ = orc.compute_codes(p[:, 0], p[:, 1], p[:, 2], 0 if scatter else 1)
    perm = orc.argsort_stable(codes)
    p, codes = p[perm], codes[perm]
    pos = [np.ascontiguousarray(p[:, k]) for k in range(3)]
    mass = np.full(n, 1.0 / n, np.float32)
    ch, par = orc.build_tree(codes)
    nm, nc, lo, hi = orc.compute_multipoles(*pos, mass, ch, par)
    return pos, codes, mass, (ch, nm, nc, lo, hi), orc.find_root(par)


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _walk(pos, tree, root, theta, soft, prec, off, count, table):
    from cnb import _lib
    n = pos[0].size
    P, T = [_cuda(a) for a in pos], [_cuda(a) for a in tree]
    f = torch.full((n, 3), 7.0, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    r = torch.tensor([root], dtype=torch.int32, device="cuda")
    st = int(torch.cuda.current_stream().cuda_stream)
    end = (theta, 1.0, soft, 1.0, r.data_ptr(), off, count, n, prec, status.data_ptr(), st)
    if table:
        m = 2 * n - 1
        tab = torch.empty((4, m, 4), device="cuda")
        _lib.call("cnb_pack_nodes", *(t.data_ptr() for t in T[1:]), T[0].data_ptr(), tab.data_ptr(), m, st)
        _lib.call("cnb_compute_forces_table", *(p.data_ptr() for p in P), tab.data_ptr(), f.data_ptr(), *end)
    else:
        _lib.call("cnb_compute_forces", *(p.data_ptr() for p in P), *(t.data_ptr() for t in T),
                  f.data_ptr(), *end)
    torch.cuda.synchronize()
    return f.cpu().numpy(), int(status.item())


# counts on both sides of every group size's limit, and ranges that start and end inside a group
@pytest.mark.parametrize("table", [False, True])
@pytest.mark.parametrize("n,off,count", [(1, 0, 1), (2, 0, 2), (37, 5, 31), (8195, 1, 8192),
                                         (8195, 0, 8193), (24600, 3, 24576), (24600, 0, 24577)])
def test_float64_matches_the_oracle(n, off, count, table):
    pos, _, _, tree, root = _tree(n, n)
    if n == 1:
        want = np.zeros((1, 3), np.float32)
    else:
        want = orc.compute_forces(*pos, *tree, 0.6, 1.0, 0.01, 1.0, root)[0]
    got, status = _walk(pos, tree, root, 0.6, 0.01, 1, off, count, table)
    assert status == 0
    inside = slice(off, min(off + count, n))
    assert np.abs(got[inside] - want[inside]).max() <= 1e-6 * max(np.abs(want).max(), 1e-30)
    outside = np.ones(n, bool)
    outside[inside] = False
    assert (got[outside] == 7.0).all()


@pytest.mark.parametrize("prec,tol", [(0, 1e-5), (1, 1e-6)])
@pytest.mark.parametrize("scatter", [False, True])
def test_group_sizes_agree(prec, tol, scatter):
    """The whole system in one call (the largest group this size takes) and in
    pieces (smaller groups): the same nodes for every target."""
    n = 12000 if scatter else 270000
    pos, _, _, tree, root = _tree(n, 3, scatter)
    whole, status = _walk(pos, tree, root, 0.7, 0.01, prec, 0, n, True)
    assert status == 0
    for off, count in ((0, 5000), (4001, 20011) if n > 30000 else (4001, 7999), (n - 30001, 30001)):
        off = max(off, 0)
        part, status = _walk(pos, tree, root, 0.7, 0.01, prec, off, count, False)
        assert status == 0
        sl = slice(off, min(off + count, n))
        assert np.abs(part[sl] - whole[sl]).max() <= tol * np.abs(whole).max()


def test_deep_chain_drops_the_reference_s_children():
    """A chain of 200 levels: every target's own 64-entry stack fills, and what
    it drops is what the oracle's walk drops."""
    n = 200
    m = 2 * n - 1
    children = np.full((m, 2), -1, np.int32)
    for k in range(n - 1):
        children[n + k] = (n + k + 1, k) if k < n - 2 else (k, k + 1)
    rng = np.random.default_rng(1)
    pos = [rng.random(n).astype(np.float32) for _ in range(3)]
    p = np.stack(pos, 1)
    nm = np.full(m, 1.0 / n, np.float32)
    nc = np.concatenate([p, np.full((n - 1, 3), 0.5, np.float32)])
    lo = np.concatenate([p, np.zeros((n - 1, 3), np.float32)])
    hi = np.concatenate([p, np.ones((n - 1, 3), np.float32)])
    tree = (children, nm, nc, lo, hi)
    want = orc.compute_forces(*pos, *tree, 0.0, 1.0, 0.01, 1.0, n)[0]
    for table in (False, True):
        got, status = _walk(pos, tree, n, 0.0, 0.01, 1, 0, n, table)
        assert status == 1      # CNB_FLAG_STACK_OVERFLOW
        assert np.abs(got - want).max() <= 1e-6 * np.abs(want).max()


# the grouped traversal's rule: groups of 2, of 4, and past the limit the buckets
@pytest.mark.parametrize("n", [1, 2, 33, 8192, 8193, 98304, 98305])
def test_exact_decisions_at_the_edges_of_the_rule(n):
    from cnb import _lib
    from cnb.core.octree import OctreeManager
    pos, codes, mass, tree, root = _tree(n, n + 5)
    P, M = [_cuda(a) for a in pos], _cuda(mass)
    tm = OctreeManager(n, node_table=True, bucket=64)
    tm.build(P, M, _cuda(codes))
    f = torch.empty((n, 3), device="cuda")
    stats = torch.zeros(4, dtype=torch.int64, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("cnb_forces_grouped", *(p.data_ptr() for p in P), tm.node_table.data_ptr(),
              tm.workspace.data_ptr(), f.data_ptr(), n, 0.5, None, _lib.MAC_REF_X, 2, 4, 1.0, 0.01, 1.0,
              0.0, stats.data_ptr(), status.data_ptr(), int(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    if n == 1:
        assert not f.any() and int(stats[0]) == 1
        return
    want, _, _, acc = orc.compute_forces(*pos, *tree, 0.5, 1.0, 0.01, 1.0, root, return_accepted=True)
    assert int(stats[0]) == acc
    assert np.abs(f.cpu().numpy() - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("theta", [0.5, 0.3])
def test_redo_pass_past_the_rule(theta):
    """The bucket kernel's second pass (buckets given up after one round, forced
    here) at a size the groups do not take: bit-identical forces."""
    from cnb import _lib
    from cnb.core.octree import OctreeManager
    n = 110592
    pos, codes, mass, _, _ = _tree(n, 9)
    P, M = [_cuda(a) for a in pos], _cuda(mass)
    tm = OctreeManager(n, node_table=True, bucket=64)
    tm.build(P, M, _cuda(codes))
    out = []
    for every in (0, 3):
        f = torch.full((n, 3), float("nan"), device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        _lib.call("cnb_exact_test_spill", every)
        try:
            _lib.call("cnb_forces_grouped", *(p.data_ptr() for p in P), tm.node_table.data_ptr(),
                      tm.workspace.data_ptr(), f.data_ptr(), n, theta, None, _lib.MAC_REF_X, 2, 2, 1.0,
                      0.01, 1.0, 0.0, None, status.data_ptr(),
                      int(torch.cuda.current_stream().cuda_stream))
        finally:
            _lib.call("cnb_exact_test_spill", 0)
        torch.cuda.synchronize()
        assert int(status.item()) == 0
        out.append(f.cpu().numpy().view(np.uint32))
    np.testing.assert_array_equal(out[0], out[1])


@pytest.mark.parametrize("n,spread", [(30000, 0.2), (30000, 1e-3)])
def test_walk_that_opens_everything(n, spread):
    """theta = 0: every body meets every body, through a stack that would
    overflow if every round took 32 nodes."""
    from cnb import _lib
    from cnb.core.octree import OctreeManager
    rng = np.random.default_rng(n)
    p = (0.5 + rng.normal(0, spread, (n, 3))) % 1.0
    p = p.astype(np.float32)
    p[p >= 1] = 0
    codes, _ = orc.compute_codes(p[:, 0], p[:, 1], p[:, 2], 1)
    perm = orc.argsort_stable(codes)
    P = [_cuda(p[perm][:, k]) for k in range(3)]
    tm = OctreeManager(n, node_table=True, bucket=64)
    tm.build(P, torch.full((n,), 1.0 / n, device="cuda"), _cuda(codes[perm]))
    f = torch.empty((n, 3), device="cuda")
    stats = torch.zeros(4, dtype=torch.int64, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("cnb_forces_grouped", *(q.data_ptr() for q in P), tm.node_table.data_ptr(),
              tm.workspace.data_ptr(), f.data_ptr(), n, 0.0, None, _lib.MAC_REF_X, 2, 4, 1.0, 0.01, 1.0, 0.0,
              stats.data_ptr(), status.data_ptr(), int(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert int(stats[0]) == n * n
