"""The upward pass over the reference's node arrays (csrc/tree.cu) uses the
leaves' counters as scratch: what they hold on entry has no effect, and a tree
whose parents name a leaf is reported and never reaches them."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _bodies(n):
    rng = np.random.default_rng(n)
    p = rng.random((n, 3)).astype(np.float32)
    codes, _ = orc.compute_codes(p[:, 0], p[:, 1], p[:, 2], 1)
    perm = orc.argsort_stable(codes)
    pos = [np.ascontiguousarray(p[perm][:, k]) for k in range(3)]
    return pos, rng.random(n).astype(np.float32), *orc.build_tree(codes[perm])


def _upward(pos, mass, ch, par, comp, leaves):
    from cnb import _lib
    n = mass.size
    m = 2 * n - 1
    c = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    P, M, CH, PA = [c(p) for p in pos], c(mass), c(ch), c(par)
    out = [torch.zeros(m, device="cuda")] + [torch.zeros((m, 3), device="cuda") for _ in range(3)]
    err = torch.zeros((m, 4), device="cuda")
    counts = torch.zeros(m, dtype=torch.int32, device="cuda")
    counts[:n] = c(leaves)
    root64 = torch.zeros(4, dtype=torch.float64, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("cnb_upward", *(p.data_ptr() for p in P), M.data_ptr(), CH.data_ptr(), PA.data_ptr(),
              *(o.data_ptr() for o in out), err.data_ptr(), counts.data_ptr(), n, int(comp), root64.data_ptr(),
              status.data_ptr(), int(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return [o.cpu().numpy().view(np.uint32) for o in out], counts.cpu().numpy(), int(status.item())


@pytest.mark.parametrize("comp", [False, True])
@pytest.mark.parametrize("n", [2, 512, 513, 5000])
def test_leaf_counters_may_hold_anything(n, comp):
    tree = _bodies(n)
    clean = _upward(*tree, comp, np.zeros(n, np.int32))
    rng = np.random.default_rng(1)
    for leaves in (np.full(n, 0x7fffffff, np.int32), np.full(n, -1, np.int32),
                   rng.integers(1, 2 * n - 1, n).astype(np.int32)):
        got, counts, status = _upward(*tree, comp, leaves)
        assert status == clean[2] == 0
        for g, w in zip(got, clean[0]):
            np.testing.assert_array_equal(g, w)
        assert (counts[:n] == 0).all() and (counts[n:] == 2).all()


# a leaf's and an internal node's parent; in the node's own block of 512 leaves and in another
@pytest.mark.parametrize("n,node,leaf", [(400, 7, 9), (400, 400 + 30, 9), (3000, 100, 2500),
                                         (3000, 3000 + 1600, 1601), (3000, 3000 + 1600, 5)])
def test_a_parent_that_is_a_leaf_is_reported(n, node, leaf):
    from cnb import _lib
    pos, mass, ch, par = _bodies(n)
    par = par.copy()
    assert par[node] >= n
    par[node] = leaf
    for comp in (False, True):
        _, counts, status = _upward(pos, mass, ch, par, comp, np.zeros(n, np.int32))
        assert status & _lib.FLAG_BAD_TOPOLOGY
        assert (counts[:n] == 0).all()
