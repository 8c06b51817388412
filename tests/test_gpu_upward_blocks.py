"""The upward pass over the reference's node arrays in two launches
(csrc/tree.cu: blocks of 512 leaves, then climbs from the nodes they leave), at
the blocks' edges: every float bit for bit as the oracle's, every counter at its
two arrivals, the leaves' counters back at zero; and on the trees the
reference's own tie rule breaks (runs of equal keys), the nodes that can be
formed."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _run(pos, mass, ch, par, mode):
    from cnb import _lib
    n = mass.size
    m = 2 * n - 1
    c = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    P, M, CH, PA = [c(p) for p in pos], c(mass), c(ch), c(par)
    out = [torch.zeros(m, device="cuda")] + [torch.zeros((m, 3), device="cuda") for _ in range(3)]
    err = torch.zeros((m, 4), device="cuda")
    counts = torch.zeros(m, dtype=torch.int32, device="cuda")
    root64 = torch.zeros(4, dtype=torch.float64, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = int(torch.cuda.current_stream().cuda_stream)
    if mode == "raw":
        _lib.call("cnb_compute_multipoles", *(p.data_ptr() for p in P), M.data_ptr(), CH.data_ptr(), PA.data_ptr(),
                  *(o.data_ptr() for o in out), counts.data_ptr(), n, status.data_ptr(), st)
    else:
        _lib.call("cnb_upward", *(p.data_ptr() for p in P), M.data_ptr(), CH.data_ptr(), PA.data_ptr(),
                  *(o.data_ptr() for o in out), err.data_ptr(), counts.data_ptr(), n, 1 if mode == "comp" else 0,
                  root64.data_ptr(), status.data_ptr(), st)
    torch.cuda.synchronize()
    return [o.cpu().numpy() for o in out], counts.cpu().numpy(), int(status.item())


@pytest.mark.parametrize("n", [2, 3, 511, 512, 513, 1023, 1024, 1025, 4097, 20000])
def test_block_edges_match_the_oracle(n):
    rng = np.random.default_rng(n)
    p = rng.random((n, 3)).astype(np.float32)
    codes, _ = orc.compute_codes(p[:, 0], p[:, 1], p[:, 2], 1)
    perm = orc.argsort_stable(codes)
    pos = [np.ascontiguousarray(p[perm][:, k]) for k in range(3)]
    mass = rng.random(n).astype(np.float32)
    ch, par = orc.build_tree(codes[perm])
    want = orc.compute_multipoles(*pos, mass, ch, par)   # normalised centres
    got, counts, status = _run(pos, mass, ch, par, "plain")
    assert status == 0
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g.view(np.uint32), np.asarray(w, np.float32).reshape(g.shape).view(np.uint32))
    assert (counts[n:] == 2).all() and (counts[:n] == 0).all()
    # compensated: the float64 sums to float32 rounding
    got, counts, status = _run(pos, mass, ch, par, "comp")
    assert status == 0
    assert abs(got[0][n if n > 1 else 0] - mass.astype(np.float64).sum()) <= 2.0 ** -24 * mass.sum()
    np.testing.assert_array_equal(got[2].view(np.uint32), np.asarray(want[2], np.float32).view(np.uint32))
    assert (counts[n:] == 2).all() and (counts[:n] == 0).all()


def test_broken_trees_form_what_can_be_formed():
    """Runs of equal keys: some node is two nodes' child and another nobody's.
    Both forms of the pass agree with a walk on the host that forms a node when
    both of the children that name it as their parent have been formed."""
    rng = np.random.default_rng(3)
    n = 3000
    codes = np.sort(rng.integers(0, 900, n).astype(np.uint64) << np.uint64(20))
    ch, par = orc.build_tree(codes)
    pos = [rng.random(n).astype(np.float32) for _ in range(3)]
    mass = np.full(n, 1.0 / 4096, np.float32)
    got, counts, _ = _run(pos, mass, ch, par, "raw")
    formed = np.zeros(2 * n - 1, bool)
    formed[:n] = True
    total = np.zeros(2 * n - 1)
    total[:n] = mass
    changed = True
    while changed:
        changed = False
        for v in range(n, 2 * n - 1):
            l, r = ch[v]
            if not formed[v] and formed[l] and formed[r] and par[l] == v and par[r] == v and l != r:
                formed[v] = True
                total[v] = total[l] + total[r]
                changed = True
    assert formed[n:].sum() < n - 1     # the tree is broken
    # masses are multiples of 2^-12 below one: exact in any order
    np.testing.assert_array_equal(got[0][formed], total[formed].astype(np.float32))
    assert (got[0][~formed] == 0).all()
    assert (counts[:n] == 0).all()
