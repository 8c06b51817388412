"""The bucket form of the exact traversal (csrc/forces_exact.cu) at a size the
group walk does not take: the accepted (body, node) pairs are the oracle's,
count for count, and the forces agree, where per-body items are taken at
shifted images (bodies around a corner of the box, so that near nodes lie at
another image on every axis), at the unshifted one, and near the bucket.

Force tolerance: float32 sums of about a thousand terms rounded to 2^-24,
random-walk error below 1e-5 of the largest force."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
N = 98304 + 1707


def _bodies(kind):
    rng = np.random.default_rng(len(kind))
    if kind == "corner":
        p = rng.normal(0, 0.02, (N, 3)) % 1.0
    elif kind == "pairs":      # close pairs on both sides of the cut d^2 = 1e-7
        half = rng.random((N // 2 + 1, 3))
        p = np.concatenate([half, (half + rng.normal(0, 2e-4, half.shape)) % 1.0])[:N]
    else:
        p = rng.random((N, 3))
    p = p.astype(np.float32)
    p[p >= 1] = 0
    return p


@pytest.mark.parametrize("bpl,warps", [(1, 8), (2, 2)])
@pytest.mark.parametrize("theta", [0.3, 0.5, 0.9])
@pytest.mark.parametrize("kind", ["uniform", "corner", "pairs"])
def test_accepted_pairs_are_the_oracle_s(kind, theta, bpl, warps):
    from cnb import _lib
    from cnb.core.octree import OctreeManager
    p = _bodies(kind)
    codes, _ = orc.compute_codes(p[:, 0], p[:, 1], p[:, 2], 1)
    perm = orc.argsort_stable(codes)
    p, codes = p[perm], codes[perm]
    pos = [np.ascontiguousarray(p[:, k]) for k in range(3)]
    mass = np.full(N, 1.0 / N, np.float32)
    ch, par = orc.build_tree(codes)
    nm, nc, lo, hi = orc.compute_multipoles(*pos, mass, ch, par)
    want, _, _, acc = orc.compute_forces(*pos, ch, nm, nc, lo, hi, theta, 1.0, 0.004, 1.0,
                                         orc.find_root(par), return_accepted=True)
    P = [torch.from_numpy(a).cuda() for a in pos]
    tm = OctreeManager(N, node_table=True, bucket=32 * bpl)
    tm.build(P, torch.from_numpy(mass).cuda(), torch.from_numpy(codes).cuda())
    f = torch.empty((N, 3), device="cuda")
    stats = torch.zeros(4, dtype=torch.int64, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("cnb_forces_grouped", *(q.data_ptr() for q in P), tm.node_table.data_ptr(),
              tm.workspace.data_ptr(), f.data_ptr(), N, theta, None, _lib.MAC_REF_X, bpl, warps, 1.0,
              0.004, 1.0, 0.0, stats.data_ptr(), status.data_ptr(),
              int(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert int(stats[0]) == acc
    assert np.abs(f.cpu().numpy() - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("soft", [0.0, 1e-21, 1e-4])
@pytest.mark.parametrize("mac,n", [(0, 4000), (0, N), (1, 4000), (3, 4000)])
def test_forces_at_vanishing_softening(mac, n, soft):
    """eps^2 zero, subnormal and small: every force is finite (a body does not
    act on itself) and, for the exact test at theta -> 0 on a small system, the
    direct sum (the other tests pick one image for a bucket, which for a pair
    half a box apart to the last bit need not be the direct sum's)."""
    from cnb import _lib
    from cnb.core.octree import OctreeManager
    p = _bodies("pairs")[:n]
    codes, _ = orc.compute_codes(p[:, 0], p[:, 1], p[:, 2], 1)
    perm = orc.argsort_stable(codes)
    p, codes = p[perm], codes[perm]
    P = [torch.from_numpy(np.ascontiguousarray(p[:, k])).cuda() for k in range(3)]
    M = torch.full((n,), 1.0 / n, device="cuda")
    tm = OctreeManager(n, node_table=True, bucket=64)
    tm.build(P, M, torch.from_numpy(codes).cuda())
    f = torch.empty((n, 3), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    theta = 0.5 if n == N else 1e-6
    _lib.call("cnb_forces_grouped", *(q.data_ptr() for q in P), tm.node_table.data_ptr(),
              tm.workspace.data_ptr(), f.data_ptr(), n, theta, None, mac, 2, 4, 1.0, soft, 1.0, 0.0, None,
              status.data_ptr(), int(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    got = f.cpu().numpy()
    assert np.isfinite(got).all()
    if n != N and mac == 0:
        t = np.arange(n)
        want = orc.direct_sum(p[:, 0], p[:, 1], p[:, 2], np.full(n, 1.0 / n, np.float32), t, 1.0, soft)
        scale = np.linalg.norm(want, axis=1)
        # 4000 float32 terms, differences of float32 coordinates exact to 2^-25 at a separation
        # of at least 3e-4: 2e-4 relative, on forces the closest pair dominates
        assert (np.linalg.norm(got - want, axis=1) <= 1e-3 * np.maximum(scale, np.median(scale))).all()
