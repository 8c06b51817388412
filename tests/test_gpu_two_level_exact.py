"""The exact test's bucket form with super-buckets (cnb_forces_two_level), at
sizes that the walk by groups does not take: the accepted (body, node) pairs are
the oracle's, count for count, also where super-buckets' lists do not fit, and
the second pass gives bit-identical forces.  The engine walks small systems by
groups, and then makes no super-bucket lists.

Force tolerance: float32 sums of about a thousand terms rounded to 2^-24,
random-walk error below 1e-5 of the largest force."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


class Case:
    def __init__(self, n, bpl, clustered):
        from cnb.core.octree import OctreeManager
        rng = np.random.default_rng(n + clustered)
        p = rng.random((n, 3))
        if clustered:
            p[: n // 2] = rng.random((8, 3))[rng.integers(0, 8, n // 2)] + rng.normal(0, 0.01, (n // 2, 3))
        p = (p % 1.0).astype(np.float32)
        p[p >= 1] = 0
        codes, _ = orc.compute_codes(p[:, 0], p[:, 1], p[:, 2], 1)
        perm = orc.argsort_stable(codes)
        self.n, self.bpl = n, bpl
        self.pos = [np.ascontiguousarray(p[perm][:, k]) for k in range(3)]
        self.mass = np.full(n, 1.0 / n, np.float32)
        self.codes = codes[perm]
        self.P = [torch.from_numpy(a).cuda() for a in self.pos]
        self.tm = OctreeManager(n, node_table=True, bucket=32 * bpl)
        self.tm.build(self.P, torch.from_numpy(self.mass).cuda(), torch.from_numpy(self.codes).cuda())

    def oracle(self, theta):
        ch, par = orc.build_tree(self.codes)
        nm, nc, lo, hi = orc.compute_multipoles(*self.pos, self.mass, ch, par)
        want, _, _, acc = orc.compute_forces(*self.pos, ch, nm, nc, lo, hi, theta, 1.0, 0.004, 1.0,
                                             orc.find_root(par), return_accepted=True)
        return want, acc

    def run(self, theta, warps, super_bodies, slots=None):
        from cnb import _lib
        n, tm = self.n, self.tm
        nbytes = _lib.load().cnb_two_level_workspace_bytes(n, super_bodies)
        if slots is not None:   # the layout: header, n records, n body slots, then list slots
            nbytes = 16 + 16 * n + (4 * n + 15) // 16 * 16 + slots * (16 + 4 * 256 + 16 * 2048)
        ws = torch.zeros((nbytes + 15) // 16 * 4, dtype=torch.int32, device="cuda")
        f = torch.full((n, 3), float("nan"), device="cuda")
        stats = torch.zeros(4, dtype=torch.int64, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        _lib.call("cnb_forces_two_level", *(p.data_ptr() for p in self.P), tm.node_table.data_ptr(),
                  tm.ranges.data_ptr(), tm.parent.data_ptr(), tm.workspace.data_ptr(), ws.data_ptr(), nbytes,
                  super_bodies, f.data_ptr(), n, theta, _lib.MAC_REF_X, self.bpl, warps, 1.0, 0.004, 1.0,
                  stats.data_ptr(), status.data_ptr(), int(torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert int(status.item()) == 0
        return f.cpu().numpy(), int(stats[0].item()), ws[:4].cpu().numpy()


@pytest.mark.parametrize("theta", [0.3, 0.6])
@pytest.mark.parametrize("n,bpl,warps,super_bodies,slots", [
    (100011, 2, 2, 512, None), (100011, 1, 8, 1024, None), (98305, 1, 4, 256, None), (100011, 2, 4, 512, 40)])
def test_accepted_pairs_are_the_oracle_s(n, bpl, warps, super_bodies, slots, theta):
    for clustered in (False, True):
        c = Case(n, bpl, clustered)
        want, acc = c.oracle(theta)
        f, pairs, hdr = c.run(theta, warps, super_bodies, slots)
        # at the larger angle most super-buckets have their lists; at the smaller one they may
        # overflow, and their buckets walk from the root
        assert 0 <= hdr[2] <= hdr[0] and (theta < 0.5 or hdr[2] < hdr[0])
        assert slots is None or hdr[0] > slots
        assert pairs == acc
        assert np.abs(f - want).max() <= 1e-5 * np.abs(want).max()


def test_lists_that_do_not_fit():
    """theta = 0: every body meets every body, no list holds that many."""
    c = Case(98305, 2, False)
    f, pairs, hdr = c.run(0.0, 2, 256)
    assert hdr[2] == hdr[0] > 0
    assert pairs == c.n * c.n


@pytest.mark.parametrize("n,bpl,warps,theta", [(98305, 2, 2, 0.5), (98305, 1, 8, 0.3), (110592, 2, 2, 0.5)])
def test_second_pass(n, bpl, warps, theta):
    from cnb import _lib
    c = Case(n, bpl, True)
    out = []
    for every in (0, 3, 1):
        _lib.call("cnb_exact_test_spill", every)
        try:
            out.append(c.run(theta, warps, 512))
        finally:
            _lib.call("cnb_exact_test_spill", 0)
        nb = int(c.tm.workspace[0].item())
        assert not bool(c.tm.workspace[4:4 + 4 * nb].view(-1, 4)[:, 3].any())   # no mark is left
    assert np.isfinite(out[0][0]).all()
    for f, pairs, _ in out[1:]:
        np.testing.assert_array_equal(f.view(np.uint32), out[0][0].view(np.uint32))
        assert pairs == out[0][1]


@pytest.mark.parametrize("n_grid,mac,groups", [(24, "ref_x", True), (47, "ref_x", False),
                                               (24, "ref_x_bucket", False)])
def test_the_engine_makes_no_lists_for_the_groups(n_grid, mac, groups):
    """A small system's force stage is the same launches and node tests with
    super-buckets and without; others make the lists."""
    from cnb import _lib, autotune
    from cnb.core.engine import SimulationEngine
    from cnb.core.state import SimulationState
    from cnb.utils import config as cfgmod
    from cnb.utils.cosmology import zeldovich_arrays
    out = []
    for sb in (0, 512):
        cfg = cfgmod.make(N_GRID=n_grid, SOFTENING=0.5 / n_grid, THETA=0.5, N_STEPS=100, A_START=0.02, A_END=0.22,
                          KEY_MODE="morton63", FORCE_MODE="grouped", MAC=mac, BODIES_PER_LANE=2, BLOCK_WARPS=2,
                          SUPER_BODIES=sb)
        st = SimulationState(n_grid ** 3, *zeldovich_arrays(n_grid, 2))
        eng = SimulationEngine(cfg, st, camera=False)
        eng.forces_only()
        eng.stats.zero_()
        before = _lib.launch_count()
        eng.compute_forces()
        eng.check()
        assert eng.walks_by_groups() == groups
        out.append((_lib.launch_count() - before, eng.stats[:2].tolist(), st.force.clone()))
    if groups:
        assert out[0][:2] == out[1][:2]
        assert bool((out[0][2] == out[1][2]).all())
        report = autotune.tune(eng, use_cache=False, save=False)
        assert report["shape"] == [2, 2, 512]
    else:
        assert out[1][0] == out[0][0] + 1
        assert out[0][1][0] == out[1][1][0]
