"""The controller's mean accelerations formed by a warp for its 32 buckets
(csrc/controller.cu: rows of 64 bodies, larger buckets one thread each) against
the oracle's features and network, and the order the buckets are handed out in
(csrc/forces_grouped.cu k_order_buckets): a stable counting sort by theta."""
import numpy as np
import pytest
import torch

from oracle import mlp

pytestmark = pytest.mark.gpu


def st():
    return int(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1000, 8192, 8193, 50001])
@pytest.mark.parametrize("spread", ["uniform", "one bin", "outside"])
def test_order_is_a_stable_counting_sort(n, spread):
    from cnb import _lib
    rng = np.random.default_rng(n)
    t = {"uniform": rng.uniform(0.2, 1.0, n), "one bin": np.full(n, 0.5),
         "outside": rng.uniform(-3.0, 4.0, n)}[spread].astype(np.float32)
    T = torch.from_numpy(t).cuda()
    ws = torch.tensor([n, 0, 0, 0], dtype=torch.int32, device="cuda")
    order = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    _lib.call("cnb_order_buckets", T.data_ptr(), ws.data_ptr(), order.data_ptr(), st())
    bins = np.clip(((t - np.float32(0.2)) * np.float32(32 / np.float32(0.8))).astype(np.int32), 0, 31)
    np.testing.assert_array_equal(order.cpu().numpy(), np.argsort(bins, kind="stable"))


@pytest.mark.parametrize("bucket", [1, 31, 64, 65, 300])
@pytest.mark.parametrize("permuted", [False, True])
def test_theta_of_buckets_of_every_size(bucket, permuted):
    """theta from the fused kernel against the oracle's features through the
    oracle's network in the same bfloat16 weights: the features agree to 1e-4
    (their own test) and the network turns that into less than 2e-4."""
    from cnb import _lib
    from cnb.controller import ThetaController
    from cnb.core.engine import SimulationEngine
    from cnb.core.state import SimulationState
    from cnb.utils import config as cfgmod
    from cnb.utils.cosmology import zeldovich_arrays
    cfg = cfgmod.make(N_GRID=12, SOFTENING=0.04, THETA=0.5, KEY_MODE="morton63", FORCE_MODE="grouped", MAC="periodic")
    pos, vel = zeldovich_arrays(12, 5)
    eng = SimulationEngine(cfg, SimulationState(12 ** 3, pos, vel), camera=False)
    eng.forces_only()
    tm, n = eng.tree_manager, eng.state.n
    ws = torch.zeros(4 + 4 * n, dtype=torch.int32, device="cuda")
    _lib.call("cnb_make_buckets", tm.ranges.data_ptr(), tm.parent.data_ptr(), n, bucket, ws.data_ptr(), st())
    nb = int(ws[0])
    acc = eng.state.force.clone()
    perm = torch.from_numpy(np.random.default_rng(1).permutation(n).astype(np.uint32)).cuda() if permuted else None
    flat = tm.node_table.cpu().numpy().reshape(-1, 4)
    m = flat.shape[0] // 4
    rec, aabb = flat[:2 * m].reshape(m, 2, 4), flat[2 * m:].reshape(m, 2, 4)
    bk = ws[4:4 + 4 * nb].view(-1, 4).cpu().numpy()
    assert bk[:, 1].max() <= bucket
    perm_h = perm.cpu().numpy() if permuted else np.arange(n, dtype=np.uint32)
    parents, acc_h = tm.parent.cpu().numpy(), acc.cpu().numpy()
    want = np.stack([mlp.bucket_features(rec, aabb, parents, b, acc_h, perm_h) for b in bk])
    ctl = ThetaController(seed=3)
    ctl.mean = torch.from_numpy(want.mean(0).astype(np.float32)).cuda()
    ctl.std = torch.from_numpy(want.std(0).astype(np.float32) + 1e-1).cuda()
    got = ctl.theta_for_buckets(tm.node_table, tm.parent, ws, n, acc, perm)[:nb].cpu().numpy()
    th, _ = mlp.forward(mlp.bf16_round(ctl.folded_params().cpu().numpy()), want.astype(np.float32), hidden_bf16=True)
    # 2e-4 as in the features' test, and a hidden unit's bfloat16 rounding that the features' 1e-4
    # can tip: 2^-9 of a unit times its weights, below 2e-3 in theta
    np.testing.assert_allclose(got, th, rtol=0, atol=2.2e-3)
