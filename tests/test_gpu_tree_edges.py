"""The radix-tree search by key prefixes (csrc/tree.cu split_of: masks below 64
shared bits, the reference's tie rule above) against the oracle, and the
bucketed upward pass (csrc/upward_table.cu: two nodes a lane, one a round)
against the one-pass form on the shapes at its limits: full buckets, chains that
form one node a round, roots at either end of the bucket.  Integers and floats
are compared bit for bit."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _chain(k, mirrored):
    """k sorted keys whose tree is a chain, open at one end or the other."""
    a = np.array([0] + [1 << b for b in range(k - 1)], np.uint64)
    return np.uint64((1 << 63) - 1) - a[::-1] if mirrored else a


def _keys(name):
    rng = np.random.default_rng(11)
    if name.startswith("chain"):
        return _chain(int(name[6:]), name[5] == "m")
    if name == "top bit":            # no shared bit at all; the last key has every bit
        return np.array([0, 1, 1 << 62, 1 << 63, (1 << 63) + 1, (1 << 64) - 1], np.uint64)
    if name == "ties":               # runs of equal keys between distinct ones
        return np.sort(rng.integers(0, 50, 3000).astype(np.uint64) << np.uint64(40))
    if name == "all equal":
        return np.full(777, 12345, np.uint64)
    if name == "pairs":              # neighbours that differ in the last bit or not at all
        return np.sort(np.repeat(rng.integers(0, 1 << 40, 700).astype(np.uint64) << np.uint64(1), 2)
                       + np.tile(np.array([0, 1], np.uint64), 700) * rng.integers(0, 2, 1400).astype(np.uint64))
    return np.sort(rng.integers(0, 1 << 63, int(name), dtype=np.uint64))


@pytest.mark.parametrize("name", ["2", "3", "257", "30000", "top bit", "ties", "all equal", "pairs", "chain 64", "chainm64"])
def test_build_matches_the_oracle(name):
    from cnb import _lib
    codes = _keys(name)
    n = codes.size
    want_ch, want_par = orc.build_tree(codes)
    K = torch.from_numpy(codes).cuda()
    ch = torch.full((2 * n - 1, 2), -1, dtype=torch.int32, device="cuda")
    par = torch.full((2 * n - 1,), -1, dtype=torch.int32, device="cuda")
    _lib.call("cnb_build_tree", K.data_ptr(), ch.data_ptr(), par.data_ptr(), n,
              int(torch.cuda.current_stream().cuda_stream))
    np.testing.assert_array_equal(ch.cpu().numpy(), want_ch)
    got = par.cpu().numpy()
    if name in ("ties", "all equal", "pairs"):
        # the tie rule can give a node two parents; which one is written last is open on a GPU
        kids = want_ch[n:].reshape(-1)
        once = np.bincount(kids, minlength=2 * n - 1) <= 1
        np.testing.assert_array_equal(got[once], want_par[once])
    else:
        np.testing.assert_array_equal(got, want_par)


@pytest.mark.parametrize("quad", [False, True])
@pytest.mark.parametrize("name", ["2", "33", "64", "65", "5000", "chain 33", "chainm33", "chain 64", "chainm64"])
def test_bucketed_upward_equals_one_pass_at_its_limits(name, quad):
    from cnb import _lib
    codes = _keys(name)
    n = codes.size
    m = 2 * n - 1
    rng = np.random.default_rng(n)
    c = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    P = [c(rng.random(n).astype(np.float32)) for _ in range(3)]
    M = c((rng.random(n) + 0.1).astype(np.float32))
    K = c(codes)
    st = int(torch.cuda.current_stream().cuda_stream)
    ch = torch.full((m, 2), -1, dtype=torch.int32, device="cuda")
    par = torch.full((m,), -1, dtype=torch.int32, device="cuda")
    rg = torch.zeros((n, 2), dtype=torch.int32, device="cuda")
    cnt = torch.zeros(m, dtype=torch.int32, device="cuda")
    root = torch.zeros(1, dtype=torch.int32, device="cuda")
    ws = torch.zeros(4 + 4 * n, dtype=torch.int32, device="cuda")
    _lib.call("cnb_build_tree_buckets", K.data_ptr(), ch.data_ptr(), par.data_ptr(), rg.data_ptr(), cnt.data_ptr(),
              root.data_ptr(), n, 64, ws.data_ptr(), 0, None, st)
    tables = []
    for buckets in (False, True):
        cnt.zero_()
        table, sums = torch.zeros(16 * m, device="cuda"), torch.zeros(4 * m, device="cuda")
        q = torch.zeros(8 * m, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        bodies = [p.data_ptr() for p in P] + [M.data_ptr(), ch.data_ptr(), par.data_ptr()]
        if buckets:
            _lib.call("cnb_upward_table_buckets", *bodies, ws.data_ptr(), cnt.data_ptr(), table.data_ptr(),
                      sums.data_ptr(), q.data_ptr() if quad else None, n, status.data_ptr(), st)
        elif quad:
            _lib.call("cnb_upward_table_quad", *bodies, cnt.data_ptr(), table.data_ptr(), sums.data_ptr(),
                      q.data_ptr(), n, status.data_ptr(), st)
        else:
            _lib.call("cnb_upward_table", *bodies, cnt.data_ptr(), table.data_ptr(), sums.data_ptr(), n,
                      status.data_ptr(), st)
        assert int(status.item()) == 0
        tables.append((table.cpu().numpy().view(np.uint32), q[8 * n:].cpu().numpy().view(np.uint32)))
    np.testing.assert_array_equal(tables[0][0], tables[1][0])
    np.testing.assert_array_equal(tables[0][1], tables[1][1])
