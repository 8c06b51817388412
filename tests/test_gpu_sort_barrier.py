"""The persistent sort's grid barriers (csrc/sort_persistent.cu), like the
one-sweep sort's look-back, are waits of blocks on one another: bounded, and
reported by CNB_FLAG_WAIT_LIMIT when they give up.  The hook
cnb_ctx_inject_barrier_fault makes one block return at its first barrier
without arriving and shortens the limit, so the others give up within
microseconds; the flag must reach the caller's status word, and after the hook
is reset the same context must sort correctly again."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _sort(ctx, keys):
    from cnb import _lib
    n = keys.size
    K = torch.from_numpy(keys).cuda()
    ko = torch.from_numpy(np.full(n, 7, np.uint64)).cuda()
    po = torch.from_numpy(np.full(n, 0xFFFFFFFF, np.uint32)).cuda()
    status = torch.zeros(2, dtype=torch.int32, device="cuda")
    st = int(torch.cuda.current_stream().cuda_stream)
    _lib.call("cnb_sort_pairs", ctx, K.data_ptr(), ko.data_ptr(), None, po.data_ptr(), n, 63, st)
    for k in range(2):   # a second take finds nothing
        _lib.call("cnb_ctx_take_flags", ctx, status.data_ptr() + 4 * k, st)
    torch.cuda.synchronize()
    assert int(status[1]) == 0
    return int(status[0]), ko.cpu().numpy(), po.cpu().numpy()


def _sorted(keys, got):
    want = np.argsort(keys, kind="stable")
    return (got[2].astype(np.int64) == want).all() and (got[1] == keys[want]).all()


# 9 and 147 blocks, chunks of up to 8 192 and of up to 14 336 keys; with the near-sorted path before it
@pytest.mark.parametrize("adaptive", [False, True])
@pytest.mark.parametrize("n,block", [(9000, 0), (9000, 8), (300007, 60), (1500007, 146)])
def test_a_block_that_never_arrives(n, block, adaptive):
    from cnb import _lib
    keys = np.random.default_rng(n).integers(0, 1 << 63, n, dtype=np.uint64)
    ctx = C.c_void_p()
    _lib.call("cnb_ctx_create", n, C.byref(ctx))
    try:
        _lib.call("cnb_ctx_set_sort_mode", ctx, _lib.SORT_ADAPTIVE if adaptive else _lib.SORT_FULL)
        for _ in range(2):
            _lib.call("cnb_ctx_inject_barrier_fault", ctx, 256, block)
            assert _sort(ctx, keys)[0] & _lib.FLAG_WAIT_LIMIT
            _lib.call("cnb_ctx_inject_barrier_fault", ctx, 0, -1)
            got = _sort(ctx, keys)
            assert got[0] == 0 and _sorted(keys, got)
    finally:
        _lib.load().cnb_ctx_destroy(ctx)


def test_a_short_limit_alone_sorts_or_reports():
    from cnb import _lib
    n = 1200007
    keys = np.random.default_rng(1).integers(0, 1 << 63, n, dtype=np.uint64)
    ctx = C.c_void_p()
    _lib.call("cnb_ctx_create", n, C.byref(ctx))
    try:
        for limit in (1, 16, 1 << 20):
            _lib.call("cnb_ctx_inject_barrier_fault", ctx, limit, -1)
            got = _sort(ctx, keys)
            assert got[0] & _lib.FLAG_WAIT_LIMIT or _sorted(keys, got)
    finally:
        _lib.load().cnb_ctx_destroy(ctx)


PART = r"""
import ctypes as C, sys
import numpy as np, torch
sys.path.insert(0, sys.argv[1])
from cnb import _lib
n = 300007
keys = np.random.default_rng(2).integers(0, 1 << 63, n, dtype=np.uint64)
K = torch.from_numpy(keys).cuda()
ko, po = torch.zeros_like(K), torch.zeros(n, dtype=torch.int32, device="cuda")
status = torch.zeros(1, dtype=torch.int32, device="cuda")
want = np.argsort(keys, kind="stable")
torch.cuda.synchronize()
try:
    part = torch.cuda.GreenContext.create(16, 0)
except RuntimeError as e:
    print("no green contexts:", e)
    sys.exit(0)
for mode in (_lib.SORT_FULL, _lib.SORT_ADAPTIVE):
    ctx = C.c_void_p()
    _lib.call("cnb_ctx_create", n, C.byref(ctx))
    _lib.call("cnb_ctx_set_sort_mode", ctx, mode)
    torch.cuda.synchronize()
    part.set_context()
    s = torch.cuda.Stream()
    _lib.call("cnb_sort_pairs", ctx, K.data_ptr(), ko.data_ptr(), None, po.data_ptr(), n, 63, int(s.cuda_stream))
    _lib.call("cnb_ctx_take_flags", ctx, status.data_ptr(), int(s.cuda_stream))
    s.synchronize()
    part.pop_context()
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert (po.cpu().numpy() == want).all() and (ko.cpu().numpy() == keys[want]).all()
    _lib.load().cnb_ctx_destroy(ctx)
print("sorted")
"""


def test_a_stream_with_part_of_the_gpu():
    """A stream of a green context of 16 multiprocessors does not hold the
    persistent sort's blocks: the one-sweep launches sort there.  (In a process
    of its own: torch keeps a pool of streams that would belong to the part.)"""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", PART, os.path.join(root, "cosmo-nbody_b200")],
                       capture_output=True, text=True, timeout=300)
    if "no green contexts" in r.stdout:
        pytest.skip(r.stdout.strip())
    assert r.returncode == 0 and "sorted" in r.stdout, r.stderr[-2000:]


def test_arguments():
    from cnb import _lib
    lib = _lib.load()
    assert lib.cnb_ctx_inject_barrier_fault(None, 1, -1) == _lib.CNB_E_INVALID_ARG
    ctx = C.c_void_p()
    _lib.call("cnb_ctx_create", 10, C.byref(ctx))
    assert lib.cnb_ctx_inject_barrier_fault(ctx, -1, -1) == _lib.CNB_E_INVALID_ARG
    assert lib.cnb_ctx_inject_barrier_fault(ctx, 0, -2) == _lib.CNB_E_INVALID_ARG
    lib.cnb_ctx_destroy(ctx)
