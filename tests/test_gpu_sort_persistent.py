"""The full radix sort as one cooperative launch (csrc/sort_persistent.cu):
chunk edges, the sizes where its form changes and past which the one-sweep
launches take over, key widths with one to eight passes, index input, in-place
buffers, and as the fallback behind the near-sorted path."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
SMS = 148


def _sort(ctx, k, bits, mode, idx=None, in_place=False):
    from cnb import _lib
    st = int(torch.cuda.current_stream().cuda_stream)
    _lib.call("cnb_ctx_set_sort_mode", ctx, _lib.SORT_ADAPTIVE if mode == "adaptive" else _lib.SORT_FULL)
    kin = k.clone()
    kout = kin if in_place else torch.empty_like(k)
    iin = None if idx is None else idx.clone()
    pout = iin if in_place and iin is not None else torch.empty(k.numel(), dtype=torch.int32, device="cuda")
    _lib.call("cnb_sort_pairs", ctx, kin.data_ptr(), kout.data_ptr(), iin.data_ptr() if iin is not None else None,
              pout.data_ptr(), k.numel(), bits, st)
    flags = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("cnb_ctx_take_flags", ctx, flags.data_ptr(), st)
    torch.cuda.synchronize()
    assert int(flags.item()) == 0
    return kout, pout.long()


@pytest.mark.parametrize("n", [1, 31, 1024, 1025, 8191, 8192, 8193, 12289, SMS * 8192, SMS * 8192 + 1,
                               SMS * 14336, SMS * 14336 + 1])
def test_stable_argsort(n):
    from cnb import _lib
    ctx = C.c_void_p()
    _lib.call("cnb_ctx_create", n, C.byref(ctx))
    try:
        rng = np.random.default_rng(n)
        for bits, keep in ((63, 63), (30, 30), (63, 9), (8, 8), (13, 4)):
            # `keep` varying high bits: long runs of equal keys, whose order must stay
            k = rng.integers(0, 1 << keep, n, dtype=np.int64) << (bits - keep)
            k = torch.from_numpy(k).cuda()
            want = torch.sort(k, stable=True)
            got, perm = _sort(ctx, k, bits, "full")
            assert torch.equal(got, want.values) and torch.equal(perm, want.indices)
            got, perm = _sort(ctx, k, bits, "adaptive")
            assert torch.equal(got, want.values) and torch.equal(perm, want.indices)
            idx = torch.randperm(n, device="cuda").to(torch.int32)
            got, perm = _sort(ctx, k, bits, "full", idx, in_place=True)
            assert torch.equal(got, want.values) and torch.equal(perm, idx[want.indices].long())
    finally:
        _lib.call("cnb_ctx_destroy", ctx)


def test_two_contexts_on_two_streams():
    """Cooperative launches of two contexts at once: the device runs them one
    after the other."""
    from cnb import _lib
    n = 500000
    ctxs = [C.c_void_p(), C.c_void_p()]
    for c in ctxs:
        _lib.call("cnb_ctx_create", n, C.byref(c))
    try:
        rng = np.random.default_rng(0)
        keys = [torch.from_numpy(rng.integers(0, 1 << 62, n, dtype=np.int64)).cuda() for _ in ctxs]
        outs = [torch.empty_like(k) for k in keys]
        perms = [torch.empty(n, dtype=torch.int32, device="cuda") for _ in ctxs]
        streams = [torch.cuda.Stream() for _ in ctxs]
        torch.cuda.synchronize()
        for _ in range(10):
            for c, k, o, p, s in zip(ctxs, keys, outs, perms, streams):
                _lib.call("cnb_sort_pairs", c, k.data_ptr(), o.data_ptr(), None, p.data_ptr(), n, 63, s.cuda_stream)
        torch.cuda.synchronize()
        for k, o, p in zip(keys, outs, perms):
            want = torch.sort(k, stable=True)
            assert torch.equal(o, want.values) and torch.equal(p.long(), want.indices)
    finally:
        for c in ctxs:
            _lib.call("cnb_ctx_destroy", c)
