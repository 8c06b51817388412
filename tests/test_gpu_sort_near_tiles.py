"""The near-sorted path's tiles of 1024, 2048 and 4096 keys (csrc/sort_near.cu):
keys displaced across tile edges, in tiles with one key, and on both sides of
the sizes where the tile changes; permutation and keys equal to numpy's stable
argsort, and the path itself must have been taken."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025, 2049, 131071, 131072, 131073, 133121, 4194303, 4194304, 4194305])
@pytest.mark.parametrize("moved", [0, 7, 900])
def test_displaced_keys_at_the_tile_edges(n, moved):
    from cnb import _lib
    tile = 1024 if n <= 1 << 17 else 2048 if n <= 1 << 22 else 4096
    rng = np.random.default_rng(n + moved)
    keys = np.sort(rng.integers(0, 1 << 62, n, dtype=np.uint64))
    if n > 4:
        k = min(moved, n // 50)
        at = rng.choice(n, k, replace=False)
        if k:
            # some at the first and last key of a tile, to far places and next door
            edge = at[: k // 2] // tile * tile
            keys[edge] = rng.integers(0, 1 << 62, edge.size, dtype=np.uint64)
            last = np.minimum(at[k // 2:] // tile * tile + tile - 1, n - 2)
            keys[last], keys[last + 1] = keys[last + 1].copy(), keys[last].copy()
    ctx = C.c_void_p()
    _lib.call("cnb_ctx_create", n, C.byref(ctx))
    try:
        _lib.call("cnb_ctx_set_sort_mode", ctx, 1)
        st = int(torch.cuda.current_stream().cuda_stream)
        K = torch.from_numpy(keys.view(np.int64).copy()).cuda()
        out, perm = torch.zeros_like(K), torch.zeros(n, dtype=torch.int32, device="cuda")
        _lib.call("cnb_sort_pairs", ctx, K.data_ptr(), out.data_ptr(), None, perm.data_ptr(), n, 63, st)
        torch.cuda.synchronize()
        want = np.argsort(keys, kind="stable")
        np.testing.assert_array_equal(perm.cpu().numpy(), want)
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), keys[want])
        stats = (C.c_int64 * 2)()
        _lib.call("cnb_ctx_sort_stats", ctx, stats)
        assert (int(stats[0]), int(stats[1])) == (1, 0) or n < 2
    finally:
        _lib.load().cnb_ctx_destroy(ctx)
