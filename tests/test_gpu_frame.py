"""Splat and colouring where their kernels branch: warps whose particles share
pixels, particle counts off the block size, frames whose sizes and addresses do
not allow four pixels a load.

Tolerances: 1.2e-4 of the brightest pixel, whose 60 000 weights arrive as at most
1 880 warp sums, each addition rounded to 2^-24 of the partial sum; the weights
are added up in float64 here (the oracle's float32 sum of 60 000 nearly equal
weights is itself 2e-4 off); colours as the other colour test."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _mvp(width, height):
    from cnb.utils import config as cfgmod
    from cnb.utils.visualizer import get_mvp_matrix
    return get_mvp_matrix(3, (0.5, 0.5, 0.5), 1.0, cfgmod.make(N_GRID=16), aspect=width / height)


def _splat64(p, mvp, width, height):
    """The oracle's pixels and weights (float32 clip coordinates), added in float64."""
    f = np.float32
    clip = [((mvp[r, 0] * p[:, 0] + mvp[r, 1] * p[:, 1]).astype(f) + mvp[r, 2] * p[:, 2]).astype(f) + mvp[r, 3]
            for r in (0, 1, 3)]
    x, y, w = (c.astype(np.float64) for c in clip)
    sx, sy = (x * (1.0 / w) + 1.0) * 0.5 * width, (1.0 - y * (1.0 / w)) * 0.5 * height
    ok = (w > 0.01) & (sx >= 0) & (sx < width) & (sy >= 0) & (sy < height)
    grid = np.zeros(width * height)
    np.add.at(grid, sy[ok].astype(np.int64) * width + sx[ok].astype(np.int64),
              (2.5 * (1.0 / w[ok])).astype(f).astype(np.float64))
    return grid.reshape(height, width)


@pytest.mark.parametrize("n", [1, 31, 511, 512, 513, 60000])
@pytest.mark.parametrize("width,height", [(1, 1), (2, 3), (16, 16), (257, 129)])
@pytest.mark.parametrize("spread", [0.3, 1e-3, 0.0])
def test_splat(n, width, height, spread):
    from cnb import _lib
    rng = np.random.default_rng(n + width)
    p = np.clip(0.5 + rng.normal(0, 1, (n, 3)) * spread, 0, 0.999).astype(np.float32)
    p = np.ascontiguousarray(p[np.lexsort(p.T)])      # neighbours on neighbouring lanes
    mvp = _mvp(width, height)
    grid = torch.zeros((height, width), device="cuda")
    P = [torch.from_numpy(np.ascontiguousarray(p[:, k])).cuda() for k in range(3)]
    M = torch.from_numpy(mvp).cuda()
    _lib.call("cnb_render_density", *(q.data_ptr() for q in P), grid.data_ptr(), M.data_ptr(), n, width, height,
              int(torch.cuda.current_stream().cuda_stream))
    got = grid.cpu().numpy().astype(np.float64)
    want = _splat64(p, mvp, width, height)
    # the same pixels as the oracle's
    np.testing.assert_array_equal(got != 0, orc.render_density(p[:, 0], p[:, 1], p[:, 2], mvp, width, height)[0] != 0)
    assert np.abs(got - want).max() <= 2 * 6e-5 * max(want.max(), 1.0)


@pytest.mark.parametrize("width,height,off", [(1, 1, 0), (3, 1, 0), (16, 9, 0), (17, 5, 0), (64, 32, 1), (33, 7, 3)])
def test_colour_of_odd_frames(width, height, off):
    from cnb import _lib
    rng = np.random.default_rng(width)
    grid = rng.random((height, width)).astype(np.float32) ** 8 * 40
    grid[rng.random(grid.shape) < 0.5] = 0.0
    n = width * height
    # off: arrays that start off a 16-byte boundary
    g = torch.zeros(n + 8, device="cuda")[off:off + n]
    g.copy_(torch.from_numpy(grid.ravel()))
    rgb = torch.full((3 * n + 8,), -1.0, device="cuda")
    rgb8 = torch.full((3 * n + 8,), 77, dtype=torch.uint8, device="cuda")
    scratch = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = int(torch.cuda.current_stream().cuda_stream)
    _lib.call("cnb_colorize", g.data_ptr(), width, height, rgb[off:].data_ptr(), rgb8[off:].data_ptr(),
              scratch.data_ptr(), st)
    torch.cuda.synchronize()
    want, want8 = orc.colorize(grid)
    got = rgb[off:off + 3 * n].cpu().numpy().reshape(height, width, 3)
    np.testing.assert_allclose(got, want, rtol=0, atol=2e-5)
    got8 = rgb8[off:off + 3 * n].cpu().numpy().reshape(height, width, 3).astype(int)
    assert np.abs(got8 - np.asarray(want8).astype(int)).max() <= 1
    assert (rgb[off + 3 * n:] == -1).all() and (rgb8[off + 3 * n:] == 77).all()
    assert (rgb[:off] == -1).all() and (rgb8[:off] == 77).all()
