"""The splat's table of a block's pixels: counts around the 2048 particles of a
block, pixels far apart (a table half full of them) and piled up.

Tolerance: a pixel's k weights arrive as sums of at most min(k, 2048) additions
in a block and one a block, each rounded to 2^-24 of the partial sum."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2047, 2048, 2049, 100001])
@pytest.mark.parametrize("width,height", [(4, 4), (33, 7), (1920, 1080), (4099, 4097)])
@pytest.mark.parametrize("ordered", [False, True])
def test_every_particle_once(n, width, height, ordered):
    from cnb import _lib
    rng = np.random.default_rng(n + width)
    # a camera that maps (x, y) to the frame, weights 2.5 / w = 2 exactly
    x = (rng.integers(0, width, n) + 0.5) / width * 2 - 1
    y = 1 - (rng.integers(0, height, n) + 0.5) / height * 2
    p = np.stack([x, y, np.zeros(n)], 1).astype(np.float32)
    if ordered:
        p = p[np.lexsort(p.T)]
    mvp = np.zeros((4, 4), np.float32)
    mvp[0, 0] = mvp[1, 1] = 1.25
    mvp[3, 3] = 1.25
    w = np.float32(1.25)
    sx = (p[:, 0] * w).astype(np.float64) * (1 / 1.25) * 0.5 * width + 0.5 * width
    sy = 0.5 * height - (p[:, 1] * w).astype(np.float64) * (1 / 1.25) * 0.5 * height
    count = np.zeros(width * height)
    np.add.at(count, sy.astype(np.int64) * width + sx.astype(np.int64), 1.0)
    grid = torch.zeros(width * height, device="cuda")
    P = [torch.from_numpy(np.ascontiguousarray(p[:, k])).cuda() for k in range(3)]
    m = torch.from_numpy(mvp).cuda()
    _lib.call("cnb_render_density", *(q.data_ptr() for q in P), grid.data_ptr(), m.data_ptr(), n, width, height,
              int(torch.cuda.current_stream().cuda_stream))
    got = grid.cpu().numpy().astype(np.float64)
    tol = (np.minimum(count, 2048) + n // 2048 + 1) * 2.0 ** -24
    assert (np.abs(got - 2.0 * count) <= tol * 2.0 * count).all()
