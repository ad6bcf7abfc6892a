"""Host-side check of the point kernels' work map (WarpMap, warp_map and
warp_point of waveqlab3d_q_gpu_b200/csrc/wql3d_point.cuh), restated here: over
many block sizes every point belongs to exactly one lane, and no warp mixes
boundary columns (the first and last six) with whole warps of central ones.
No GPU is involved."""
import numpy as np
import pytest

EDGE = 6


def warp_map(nx, ny):
    m = (nx - 2 * EDGE) // 32
    ec = nx - 32 * m
    if ec > 32:
        m += 1
        ec = 2 * EDGE
    e = 1 if ec <= 16 else 2
    return m, ec, e, 2 * m + e, (ny + 1) // 2


def points(nx, ny, nz):
    m, ec, e, per, pairs = warp_map(nx, ny)
    w = np.arange(per * pairs * nz)[:, None]
    lane = np.arange(32)[None, :]
    g, k = w // per, w % per
    zi = g // pairs
    z = zi + 1 + 0 * lane
    y = 2 * (g - zi * pairs) + 1 + 0 * lane
    main = (k < 2 * m) & (lane >= 0)
    row = (k >= m).astype(int) if m else 0 * k
    xm = EDGE + 1 + 32 * (k - row * m) + lane
    ym = y + row
    okm = (ym <= ny) & (xm <= nx - EDGE)
    if e == 1:
        r = (lane >= ec).astype(int) + 0 * k
        c = lane - r * ec
        ye = y + r
    else:
        c = lane + 0 * k
        ye = y + (k - 2 * m)
    xe = np.where(c < EDGE, c + 1, nx - ec + 1 + c)
    oke = (c < ec) & (ye <= ny)
    return main, np.where(main, xm, xe), np.where(main, ym, ye), z, np.where(main, okm, oke)


@pytest.mark.parametrize("ny,nz", [(13, 13), (14, 15)])
def test_every_point_once(ny, nz):
    for nx in list(range(13, 121)) + [128, 145, 176, 201, 224, 300]:
        main, x, y, z, ok = points(nx, ny, nz)
        assert x[ok].min() >= 1 and x[ok].max() <= nx and z.max() <= nz
        idx = (x[ok] - 1) + nx * ((y[ok] - 1) + ny * (z[ok] - 1))
        assert len(idx) == nx * ny * nz and len(np.unique(idx)) == len(idx), nx
        inner = (x > EDGE) & (x <= nx - EDGE)
        assert np.all(inner[main & ok])
