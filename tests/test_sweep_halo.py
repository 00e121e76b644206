"""The window rule of the sweep kernel (csrc/mgp_sweep.cu): a CTA that makes K
sweeps of a tile in one launch computes every cell of its window, the tile and
4 K + 2 columns left, 4 K right and 4 K + 2 rows either side, clipped to the
domain.  Here the cells a tile's result depends on are walked backwards through
the sweep's passes (corners, edge colours, interior colours, ghost fill), for
every tile of partitions at the largest tile widths, and must lie inside that
window."""
import numpy as np
import pytest

COLOURS = ((0, 0), (1, 1), (1, 0), (0, 1))


def _dilate(m, left, right, down, up):
    """m shifted onto every offset of the box [-left, right] x [-down, up] (axis 0 is y)."""
    out = m.copy()
    for dj in range(-down, up + 1):
        for di in range(-left, right + 1):
            s = np.zeros_like(m)
            ys, yd = slice(max(0, -dj), m.shape[0] - max(0, dj)), slice(max(0, dj), m.shape[0] - max(0, -dj))
            xs, xd = slice(max(0, -di), m.shape[1] - max(0, di)), slice(max(0, di), m.shape[1] - max(0, -di))
            s[yd, xd] = m[ys, xs]
            out |= s
    return out


def _needed(nx, ny, tile, K):
    """Cells whose value before the launch the tile's cells depend on."""
    X0, X1, Y0, Y1 = tile
    need = np.zeros((ny, nx), bool)
    need[Y0:Y1, X0:X1] = True
    jj, ii = np.mgrid[0:ny, 0:nx]
    xl, xh, yl, yh = ii == 0, ii == nx - 1, jj == 0, jj == ny - 1
    ex, ey = xl | xh, yl | yh

    def passed(mask):
        nonlocal need
        u = need & mask
        need = need | _dilate(u & ~ex & ~ey, 1, 1, 1, 1)
        need |= _dilate(u & yl & ~ex, 1, 1, 0, 2) | _dilate(u & yh & ~ex, 1, 1, 2, 0)
        need |= _dilate(u & xl & ~ey, 0, 2, 1, 1) | _dilate(u & xh & ~ey, 2, 0, 1, 1)
        need |= _dilate(u & xl & yl, 0, 2, 0, 2) | _dilate(u & xh & yl, 2, 0, 0, 2)
        need |= _dilate(u & xl & yh, 0, 2, 2, 0) | _dilate(u & xh & yh, 2, 0, 2, 0)

    for _ in range(K):
        passed(ex & ey)
        for part in (ex ^ ey, ~ex & ~ey):
            for ci, cj in reversed(COLOURS):
                passed(part & (ii % 2 == ci) & (jj % 2 == cj))
        # Dirichlet ghosts read three cells inward from the side at the sweep's start
        need |= _dilate(need & yl, 0, 0, 0, 2) | _dilate(need & yh, 0, 0, 2, 0)
        need |= _dilate(need & xl, 0, 2, 0, 0) | _dilate(need & xh, 2, 0, 0, 0)
    return need


def _tiles(n, g):
    h = (n + 1) // 2
    return [(2 * (t * h // g), min(n, 2 * ((t + 1) * h // g))) for t in range(g)]


def _even_tiles(n, g):
    """The large tiles' bounds: pairs of cells, the first h % g tiles one pair wider."""
    h = (n + 1) // 2
    lo = [2 * (t * (h // g) + min(t, h % g)) for t in range(g)]
    return [(a, min(n, a + 2 * (h // g + (t < h % g)))) for t, a in enumerate(lo)]


@pytest.mark.parametrize("WX,wy", [(64, 56), (64, 32), (32, 48)])
@pytest.mark.parametrize("K", [1, 2, 4])
@pytest.mark.parametrize("nx,ny", [(130, 118), (131, 117), (65, 96), (200, 33), (66, 67), (97, 34), (64, 70)])
def test_window_holds_what_the_tile_needs(nx, ny, K, WX, wy):
    tx, ty = WX - (8 * K + 2), wy - (8 * K + 4)
    if tx < 8 or ty < 8:
        pytest.skip("no such tile")
    gx = 1 if nx <= WX else -(-((nx + 1) // 2) // (tx // 2))
    gy = 1 if ny <= wy else -(-((ny + 1) // 2) // (ty // 2))
    for X0, X1 in _tiles(nx, gx):
        for Y0, Y1 in _tiles(ny, gy):
            ox, wx1 = max(0, X0 - (4 * K + 2)), min(nx, X1 + 4 * K)
            oy, wy1 = max(0, Y0 - (4 * K + 2)), min(ny, Y1 + 4 * K + 2)
            assert 0 < X1 - X0 and 0 < Y1 - Y0 and wx1 - ox <= WX and wy1 - oy <= wy and ox % 2 == 0 and oy % 2 == 0
            need = _needed(nx, ny, (X0, X1, Y0, Y1), K)
            need[oy:wy1, ox:wx1] = False
            assert not need.any(), (X0, X1, Y0, Y1)


@pytest.mark.parametrize("nx,ny", [(190, 100), (191, 101), (200, 97), (182, 84), (183, 120), (120, 200), (60, 90), (300, 40)])
def test_large_tiles_cover_the_grid_and_their_windows_hold_what_they_need(nx, ny):
    """The one-sweep tiles of a large level (sweep_large_tiles): a frame of bands with the halo above, and inside it
    tiles that need 4 columns left, 2 right and 4 rows either side."""
    WX, WY = 64, 32
    b0, b1, b = WX - 4, WX - 6, WY - 6
    if nx < b0 + b1 + WX or ny < 2 * b + WY:
        regions = [(0, nx, 0, ny, WX if nx <= WX else 54, WY if ny <= WY else 20, False)]
    else:
        xr, yt = (nx - b1 + 1) & ~1, (ny - b + 1) & ~1
        regions = [(0, nx, 0, b, 54, b, False), (0, nx, yt, ny, 54, b, False), (0, b0, b, yt, b0, 20, False),
                   (xr, nx, b, yt, b1, 20, False), (b0, xr, b, yt, WX - 6, WY - 8, True)]
    seen = np.zeros((ny, nx), int)
    for x0, x1, y0, y1, tx, ty, inner in regions:
        gx, gy = (-(-((n + 1) // 2) // (t // 2)) for n, t in ((x1 - x0, tx), (y1 - y0, ty)))
        for X0, X1 in _even_tiles(x1 - x0, gx):
            for Y0, Y1 in _even_tiles(y1 - y0, gy):
                X, Y = (x0 + X0, x0 + X1), (y0 + Y0, y0 + Y1)
                seen[Y[0]:Y[1], X[0]:X[1]] += 1
                l, r, d, u = (4, 2, 4, 4) if inner else (6, 4, 6, 6)
                if inner:   # the whole window is loaded without bounds, and swept as interior cells
                    assert X[0] - l >= 1 and X[0] - l + WX <= nx - 1 and Y[0] - d >= 1 and Y[0] - d + WY <= ny - 1
                ox, wx1, oy, wy1 = max(0, X[0] - l), min(nx, X[1] + r), max(0, Y[0] - d), min(ny, Y[1] + u)
                assert wx1 - ox <= WX and wy1 - oy <= WY and ox % 2 == 0 and oy % 2 == 0
                need = _needed(nx, ny, X + Y, 1)
                need[oy:wy1, ox:wx1] = False
                assert not need.any(), (X, Y)
    assert (seen == 1).all()
