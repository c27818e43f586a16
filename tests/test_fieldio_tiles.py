"""The field copies' loops (gf_fieldio.cu: tiles of 32 cells, eight warps, a warp per field in the gather and per cell
in the scatter) restated thread by thread: every read and write inside its array, every element written once."""
import numpy as np
import pytest

CELLS, WARPS, IN_FLIGHT = 32, 8, 8


def gather(fields, T, p, n, nS, ld, grid):
    ne = nS + 2
    lt = ne | 1
    src = list(fields) + [T, p]
    y = np.full(n * ld, np.nan)
    for b in range(grid):
        for c0 in range(b * CELLS, n, grid * CELLS):
            nc = min(n - c0, CELLS)
            tile = np.full(CELLS * lt, np.nan)
            for wid in range(WARPS):
                for e0 in range(wid, ne, WARPS * IN_FLIGHT):
                    for e in range(e0, e0 + IN_FLIGHT * WARPS, WARPS):
                        for l in range(32):
                            if e < ne and l < nc:
                                assert np.isnan(tile[l * lt + e])
                                tile[l * lt + e] = src[e][c0 + l]
            for wid in range(WARPS):
                for j in range(wid, nc, WARPS):
                    for l in range(32):
                        for e in range(l, ne, 32):
                            assert np.isnan(y[(c0 + j) * ld + e])
                            y[(c0 + j) * ld + e] = tile[j * lt + e]
    return y.reshape(n, ld)


def scatter(RR, n, nS, ld, grid):
    lt = nS | 1
    out = np.full((nS, n), np.nan)
    for b in range(grid):
        for c0 in range(b * CELLS, n, grid * CELLS):
            nc = min(n - c0, CELLS)
            tile = np.full(CELLS * lt, np.nan)
            for wid in range(WARPS):
                for l in range(32):
                    for i0 in range(l, nS, 64):
                        for j in range(wid, wid + CELLS, WARPS):
                            for i in (i0, i0 + 32):
                                if j < nc and i < nS:
                                    assert np.isnan(tile[j * lt + i])
                                    tile[j * lt + i] = RR[(c0 + j) * ld + i]
            for wid in range(WARPS):
                for l in range(nc):
                    for i in range(wid, nS, WARPS):
                        assert np.isnan(out[i, c0 + l])
                        out[i, c0 + l] = tile[l * lt + i]
    return out


@pytest.mark.parametrize("n, nS, ld, grid", [(1, 1, 3, 1), (31, 10, 12, 1), (33, 62, 66, 2), (70, 63, 65, 1), (97, 7, 9, 2),
                                             (40, 33, 40, 1), (5, 300, 302, 1)])
def test_tiles(n, nS, ld, grid):
    rng = np.random.default_rng(n * 1000 + nS)
    fields = [rng.standard_normal(n) for _ in range(nS)]
    T, p = rng.uniform(300, 3000, n), rng.uniform(1e5, 4e6, n)
    y = gather(fields, T, p, n, nS, ld, grid)
    assert np.array_equal(y[:, :nS + 2], np.column_stack(fields + [T, p])) and np.isnan(y[:, nS + 2:]).all()
    RR = rng.standard_normal((n, ld))
    assert np.array_equal(scatter(RR.ravel(), n, nS, ld, grid), RR[:, :nS].T)
