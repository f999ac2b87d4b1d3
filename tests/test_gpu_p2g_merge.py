"""P2G's merging of neighbouring lanes (pairs of one cell, chains of cells along
z) against the oracle's P2G, on arrangements where it can go wrong: one to
seven points in a cell, gaps, the end of a column, orders other than the cell
order, disabled points in between, the ends of warps and blocks."""
import numpy as np
import pytest

from icempm_3dm_b200 import PRECISION_FP64, PRECISION_MIXED, MPMHandle
from icempm_3dm_b200.layout import (ACCUM_FIXED, ACCUM_FLOAT, BP00, FE00, IDX_UTILITY, POSX, STATUS_CRUSHED,
                                    STATUS_DISABLED, VELX)
from icempm_3dm_b200 import generator as gen
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _arrangement(kind, n):
    prms, soa, _ = gen.small_block(n=max(n, 64), seed=9)
    soa = np.ascontiguousarray(soa[:, :n])
    rng = np.random.default_rng(n)
    h, gz = prms.cellsize, prms.GridZ
    if kind == "runs":          # cells along z with 1..7 points each, every fifth cell empty
        z, per = 0, []
        while len(per) < n:
            if z % 5 != 4:
                per += [z] * (1 + z % 7)
            z += 1
        cz = np.array(per[:n])
    elif kind == "columns":     # whole columns, so that warps pass from the top of one to the bottom of the next
        cz = np.arange(n)
    else:                       # "shuffled": no two neighbours in order
        cz = rng.permutation(n)
    depth = gz - 3              # base cells 0 .. gz - 3
    col, cz = cz // depth, cz % depth
    nx, ny = prms.GridXTotal - 3, prms.GridY - 3
    cell = np.stack([1 + (col // ny) % nx, col % ny, cz])
    soa[POSX:POSX + 3] = (cell + 0.5 + rng.uniform(0.02, 0.98, (3, n))) * h
    soa[VELX:VELX + 3] = rng.standard_normal((3, n))
    soa[BP00:BP00 + 9] = 5 * rng.standard_normal((9, n))
    soa[FE00:FE00 + 9] += 1e-3 * rng.standard_normal((9, n))
    bits = np.where(rng.random(n) < 0.1, STATUS_CRUSHED, 0).astype(np.int64)
    bits[rng.random(n) < 0.05] |= STATUS_DISABLED
    soa[IDX_UTILITY] = bits.view(np.float64)
    return prms, soa


# FP64: the sums differ by their order (some 50 terms of 1.1e-16), and the stress
# of a strain of 1e-3 by the rounding of F F^T, 1.1e-16 / 1e-3 over some five
# operations (bound 1e-12 of the largest sum). Mixed: a position held to 2^-21
# cells moves a weight by 7e-7 along each axis, and payload and weights take
# some ten roundings of 6e-8 (bound 4e-6); the fixed-point sums add 2^-44.
@pytest.mark.parametrize("kind", ["runs", "columns", "shuffled"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 1000])
def test_p2g_merge(kind, n):
    prms, soa = _arrangement(kind, n)
    ref, err = po.p2g(prms, soa, n)
    assert err == 0
    for precision, accum, bound in ((PRECISION_FP64, ACCUM_FLOAT, 1e-12), (PRECISION_MIXED, ACCUM_FLOAT, 4e-6),
                                    (PRECISION_MIXED, ACCUM_FIXED, 4e-6)):
        with MPMHandle(prms, n, precision) as h:
            h.set_grid_accumulation(accum)
            h.upload(soa)
            h.reset_grid()
            h.p2g()
            assert h.error() == 0
            got = h.grid(0)
        for k in range(4):
            scale = np.abs(ref[k]).max()
            assert np.abs(got[k] - ref[k]).max() <= bound * scale + 1e-300, (precision, accum, k)


def test_p2g_of_points_outside_the_grid():
    """The part of a stencil that lies in the grid, for points that leave it on
    one to three sides, among them coordinates between -0.5 and 0.5 cells: their
    base is 0 and their weights are not in [0, 1]."""
    prms, soa, _ = gen.small_block(n=1000, seed=9, halo=3)
    h = prms.cellsize
    at = [[lo, -0.9, -0.3, 0.2, 4.7, g - 1.7, g - 0.6, g + 0.4]
          for lo, g in ((-3.8, prms.GridXTotal), (-1.4, prms.GridY), (-1.4, prms.GridZ))]
    x = np.stack(np.meshgrid(*at, indexing="ij")).reshape(3, -1)
    n = x.shape[1]
    rng = np.random.default_rng(1)
    soa = np.ascontiguousarray(np.repeat(soa[:, :1], n, axis=1))
    soa[POSX:POSX + 3] = x * h
    soa[VELX:VELX + 3] = rng.standard_normal((3, n))
    soa[BP00:BP00 + 9] = 5 * rng.standard_normal((9, n))
    for k in (n, 300, 1):
        ref, err = po.p2g(prms, soa, k)
        assert err != 0
        with MPMHandle(prms, n, PRECISION_FP64) as hd:
            hd.upload(np.ascontiguousarray(soa[:, :k]))
            hd.reset_grid()
            hd.p2g()
            assert 70 <= hd.error() <= 75
            got = hd.grid(0)
        for c in range(4):
            # the order of the sums, as above
            assert np.abs(got[c] - ref[c]).max() <= 1e-12 * np.abs(ref[c]).max() + 1e-300
