"""A handle that a diverged run left non-finite node velocities in gives, after
an upload, what a new handle gives. The points lie on a lattice at exactly half
a cell, so that each touches nodes beyond its own with a weight of exactly 0:
what such an empty node holds must not be left over from an earlier run (0 times
a NaN)."""
import numpy as np
import pytest

from icempm_3dm_b200 import PRECISION_FP64, PRECISION_FP64_SVD64, PRECISION_MIXED, MPMHandle
from icempm_3dm_b200 import generator as gen
from icempm_3dm_b200._lib import MPMError
from icempm_3dm_b200.layout import BP00, FE00, IDX_JP_INV, N_PTS_ARRAYS, POSX, VELX

pytestmark = pytest.mark.gpu

H = 1.0 / 128      # a power of two: x / h - base is exactly 0.5
SIDE = 6
STEPS = 4


def _lattice(first):
    """SIDE^3 points, one per cell at its middle, in a block of twice that size."""
    prms, _, _ = gen.small_block(n=400, seed=1, dims=(2 * SIDE * H, 2 * SIDE * H, 2 * SIDE * H), h=H)
    k = first + np.stack(np.meshgrid(*[np.arange(SIDE)] * 3, indexing="ij")).reshape(3, -1)
    soa = np.zeros((N_PTS_ARRAYS, SIDE ** 3))
    soa[POSX:POSX + 3] = (k + 0.5) * H
    soa[[FE00, FE00 + 4, FE00 + 8]] = 1.0
    soa[IDX_JP_INV] = 1.0
    return prms, soa


def _run(h, api):
    if api == "adjoint":
        return h.adjoint_forward(STEPS, 2)
    if api == "phases":
        for _ in range(STEPS):
            h.reset_grid()
            h.p2g()
            h.update_nodes(0.0, 0.0)
            h.g2p(0)
        return None
    return h.step(STEPS)


@pytest.mark.parametrize("precision,api", [(PRECISION_FP64, "step"), (PRECISION_FP64, "phases"),
                                           (PRECISION_FP64_SVD64, "step"), (PRECISION_FP64_SVD64, "adjoint"),
                                           (PRECISION_MIXED, "step"), (PRECISION_MIXED, "phases"),
                                           (PRECISION_MIXED, "adjoint")])
def test_a_new_run_starts_clean(precision, api):
    prms, soa = _lattice(first=5)
    wild = soa.copy()
    wild[POSX:POSX + 3] += 0.75 * H                # now the lattice's outer nodes have mass
    wild[VELX:VELX + 3] = np.nan
    n = soa.shape[1]

    def clean(h):
        h.update_constants(prms)
        h.upload(soa)
        _run(h, api)
        return h.download()

    with MPMHandle(prms, n, precision) as h:
        ref = clean(h)
    assert np.isfinite(ref).all() and np.abs(ref[VELX + 1]).min() > 0
    with MPMHandle(prms, n, precision) as h:
        h.update_constants(prms)
        h.upload(wild)
        try:
            _run(h, api)                           # FP64: an error code, positions outside the grid
        except MPMError:
            pass
        out = clean(h)
    # The order of the sums of a node: 2^-53 or 2^-24 of at most 27 terms, over
    # four substeps. The lattice falls as one, so C is rounding itself: 4 / h
    # times sums of w v that cancel, hence the scale 4 / h |v| for it.
    tol = 1e-4 if precision == PRECISION_MIXED else 1e-12
    vmax = np.abs(ref[VELX:VELX + 3]).max()
    assert np.isfinite(out).all()
    for row, k, scale in ((POSX, 3, 1.0), (VELX, 3, vmax), (FE00, 9, 1.0), (BP00, 9, 4 / H * vmax)):
        assert np.abs(out[row:row + k] - ref[row:row + k]).max() <= tol * scale
