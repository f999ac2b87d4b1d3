"""The return map of crushed points in 64 bits against the oracle's SVD form,
over the deformations it branches on: nearly undeformed, moderate and large
strain, equal principal stretches (all three, two), tension and recompaction
(apex), strong compression and inversion (det F below the polar form's limit)."""
import ctypes

import numpy as np
import pytest

from icempm_3dm_b200 import PRECISION_FP64_SVD64, PRECISION_MIXED, MPMHandle
from icempm_3dm_b200._lib import LIB
from icempm_3dm_b200 import generator as gen
from icempm_3dm_b200.layout import FE00, IDX_JP_INV, IDX_UTILITY, STATUS_CRUSHED
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _rotations(rng, n):
    q, _ = np.linalg.qr(rng.standard_normal((n, 3, 3)))
    q[:, :, 0] *= np.sign(np.linalg.det(q))[:, None]
    return q


def _deformations(rng, n):
    """(n, 3, 3) F = U diag(s) V^T, a ninth of them of each kind."""
    s = np.ones((n, 3))
    kind = np.arange(n) % 9
    g = rng.standard_normal((n, 3))
    s += np.select([kind == 0, kind == 1, kind == 2], [1e-6, 1e-3, 2e-2], 0.0)[:, None] * g
    s[kind == 3] = np.exp(0.4 * g[kind == 3])                       # large strain
    s[kind == 4] = 1.0 + 1e-2 * np.abs(g[kind == 4][:, :1])          # equal stretches, tension
    s[kind == 5] = 1.0 - 1e-2 * np.abs(g[kind == 5][:, :1])          # equal stretches, compression
    s[kind == 6, 2] = 0.97                                          # two equal
    s[kind == 7] = [0.5, 0.4, 0.2]                                  # det 0.04: the SVD form
    s[kind == 8, 2] *= -0.9                                         # inverted: the SVD form
    return np.einsum("nij,nj,nkj->nik", _rotations(rng, n), s, _rotations(rng, n)), kind


def _block(inverted):
    prms, soa, _ = gen.small_block(n=1801, seed=3)
    rng = np.random.default_rng(4)
    n = soa.shape[1]
    F, kind = _deformations(rng, n)
    if not inverted:
        F[kind == 8] = np.eye(3)
    soa[FE00:FE00 + 9] = F.reshape(n, 9).T
    soa[IDX_JP_INV] = np.where(rng.random(n) < 0.3, 0.99, 1.01)
    soa[IDX_UTILITY] = np.full(n, STATUS_CRUSHED, dtype=np.int64).view(np.float64)
    prms.InitialTimeStep = 1e-10          # F_tr = F to 1e-9: the stresses of these states would move the points
    LIB.mpm_params_compute_helper_variables(ctypes.byref(prms))
    return prms, soa, kind


# The oracle's 24 Jacobi rotations leave an error of some 1e-14 in U and V;
# near-equal stretches do not amplify it, since F' is smooth in F there.
# Measured 2e-14; mixed holds F - I in 32 bits (2^-24 of |F - I| <= 2: 1.2e-7
# per entry, on input and output).
# The 32-bit stress of the mixed P2G has no value for det F < 0.
@pytest.mark.parametrize("precision,bound", [(PRECISION_FP64_SVD64, 1e-12), (PRECISION_MIXED, 1e-6)])
def test_return_map_over_all_branches(precision, bound):
    prms, soa, kind = _block(inverted=precision != PRECISION_MIXED)
    n = soa.shape[1]
    sim = po.OracleSim(prms, soa.copy(), n, svd_mode=1)
    _, err = sim.step(1)
    assert err == 0
    with MPMHandle(prms, n, precision) as h:
        h.upload(soa)
        h.step(1)
        out = h.download()
    ref = sim.soa
    good = np.isfinite(ref[FE00:FE00 + 9]).all(axis=0)
    assert good.sum() > 0.8 * n
    for k in range(9):
        m = good & (kind == k)
        d = np.abs(out[FE00:FE00 + 9, m] - ref[FE00:FE00 + 9, m]).max()
        assert d < bound, (k, d)
        # Jp_inv is scaled by 1 / det F, whose relative error is tr(F^-1 dF) <= 3 |dF| / smallest stretch
        smin = np.linalg.svd(soa[FE00:FE00 + 9, m].T.reshape(-1, 3, 3), compute_uv=False)[:, 2]
        dj = (np.abs(out[IDX_JP_INV, m] / ref[IDX_JP_INV, m] - 1) * np.minimum(smin, 1)).max()
        assert dj < bound, (k, dj)
