"""FP64 substeps inside one call (velocities in a buffer of their own, the sums
cleared by the update) against substeps one by one (in place): the same states
and forces, and the grid that a call leaves behind holds m and v of its last
substep either way."""
import numpy as np
import pytest

from icempm_3dm_b200 import PRECISION_FP64, PRECISION_FP64_SVD64, MPMHandle
from icempm_3dm_b200.layout import BP00, FE00, POSX, VELX
from tests.helpers import perturbed_block, util_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_FP64_SVD64])
@pytest.mark.parametrize("n", [1, 65, 3000])
def test_substeps_together_and_apart(precision, n):
    prms, soa = perturbed_block(n=max(n, 500), seed=5, ind_velocity=1.0)
    soa = np.ascontiguousarray(soa[:, :n])
    steps = 6
    got = []
    for calls in ([steps], [1] * steps, [4, 2]):
        with MPMHandle(prms, n, precision) as h:
            h.upload(soa)
            h.sort()
            hist = np.concatenate([h.step(c) for c in calls])
            got.append((hist, h.download(), h.grid(0), h.active_nodes()))
    ref = got[1]
    assert ref[3] > 0
    for hist, out, grid, active in got:
        # the order of the FP64 atomics: 1e-16 of the sums, over six substeps
        assert np.abs(hist - ref[0]).max() <= 1e-10 * max(np.abs(ref[0]).max(), 1e-300)
        for row, k in ((POSX, 3), (VELX, 3), (FE00, 9), (BP00, 9)):
            scale = np.abs(ref[1][row:row + k]).max()
            assert np.abs(out[row:row + k] - ref[1][row:row + k]).max() <= 1e-9 * scale
        assert np.array_equal(util_bits(out), util_bits(ref[1]))
        assert active == ref[3]
        for c in range(4):
            assert np.abs(grid[c] - ref[2][c]).max() <= 1e-9 * max(np.abs(ref[2][c]).max(), 1e-300)
