"""Device memory that runs out: the handle does without the buffers that only save
time, and gives the same results. The allocations that fail are chosen through a
test hook; no memory is really used up."""
import numpy as np
import pytest

from icempm_3dm_b200 import PRECISION_FP64, PRECISION_FP64_SVD64, PRECISION_MIXED, MPMHandle
from icempm_3dm_b200._lib import LIB, MPMError
from icempm_3dm_b200.layout import ACCUM_FIXED, BP00, FE00, POSX, VELX
from tests.helpers import perturbed_block, util_bits

pytestmark = pytest.mark.gpu

STEPS = 6


def _block():
    return perturbed_block(n=1500, seed=6, crushed_frac=0.2, ind_velocity=1.0, dims=(0.12, 0.08, 0.08))


def _same(a, b):
    # the order of the FP64 atomics: 1e-16 of the sums, over six substeps
    (ha, oa), (hb, ob) = a, b
    assert np.abs(ha - hb).max() <= 1e-10 * max(np.abs(hb).max(), 1e-300)
    for row, k in ((POSX, 3), (VELX, 3), (FE00, 9), (BP00, 9)):
        assert np.abs(oa[row:row + k] - ob[row:row + k]).max() <= 1e-9 * np.abs(ob[row:row + k]).max()
    assert np.array_equal(util_bits(oa), util_bits(ob))


@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_FP64_SVD64])
def test_substeps_without_a_buffer_for_the_velocities(precision):
    prms, soa = _block()
    got = []
    for fail in (0, 2):                       # the step's second allocation, after the force history's
        with MPMHandle(prms, soa.shape[1], precision) as h:
            h.upload(soa)
            LIB.mpm_testing_fail_alloc(h._h, fail)
            hist = h.step(STEPS)
            assert LIB.mpm_testing_fail_alloc(h._h, 0) == 0
            got.append((hist, h.download()))
    _same(got[1], got[0])


def test_the_velocity_buffer_is_given_up_for_a_sort_within_a_run():
    prms, soa = _block()
    got = []
    for fail in (0, 1):                       # the first sort's scratch, after two substeps
        with MPMHandle(prms, soa.shape[1], PRECISION_FP64) as h:
            h.upload(soa)
            h.step(STEPS)
            h.update_constants(prms)
            h.upload(soa)
            h.set_sort_interval(2)
            LIB.mpm_testing_fail_alloc(h._h, fail)
            hist = h.step(STEPS)
            assert LIB.mpm_testing_fail_alloc(h._h, 0) == 0
            out = np.empty_like(soa)
            out[:, h.ids()] = h.download()
            got.append((hist, out))
    _same(got[1], got[0])


@pytest.mark.parametrize("precision", [PRECISION_FP64_SVD64, PRECISION_MIXED])
def test_gradient_with_one_velocity_buffer_for_the_segment(precision):
    prms, soa = _block()
    n, every = soa.shape[1], 4                # a segment of four substeps, and one of two

    def gradient(fail):
        with MPMHandle(prms, n, precision) as h:
            if precision == PRECISION_MIXED:
                h.set_grid_accumulation(ACCUM_FIXED)          # the same forward from run to run
            h.upload(soa, cohesion=np.full(n, 3e5))
            LIB.mpm_testing_fail_alloc(h._h, fail)
            hist = h.adjoint_forward(STEPS, every)
            left = LIB.mpm_testing_fail_alloc(h._h, 0)
            s0 = h.sensors()[0]
            out = [h.adjoint_backward(np.ones((STEPS, 3))) for _ in range(2)]
            return left, (hist, out[0][0], out[0][1], out[1][0], h.adjoint_state(), s0, h.sensors()[0])

    left, ref = gradient(0)
    assert np.abs(ref[1]).max() > 0
    fail = lean = 0
    while True:
        fail += 1
        try:
            left, got = gradient(fail)
        except MPMError as e:                 # a buffer that it cannot do without
            assert e.code == 100
            continue
        if left:                              # fewer allocations than that
            break
        lean += 1
        for a, b in zip(got, ref):
            a, b = np.asarray(a), np.asarray(b)
            # the order of the FP64 atomics: 1e-16 of the sums, over six substeps
            assert np.abs(a - b).max() <= 1e-9 * max(np.abs(b).max(), 1e-300)
    assert lean >= every - 1
