"""Device memory that runs out: the handle does without the buffers that only save
time, and gives the same results; a call that needs more than there is says so,
and can be made again when there is memory. The allocations that fail are chosen
through a test hook; no memory is really used up."""
import numpy as np
import pytest

from icempm_3dm_b200 import PRECISION_FP64, PRECISION_FP64_SVD64, PRECISION_MIXED, MPMHandle
from icempm_3dm_b200._lib import LIB, MPMError, check, dptr
from icempm_3dm_b200.layout import ACCUM_FIXED, BP00, FE00, POSX, VELX
from tests.helpers import perturbed_block, util_bits

pytestmark = pytest.mark.gpu

STEPS = 6
COHESION = 3e5


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
            h.upload(soa, cohesion=np.full(n, COHESION))
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


def _upload_cohesion(h, n):
    c = COHESION * (1.0 + 0.3 * np.sin(np.arange(n)))
    check(LIB.mpm_upload_cohesion(h._h, dptr(c), n), "mpm_upload_cohesion")


def _frame(h, n):
    f = h.frame_records(1, True)
    return [np.asarray(f[name], dtype=np.float64) for name in f.dtype.names]


CALLS = {
    "sort": lambda h, n: (h.sort(), h.ids())[1:],
    "step": lambda h, n: (h.step(STEPS),),
    "cohesion": lambda h, n: (_upload_cohesion(h, n), h.step(STEPS))[1:],
    "frame": _frame,
    "gradient": lambda h, n: (h.adjoint_forward(STEPS, 4), *h.adjoint_backward(np.ones((STEPS, 3)))),
    "fixed": lambda h, n: (h.set_grid_accumulation(ACCUM_FIXED), h.step(STEPS))[1:],
}


@pytest.mark.parametrize("call,precision,cohesion", [
    ("sort", PRECISION_FP64, True), ("sort", PRECISION_MIXED, True), ("sort", PRECISION_MIXED, False),
    ("step", PRECISION_FP64, False), ("step", PRECISION_MIXED, True), ("cohesion", PRECISION_MIXED, False),
    ("cohesion", PRECISION_FP64, False), ("frame", PRECISION_FP64, False), ("frame", PRECISION_MIXED, False),
    ("gradient", PRECISION_FP64_SVD64, True), ("gradient", PRECISION_MIXED, True), ("fixed", PRECISION_MIXED, False)])
def test_a_call_that_found_no_memory_can_be_made_again(call, precision, cohesion):
    prms, soa = _block()
    # the order in which a sort has something to do, and 256 Ki points of room: two levels of its scans
    soa = np.ascontiguousarray(soa[:, np.random.default_rng(3).permutation(soa.shape[1])])
    n, room = soa.shape[1], 1 << 18

    def run(fail):
        """What the call and the state after it are, with the fail-th allocation failing first."""
        with MPMHandle(prms, room, precision) as h:
            if precision == PRECISION_MIXED and call != "fixed":
                h.set_grid_accumulation(ACCUM_FIXED)          # the same sums from run to run
            h.upload(soa, cohesion=np.full(n, COHESION) if cohesion else None)
            LIB.mpm_testing_fail_alloc(h._h, fail)
            failed = False
            try:
                got = CALLS[call](h, n)
            except MPMError as e:
                assert e.code == 100
                failed = True
            left = LIB.mpm_testing_fail_alloc(h._h, 0)
            if failed:
                got = CALLS[call](h, n)
            return left, failed, [np.asarray(g, dtype=np.float64) for g in got] + [h.download().copy(), h.ids()]

    def plain(fail):
        """The run that a cohesion which found no memory must leave without cohesion."""
        with MPMHandle(prms, room, precision) as h:
            h.upload(soa)
            if fail:
                LIB.mpm_testing_fail_alloc(h._h, fail)
                with pytest.raises(MPMError):
                    _upload_cohesion(h, n)
            return h.step(STEPS)

    if call == "cohesion":
        a = plain(0)
        for fail in (1, 2) if precision == PRECISION_MIXED else (1,):
            # FP32 sums in another order
            assert np.abs(plain(fail) - a).max() <= 1e-4 * np.abs(a).max()
    _, _, ref = run(0)
    failures = fail = 0
    while True:
        fail += 1
        left, failed, got = run(fail)
        if left:                              # fewer allocations than that
            break
        failures += failed
        for a, b in zip(got, ref):
            if a.dtype == np.uint32:
                assert np.array_equal(a, b)
            elif a.size:
                # the order of the FP64 atomics: 1e-16 of the sums, over six substeps
                ok = np.isfinite(b)
                assert np.abs(a - b)[ok].max() <= 1e-9 * max(np.abs(b[ok]).max(), 1e-300)
    assert failures >= (1 if call in ("step", "fixed", "cohesion") else 5)


def test_a_forward_that_found_no_memory_leaves_the_one_before():
    prms, soa = _block()
    n = soa.shape[1]
    fail = 0
    while True:
        fail += 1
        with MPMHandle(prms, n, PRECISION_FP64_SVD64) as h:
            h.upload(soa, cohesion=np.full(n, COHESION))
            h.adjoint_forward(STEPS, 2)
            ref = h.adjoint_backward(np.ones((STEPS, 3)))
            LIB.mpm_testing_fail_alloc(h._h, fail)
            code = LIB.mpm_adjoint_forward(h._h, 10, 10, None)
            left = LIB.mpm_testing_fail_alloc(h._h, 0)
            if left:
                break
            if code:
                assert code == 100
                h._adj_steps = STEPS
                got = h.adjoint_backward(np.ones((STEPS, 3)))
                assert np.abs(got[0] - ref[0]).max() <= 1e-9 * np.abs(ref[0]).max()
    assert fail > 10
