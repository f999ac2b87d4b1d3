"""The sort of a mixed handle, on its 32-bit rows: the same stable permutation
as the oracle's on the positions that a download gives, every row moved bit for
bit, the upper halves of the utility words, ids and cohesion with it."""
import numpy as np
import pytest

from icempm_3dm_b200 import PRECISION_FP64, PRECISION_MIXED, MPMHandle
from icempm_3dm_b200.layout import IDX_P, IDX_Q, IDX_UTILITY, STATUS_DISABLED
from oracle import pyoracle as po
from tests.helpers import perturbed_block

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [PRECISION_MIXED, PRECISION_FP64])
@pytest.mark.parametrize("n,disabled", [(1, 0.0), (33, 0.3), (257, 0.05), (5000, 0.1), (5000, 0.0)])
def test_rows_and_words_move_together(precision, n, disabled):
    prms, soa = perturbed_block(n=max(n, 500), seed=6, crushed_frac=0.2)
    rng = np.random.default_rng(n)
    soa = np.ascontiguousarray(soa[:, rng.permutation(soa.shape[1])[:n]])
    bits = soa[IDX_UTILITY].view(np.int64).copy()
    bits |= rng.integers(0, 1 << 30, n) << 32
    bits |= rng.integers(0, 200, n)
    bits[rng.random(n) < disabled] |= STATUS_DISABLED
    soa[IDX_UTILITY] = bits.view(np.float64)
    soa[IDX_P], soa[IDX_Q] = rng.standard_normal(n), rng.random(n)
    coh = 3e5 * np.exp(0.3 * rng.standard_normal(n))
    with MPMHandle(prms, n + 7, precision) as h:
        h.upload(soa, cohesion=coh)
        before, c0 = h.download().copy(), h.cohesion().copy()
        perm = po.sort_permutation(prms, np.ascontiguousarray(before), n)
        for _ in range(2):          # sorted again: nothing moves
            h.sort()
            after = h.download()
            assert np.array_equal(h.ids(), perm)
            assert np.array_equal(after.view(np.int64), before[:, perm].view(np.int64))
            assert np.array_equal(h.cohesion(), c0[perm])
