"""The reverse sweep on three lanes per particle (small runs) and on one: the
gradients of a block just below the switch and of the same block with points
far from it added beyond the switch agree on the block's points, with counts that
leave warps of ten particles partly filled."""
import numpy as np
import pytest
import torch

from icempm_3dm_b200 import PRECISION_FP64_SVD64, MPMHandle
from icempm_3dm_b200.layout import N_PTS_ARRAYS, POSX
from tests.helpers import perturbed_block

pytestmark = pytest.mark.gpu

STEPS, EVERY = 4, 2


def _gradient(prms, soa):
    n = soa.shape[1]
    with MPMHandle(prms, n, PRECISION_FP64_SVD64) as h:
        h.upload(soa, cohesion=np.full(n, 3e5))
        h.adjoint_forward(STEPS, EVERY)
        w = np.random.default_rng(2).standard_normal((STEPS, 3))
        dc, dE = h.adjoint_backward(w)
        return dc, dE, h.adjoint_state()


@pytest.mark.parametrize("n", [1, 9, 10, 11, 41, 601])
def test_three_lanes_against_one(n):
    prms, soa = perturbed_block(n=601, seed=3, crushed_frac=0.3, ind_velocity=0.5, dims=(0.12, 0.08, 0.08))
    prms.GridXTotal += 600                     # room for the added points, far beyond the block
    prms.DomainDimensionX = prms.GridXTotal * prms.cellsize
    # the n points nearest to the indenter, started two cells further in: every
    # size has contact in the first substep (the loss is a sum over the forces)
    prms.indenter_x_initial += 2 * prms.cellsize
    prms.indenter_x = prms.indenter_x_initial
    d = np.hypot(soa[POSX] - prms.indenter_x, soa[POSX + 1] - prms.indenter_y)
    soa = np.ascontiguousarray(soa[:, np.argsort(d, kind="stable")[:n]])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    extra = 192 * sms + 1 - n
    more = np.zeros((N_PTS_ARRAYS, extra))
    more[:] = soa[:, :1]
    rng = np.random.default_rng(4)
    lo = (prms.GridXTotal - 550) * prms.cellsize
    for d, (a, b) in enumerate(((lo, lo + 500 * prms.cellsize), (5 * prms.cellsize, (prms.GridY - 6) * prms.cellsize),
                                (5 * prms.cellsize, (prms.GridZ - 6) * prms.cellsize))):
        more[POSX + d] = rng.uniform(a, b, extra)
    few = _gradient(prms, soa)
    many = _gradient(prms, np.ascontiguousarray(np.concatenate([soa, more], axis=1)))
    assert np.abs(few[2]).max() > 0 and few[1] != 0
    assert n < 41 or np.abs(few[0]).max() > 0
    # the added points share no node with the block or the indenter: the same
    # derivative, up to the order of FP64 sums (1e-16 of terms that cancel by up
    # to 1e3 over the four substeps)
    for a, b in ((few[0], many[0][:n]), (few[2], many[2][:, :n]), (np.array(few[1]), np.array(many[1]))):
        scale = max(np.abs(a).max(), 1e-300)
        assert np.abs(a - b).max() <= 1e-10 * scale
