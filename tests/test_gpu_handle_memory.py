"""Handles share one bounded pool of device memory: handles made, used and
destroyed one after another and from several threads on streams of their own
give the results of a handle alone, and what stays reserved is bounded."""
import threading

import numpy as np
import pytest
import torch

from icempm_3dm_b200 import PRECISION_FP64_SVD64, MPMHandle, release_memory
from tests.helpers import perturbed_block

pytestmark = pytest.mark.gpu

KEEP = 1 << 30      # bytes the pool may keep without an owner


def _gradient(seed, stream=None):
    prms, soa = perturbed_block(n=1200 + 100 * seed, seed=seed, crushed_frac=0.3, ind_velocity=0.5,
                                dims=(0.12, 0.08, 0.08))
    with MPMHandle(prms, soa.shape[1], PRECISION_FP64_SVD64) as h:
        if stream is not None:
            h.set_stream(stream.cuda_stream)
        h.upload(soa, cohesion=np.full(soa.shape[1], 3e5))
        hist = h.adjoint_forward(6, 3)
        dc, dE = h.adjoint_backward(np.ones((6, 3)))
        return hist, dc, dE


def _same(a, b):
    # the order of the FP64 atomics: 1e-16 of the sums, over six substeps
    for x, y in zip(a, b):
        scale = max(np.abs(np.asarray(y)).max(), 1e-300)
        assert np.abs(np.asarray(x) - np.asarray(y)).max() <= 1e-9 * scale


def test_threads_and_streams_share_the_pool():
    alone = [_gradient(s) for s in range(4)]
    got = [[] for _ in range(4)]

    def work(k):
        st = torch.cuda.Stream()
        for _ in range(5):
            got[k].append(_gradient(k, st))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(4):
        assert len(got[k]) == 5
        for g in got[k]:
            _same(g, alone[k])


def test_what_stays_reserved_is_bounded():
    _gradient(1)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    prms, soa = perturbed_block(n=1200, seed=1)
    with MPMHandle(prms, 12_000_000) as h:          # 2.7 GB of particle rows alone
        h.upload(soa)
        h.sort()
        assert before - torch.cuda.mem_get_info()[0] > 2 * KEEP
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] <= KEEP + (64 << 20)


def test_what_stays_reserved_can_be_given_back():
    release_memory()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    prms, soa = perturbed_block(n=1200, seed=1)
    with MPMHandle(prms, 12_000_000) as h:
        h.upload(soa)
        h.step(2)
        release_memory()                      # what a living handle holds stays with it
        assert np.isfinite(h.download()).all()
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] > KEEP // 2
    release_memory()
    # a page of the driver's own bookkeeping at most
    assert before - torch.cuda.mem_get_info()[0] <= 64 << 20
