"""A training step taken again from the same state: what has to come out the
same bit for bit, and how far the order of the FP32 atomics may carry the rest."""
import numpy as np
import pytest
import torch

from kiraray_gb300.nrc import NeuralRadianceCache
from tests.test_nrc_gpu import _records, _rel, _targets

pytestmark = pytest.mark.gpu


def _cache(epsilon=1e-8):
    cache = NeuralRadianceCache((-1, -1, -1), (1, 1, 1), seed=3, epsilon=epsilon)
    rng = np.random.default_rng(1)
    cache.set_params(1, (rng.random(cache.params(1).size, dtype=np.float32) - np.float32(0.5)) * np.float32(0.6))
    return cache


def _batch(n):
    rec = _records(n, n)
    return torch.from_numpy(rec).cuda(), torch.from_numpy(_targets(rec)).cuda()


def _same(a, b):
    return np.array_equal(np.asarray(a).view(np.uint32), np.asarray(b).view(np.uint32))


def test_one_record_gives_the_same_bits(krr_lib, cuda):
    """One thread's atomics have one order: parameters, loss and predictions
    of three steps are the same whenever they are taken."""
    r, t = _batch(1)
    first = None
    for _ in range(3):
        c = _cache()
        got = []
        for _ in range(3):
            loss = c.train_step(r, t)
            got += [np.float32(loss), c.params(0), c.params(1), c.query(r).cpu().numpy()]
        first = first or got
        assert all(_same(x, y) for x, y in zip(first, got))


@pytest.mark.parametrize("n", [2, 127, 128])
def test_one_tile_gives_the_layers_the_same_bits(krr_lib, cuda, n):
    """A batch of one tile has its layers' gradient from one block, each sum
    added once: the layers after a step are the same bit for bit."""
    r, t = _batch(n)
    first = None
    for _ in range(3):
        c = _cache()
        c.train_step(r, t)
        first = c.params(0) if first is None else first
        assert _same(first, c.params(0))


@pytest.mark.parametrize("epsilon", [1e-8, 1e-15])
def test_full_batch_spread(krr_lib, cuda, epsilon):
    """65,536 records, the order of the atomics left to chance.  The layers'
    sums of 152 terms and an entry's sum of some hundreds err by less than
    1e-5 of the largest gradient.  A parameter's step then errs where its
    gradient is of that size or of epsilon's, by a learning rate at most, or
    the BF16 copy rounds the other way (2^-9): one such layer weight moves a
    64-wide layer's outputs by 2^-9 / 8 = 2^-12 of their norm, and no more than
    some in a thousand of the table's entries are near enough to matter.
    2^-10 of the predictions' norm bounds that with room."""
    r, t = _batch(65536)
    a, b = _cache(epsilon), _cache(epsilon)
    (ga, ta, la), (gb, tb, lb) = a.gradients(r, t), b.gradients(r, t)
    assert abs(la - lb) <= 1e-5 * abs(la)
    assert np.abs(ga - gb).max() <= 1e-5 * np.abs(ga).max()
    assert np.abs(ta - tb).max() <= 1e-5 * np.abs(ta).max()
    for c in (a, b):
        c.train_step(r, t)
    assert _rel(a.query(r).cpu().numpy(), b.query(r).cpu().numpy()) < 2.0 ** -10
