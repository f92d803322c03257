"""The cache's hash-grid gathers, two lanes to a row, at the edges of their
groups: levels that do not fill a group of four, dense and hashed levels in
one group, row counts around a tile and a warp's rows, and the activations
that training keeps of such tiles."""
import numpy as np
import pytest
import torch

from kiraray_gb300.nrc import NeuralRadianceCache
from oracle import nrc_ref as R
from tests.test_nrc_gpu import _oracle, _records, _rel, _targets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels,log2_table,hidden", [(1, 14, 1), (3, 10, 2), (4, 14, 5), (5, 8, 3), (8, 12, 2),
                                                      (9, 12, 5), (13, 14, 6), (16, 10, 5)])
def test_levels_and_rows(krr_lib, cuda, levels, log2_table, hidden):
    """Predictions against the CUDA-core kernels.  Both encode in the same
    order of operations, and round to BF16 (2^-9) at the same places; only the
    FP32 sums of the layers differ, so that an activation may round the other
    way: 2^-8 of the norm bounds that with room."""
    kw = dict(n_levels=levels, log2_table_size=log2_table, base_resolution=4, max_resolution=300,
              hidden_layers=hidden)
    tc = NeuralRadianceCache((-1, -1, -1), (1, 1, 1), tensor_cores=1, **kw)
    ref = NeuralRadianceCache((-1, -1, -1), (1, 1, 1), tensor_cores=0, **kw)
    rng = np.random.default_rng(levels)
    table = (rng.random(tc.params(1).size, dtype=np.float32) - np.float32(0.5))
    for c in (tc, ref):
        c.set_params(0, ref.params(0))
        c.set_params(1, table)
    q = torch.from_numpy(_records(1000, levels)).cuda()
    whole = tc.query(q).cpu().numpy()
    assert _rel(whole, ref.query(q).cpu().numpy()) < 2.0 ** -8
    for n in (1, 15, 16, 17, 127, 128, 129, 999):
        assert np.array_equal(tc.query(q[:n].contiguous()).cpu().numpy(), whole[:n]), n


@pytest.mark.parametrize("n", [1, 17, 130, 3001])
@pytest.mark.parametrize("levels", [1, 7, 16])
def test_table_gradient(krr_lib, cuda, levels, n):
    """The gradient that the kept activations give, against the oracle's (64
    bits, BF16 rounding of the layers' operands): 3e-2 of the norm, as for the
    trained cache."""
    cache = NeuralRadianceCache((-1, -1, -1), (1, 1, 1), n_levels=levels, log2_table_size=10, base_resolution=4,
                                max_resolution=200)
    rng = np.random.default_rng(n)
    cache.set_params(1, (rng.random(cache.params(1).size, dtype=np.float32) - np.float32(0.5)))
    rec = _records(n, n)
    tgt = _targets(rec)
    _, gt, _ = cache.gradients(torch.from_numpy(rec).cuda(), torch.from_numpy(tgt).cuda())
    grid, mlp, table, info = _oracle(cache, (-1, -1, -1), (1, 1, 1))
    X0, cs = R.encode(grid, table, rec)
    y, acts = R.forward(mlp, X0)
    _, dy = R.loss_and_grad(y, tgt.astype(np.float64))
    _, dX0 = R.backward(mlp, acts, dy, loss_scale=cache.cfg.loss_scale)
    assert _rel(gt, R.table_grad(grid, cs, dX0, info.n_table_entries)) < 3e-2


@pytest.mark.parametrize("hidden", [1, 2, 5, 6, 7])
@pytest.mark.parametrize("n", [1, 129, 20000])
def test_layer_gradients(krr_lib, cuda, hidden, n):
    """Every layer's gradient at each depth (seven hidden layers take the
    CUDA-core kernels), with no full tile, a partial one and several per
    block, against the oracle: 3e-2 of the norm, as for the trained cache."""
    cache = NeuralRadianceCache((-1, -1, -1), (1, 1, 1), n_levels=6, log2_table_size=12, base_resolution=4,
                                max_resolution=100, hidden_layers=hidden)
    rng = np.random.default_rng(n)
    cache.set_params(1, (rng.random(cache.params(1).size, dtype=np.float32) - np.float32(0.5)))
    rec = _records(n, n)
    tgt = _targets(rec)
    gm, gt, loss = cache.gradients(torch.from_numpy(rec).cuda(), torch.from_numpy(tgt).cuda())
    grid, mlp, table, info = _oracle(cache, (-1, -1, -1), (1, 1, 1))
    X0, cs = R.encode(grid, table, rec)
    y, acts = R.forward(mlp, X0)
    want, dy = R.loss_and_grad(y, tgt.astype(np.float64))
    gW, dX0 = R.backward(mlp, acts, dy, loss_scale=cache.cfg.loss_scale)
    assert abs(loss - want) < 1e-2 * want
    o = 0
    for l in range(mlp.layers):
        rows = R.WIDTH if l + 1 < mlp.layers else R.OUT_PAD
        assert _rel(gm[o:o + rows * R.IN].reshape(rows, R.IN), gW[l]) < 3e-2, f"layer {l}"
        o += rows * R.IN
    assert _rel(gt, R.table_grad(grid, cs, dX0, info.n_table_entries)) < 3e-2


@pytest.mark.parametrize("levels,hidden,ema", [(1, 1, 0.0), (5, 3, 0.75), (16, 7, 0.0)])
def test_adam_steps(krr_lib, cuda, levels, hidden, ema):
    """Four steps on alternating batches against Adam in 64 bits on the
    gradients that the cache reports: parameters without a gradient in a
    step, or in any, among them.  A gradient carries the noise of FP32 atomics
    (1e-6 of the largest), so only those above 1e-3 of the largest, or exactly
    zero, in every step are compared: 1e-3 of the gradient's relative error,
    doubled by m / sqrt(v), bounds a step's error by 2e-3 learning rates."""
    cache = NeuralRadianceCache((-1, -1, -1), (1, 1, 1), n_levels=levels, log2_table_size=10, base_resolution=4,
                                max_resolution=60, hidden_layers=hidden, epsilon=1e-12, ema_decay=ema)
    lr, b1, b2 = cache.cfg.learning_rate, cache.cfg.beta1, cache.cfg.beta2
    first = [cache.params(k).astype(np.float64) for k in (0, 1)]
    w = [x.copy() for x in first]
    m = [np.zeros_like(x) for x in first]
    v = [np.zeros_like(x) for x in first]
    sure = [np.ones(x.shape, bool) for x in first]
    idle = [np.ones(x.shape, bool) for x in first]
    for s in range(4):
        rec = _records(300, 10 + s % 2)
        if s % 2:
            rec[:, :3] *= 0.3
        r, t = torch.from_numpy(rec).cuda(), torch.from_numpy(_targets(rec)).cuda()
        grads = cache.gradients(r, t)[:2]
        cache.train_step(r, t)
        for k in (0, 1):
            g = grads[k].astype(np.float64).reshape(-1)
            sure[k] &= (g == 0) | (np.abs(g) > 1e-3 * np.abs(g).max())
            idle[k] &= g == 0
            m[k] = b1 * m[k] + (1 - b1) * g
            v[k] = b2 * v[k] + (1 - b2) * g * g
            w[k] -= lr * (m[k] / (1 - b1 ** (s + 1))) / (np.sqrt(v[k] / (1 - b2 ** (s + 1))) + 1e-12)
    for k in (0, 1):
        got = cache.params(k).astype(np.float64)
        assert sure[k].sum() > 50
        assert np.abs(got - w[k])[sure[k]].max() <= 4 * 2e-3 * lr
        assert np.array_equal(got[idle[k]], first[k][idle[k]])
    # the copies that the kernels read are those of the masters
    q = torch.from_numpy(_records(400, 3)).cuda()
    other = NeuralRadianceCache((-1, -1, -1), (1, 1, 1), n_levels=levels, log2_table_size=10, base_resolution=4,
                                max_resolution=60, hidden_layers=hidden)
    for k in (0, 1):
        other.set_params(k, cache.params(k + 2 if ema else k))
    assert np.array_equal(cache.query(q).cpu().numpy(), other.query(q).cpu().numpy())
