"""Gradient kernels of the warm-start network at the edges of their sample slabs.

`k_mlp_wgrad` gives each of 74 CTAs a slab of samples in chunks of 16; sizes below one slab
(empty CTAs), one past a chunk, one past 74 chunks and a large ragged batch.  Tolerances of
the existing gradient test: FP32 passes against the float64 oracle, 1e-3 in the norm.
"""
import numpy as np
import pytest

import oracle as O
from oracle import mlp as OM
from paraexastolog_b200 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("S", [1, 17, 73, 130, 1185, 9001])
def test_gradient_sizes(S):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import paraexastolog_b200 as esl
    n = 12
    net_g = synth.precision_network(seed=3, n=n)
    rng = np.random.default_rng(S)
    rates = synth.log_uniform_rates(rng, n, 40)
    ctx = esl.Context(0)
    mlp = esl.Mlp(ctx, esl.Net.build(ctx, esl.Model.parse(net_g.bnet), rates[0]), seed=5)
    om = O.Model(text=net_g.bnet)
    sym, F = om.analyse(rates[0]), om.flip_masks(rates[0])
    ks, vs = rng.integers(0, 40, S), rng.integers(0, 1 << n, S)
    t = rng.normal(0, 1, S).astype(np.float32)
    p = mlp.get_params()
    p[OM.N_PARAMS - 129:OM.N_PARAMS - 1] += 0.05  # non-trivial head
    mlp.set_params(p, 0.0, 1.0)
    loss, g = mlp.loss_grad(rates, ks, vs, t)
    lr, gr = OM.loss_grad(p, OM.features(n, sym.T, F, OM.reach_bits(sym, F), rates, ks, vs), t)
    assert abs(loss - lr) <= 1e-4 * abs(lr), (loss, lr)
    assert np.linalg.norm(g - gr) <= 1e-3 * np.linalg.norm(gr)
