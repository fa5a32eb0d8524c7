"""The whole-system form and the absorption matrix as one resident block (up to 13 nodes).

Sizes from three transient states to the limit, and one node above it (the previous path).
x_inf and L against the oracle up to n = 10 (L1 and max-abs 1e-9, as the other parity tests);
at every size L x0 must give the masses of the level sweep's answer for other initial
distributions, to 1e-9.
"""
import numpy as np
import pytest

import oracle as O
from paraexastolog_b200 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,seed", [(2, 1), (3, 2), (5, 3), (8, 4), (10, 5), (13, 6), (14, 7)])
def test_whole_block(n, seed):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import paraexastolog_b200 as esl
    rng = np.random.default_rng(seed)
    net_g = synth.random_table_network(rng, n, [min(2, n)], 0.5)
    rates = synth.log_uniform_rates(rng, n, 1)[0]
    x0 = rng.dirichlet(np.ones(1 << n), size=3)
    ctx = esl.Context(0, torch.cuda.Stream())
    net = esl.Net.build(ctx, esl.Model.parse(net_g.bnet), rates)
    torch.cuda.synchronize()
    res = esl.solve(ctx, net, rates, x0[0], want_R=True, want_L=True)
    assert res.report.converged == 1
    L, xi = res.L.cpu().numpy(), res.x_inf.cpu().numpy()
    np.testing.assert_allclose(L.sum(0), 1.0, atol=1e-9, rtol=0)
    order, offsets, _, _ = [t.cpu().numpy() for t in net.export()]
    sweep = esl.solve_batch(ctx, net, rates, x0, method=esl.METHOD_DIRECT).x_inf[0].cpu().numpy()
    assert np.abs(xi - sweep[0]).sum() <= 1e-9
    for r in range(3):
        masses = [sweep[r][order[offsets[t]:offsets[t + 1]]].sum() for t in range(net.T)]
        np.testing.assert_allclose(L @ x0[r], masses, atol=1e-9, rtol=0)
    if n <= 10:
        sym = O.Model(text=net_g.bnet).analyse(rates)
        ox, _ = sym.solve(x0[0], rates)
        assert np.abs(xi - ox).sum() <= 1e-9
        assert np.abs(L - sym.absorption(rates)).max() <= 1e-9
