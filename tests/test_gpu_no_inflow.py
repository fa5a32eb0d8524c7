"""SCCs that receive no mass, and rates outside the range of single precision.

The network is a d-cube that flips freely behind two exits (one transient SCC of 2^d states,
2^(d-1) odd rows), solved by elimination up to 16 odd rows and by Krylov above.  Its answer
does not change when every rate is multiplied by one constant, so each scale is compared
with scale 1, for an x0 that puts mass on the transient SCC and one that puts none there.

Tolerance: the solver's 1e-10 relative residual, held to L1 <= 1e-9 as in the parity tests.
"""
import numpy as np
import pytest

from paraexastolog_b200 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("d", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("scale", [1e-40, 1e-30, 1e40])
def test_no_inflow_and_extreme_rates(d, scale):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import paraexastolog_b200 as esl
    n = d + 2
    lines = [f"x{i:02d}, !x{i:02d}" for i in range(d)]
    lines += ["e, e | (x00 & x01 & !f)", "f, f | (!x00 & x01 & !e)"]
    m = esl.Model.parse("targets, factors\n" + "\n".join(lines) + "\n")
    rng = np.random.default_rng(d)
    rates = synth.log_uniform_rates(rng, n, 3)
    x0 = np.zeros((2, 1 << n))
    x0[0] = rng.dirichlet(np.ones(1 << n))
    exits = sum(1 << m.names.index(name) for name in ("e", "f"))
    v = np.arange(1 << n)
    x0[1, (v & exits) != 0] = 1.0
    x0[1] /= x0[1].sum()
    ctx = esl.Context(0, torch.cuda.Stream())
    net = esl.Net.build(ctx, m, rates[0])
    torch.cuda.synchronize()
    want = esl.solve_batch(ctx, net, rates, x0, method=esl.METHOD_DIRECT).x_inf.cpu().numpy()
    res = esl.solve_batch(ctx, net, rates * scale, x0, method=esl.METHOD_DIRECT)
    got = res.x_inf.cpu().numpy()
    assert res.report.converged == 1
    assert np.isfinite(got).all()
    assert np.abs(got - want).sum(-1).max() <= 1e-9
