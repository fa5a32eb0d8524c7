"""What `esl_report` says of the whole-system form on both sides of the 13 nodes up to which it
is one resident block."""
import numpy as np
import pytest

from paraexastolog_b200 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def esl():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import paraexastolog_b200 as E
    E.lib()
    return E


@pytest.mark.parametrize("n", [8, 12, 13, 14])
def test_refinement_steps_are_reported(esl, n):
    net_g = synth.random_table_network(np.random.default_rng(n), n, [2], 0.5)
    rng = np.random.default_rng(1)
    rates = synth.log_uniform_rates(rng, n, 1)[0]
    ctx = esl.Context(0, torch.cuda.Stream())
    net = esl.Net.build(ctx, esl.Model.parse(net_g.bnet), rates)
    torch.cuda.synchronize()
    res = esl.solve(ctx, net, rates, rng.dirichlet(np.ones(1 << n)))
    assert res.report.converged == 1
    assert 1 <= res.report.refinements <= 6
    assert res.report.iterations >= res.report.refinements
