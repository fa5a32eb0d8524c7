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


@pytest.mark.parametrize("n,B,R", [(10, 20, 1), (11, 7, 3)])
def test_only_missed_systems_leave_the_block(esl, n, B, R):
    """With a budget that some systems miss, the others keep the block's answer.

    At a tolerance of 1e-4 the two solvers stop at different answers (about 1e-5 apart), the
    block's own in a batch and alone differ by rounding only (1e-9 leaves four digits)."""
    net_g = synth.precision_network(seed=4, n=n)
    rng = np.random.default_rng(n)
    rates = synth.log_uniform_rates(rng, n, B)
    x0 = rng.dirichlet(np.ones(1 << n), size=R)
    ctx = esl.Context(0, torch.cuda.Stream())
    net = esl.Net.build(ctx, esl.Model.parse(net_g.bnet), rates[0])
    torch.cuda.synchronize()

    def solve(b, r, iters):
        o = dict(method=esl.METHOD_FP64, tol=1e-4, max_iters=iters, max_refine=1, marginals=False)
        res = esl.solve_batch(ctx, net, rates[b], x0[r], **o)
        return res.x_inf.cpu().numpy(), res.report

    for iters in range(2, 60):
        alone = [[solve(slice(b, b + 1), slice(r, r + 1), iters) for r in range(R)] for b in range(B)]
        missed = np.array([[rep.fallback_systems for _, rep in row] for row in alone])
        if 0 < missed.sum() <= missed.size // 2:
            break
    else:
        pytest.fail("no budget separates the systems")
    got, rep = solve(slice(0, B), slice(0, R), iters)
    assert rep.converged == 1 and rep.fallback_systems == missed.sum()
    want = np.stack([np.stack([x[0, 0] for x, _ in row]) for row in alone])
    assert np.abs(got - want).sum(-1)[missed == 0].max() <= 1e-9
    np.testing.assert_allclose(got.sum(-1), 1.0, atol=1e-3, rtol=0)
