"""The bounded waits at the barriers of the cooperative launches, made to run out.

`ESL_BARRIER_TIMEOUT_TEST=1` lets the barriers expect one arrival that never comes and cuts
the bound to about a thousand polls: every CTA gives up, the kernel ends, the call returns
ESL_ERR_TIMEOUT (-5) and the context stays usable.
"""
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


@pytest.mark.parametrize("n", [6, 14, 18])
def test_graph_barrier_timeout(esl, monkeypatch, n):
    net_g = synth.precision_network(seed=3, n=n)
    rates = synth.log_uniform_rates(np.random.default_rng(n), n, 1)[0]
    ctx = esl.Context(0, torch.cuda.Stream())
    m = esl.Model.parse(net_g.bnet)
    want = [t.cpu().numpy() for t in esl.Net.build(ctx, m, rates).export()]
    monkeypatch.setenv("ESL_BARRIER_TIMEOUT_TEST", "1")
    with pytest.raises(esl.EslError) as e:
        esl.Net.build(ctx, m, rates)
    assert e.value.code == -5
    monkeypatch.delenv("ESL_BARRIER_TIMEOUT_TEST")
    for a, b in zip(want, esl.Net.build(ctx, m, rates).export()):
        assert np.array_equal(a, b.cpu().numpy())


@pytest.mark.parametrize("d,B", [(14, 1), (14, 4), (16, 32)])
@pytest.mark.parametrize("terminal", [False, True])
def test_solver_barrier_timeout(esl, monkeypatch, d, B, terminal):
    """An SCC beyond a cluster (or a CTA, for fewer than eight systems) on the cooperative grid:
    the transient cube, whose nodes stop behind its exits, or also terminal cubes."""
    n = d + 2
    stop = "" if terminal else " & !e & !f"
    lines = [f"x{i:02d}, !x{i:02d}{stop}" for i in range(d)]
    lines += ["e, e | (x00 & x01 & !f)", "f, f | (!x00 & x01 & !e)"]
    rng = np.random.default_rng(d)
    rates = synth.log_uniform_rates(rng, n, B)
    x0 = synth.dirichlet_subspace_x0(rng, n, np.arange(4))[None]
    ctx = esl.Context(0, torch.cuda.Stream())
    net = esl.Net.build(ctx, esl.Model.parse("targets, factors\n" + "\n".join(lines) + "\n"), rates[0])
    torch.cuda.synchronize()
    want = esl.solve_batch(ctx, net, rates, x0, method=esl.METHOD_DIRECT).x_inf.cpu().numpy()
    monkeypatch.setenv("ESL_BARRIER_TIMEOUT_TEST", "1")
    with pytest.raises(esl.EslError) as e:
        esl.solve_batch(ctx, net, rates, x0, method=esl.METHOD_DIRECT)
    assert e.value.code == -5
    monkeypatch.delenv("ESL_BARRIER_TIMEOUT_TEST")
    res = esl.solve_batch(ctx, net, rates, x0, method=esl.METHOD_DIRECT)
    assert res.report.converged == 1
    assert np.abs(res.x_inf.cpu().numpy() - want).sum(-1).max() <= 1e-9
