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
