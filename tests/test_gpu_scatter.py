"""x_inf and marginals of terminal states (`k_scatter_xinf`) at its block and part sizes.

Without edges every state is a terminal SCC of its own and x_inf is x0, number for number; the
marginals are sums of x0 over the states with a node on (FP64, 1e-12).  From less than a block
of states to several per thread; one system, a few, more than fill the GPU.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,K", [(1, 1), (3, 700), (7, 1), (8, 5), (10, 1), (12, 3), (12, 700), (17, 1), (16, 40)])
@pytest.mark.parametrize("marginals", [True, False])
def test_scatter_of_terminal_states(n, K, marginals):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import paraexastolog_b200 as esl
    N = 1 << n
    ctx = esl.Context(0, torch.cuda.Stream())
    net = esl.Net.from_csc(ctx, n, torch.zeros(N + 1, dtype=torch.int32, device="cuda"),
                           torch.zeros(1, dtype=torch.int32, device="cuda"))
    assert net.T == N
    x0 = np.random.default_rng(n).dirichlet(np.ones(N), size=K)
    torch.cuda.synchronize()
    res = esl.solve_batch(ctx, net, np.ones((1, 2 * n)), x0, method=esl.METHOD_DIRECT, marginals=marginals)
    assert np.array_equal(res.x_inf[0].cpu().numpy(), x0)
    if marginals:
        on = (np.arange(N)[:, None] >> np.arange(n)) & 1
        np.testing.assert_allclose(res.marginals[0].cpu().numpy(), x0 @ on, atol=1e-12, rtol=0)
