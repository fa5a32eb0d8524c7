"""The SCC decomposition and the levels on chains as long as the state space.

The reflected Gray code visits every state once: with the one flip per state that follows it
the graph is a chain of 2^m singletons and levels.  Times a node that flips freely it is a
chain of 2^m SCCs of two states.  Order, offsets and levels are known in closed form; the
default budgets and little more sweeps than levels must do.
"""
import numpy as np
import pytest

import hypercube as H

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("m,free", [(3, 0), (8, 0), (8, 1), (10, 0), (11, 1), (12, 0), (13, 1)])
@pytest.mark.parametrize("spare", [None, 8])
def test_gray_code_chain(m, free, spare):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import paraexastolog_b200 as esl
    n, L = m + free, 1 << m
    k = np.arange(L, dtype=np.int64)
    gray = k ^ (k >> 1)
    F = np.zeros(1 << n, np.uint32)
    F[gray[:-1]] = (gray[:-1] ^ gray[1:]).astype(np.uint32)
    if free:
        F[:L] |= np.uint32(1 << m)
        F[L:] = F[:L]
    ctx = esl.Context(0, torch.cuda.Stream())
    if spare is not None:
        ctx.set_budgets(graph_sweeps=L + spare)
    net = esl.Net.from_csc(ctx, n, *(torch.as_tensor(a, device="cuda") for a in H.csc(F)))
    order, offsets, levels, labels = [t.cpu().numpy() for t in net.export()]
    size = 1 << free
    chain = np.concatenate((gray[-1:], gray[:-1]))
    want = (chain[:, None] + (np.arange(size) << m)[None]).reshape(-1)
    assert net.n_sccs == L and net.T == 1
    assert np.array_equal(order, want)
    assert np.array_equal(offsets, size * np.arange(L + 1))
    assert np.array_equal(levels, np.concatenate(([1], np.arange(L, 1, -1))))
    assert np.array_equal(labels, np.arange(1 << n) % L)
