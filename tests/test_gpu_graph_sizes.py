"""The one-launch SCC decomposition (`k_scc`) at its ownership edges, against the oracle.

Sizes: less than one 32-state chunk (n = 1, 4), one chunk (5), one CTA (10), two (11), a
grid of one state per thread (16), several states per thread (18); cyclic and mostly
acyclic networks, with and without zero rates.  Whole numbers: equality.
"""
import numpy as np
import pytest

import oracle as O
from paraexastolog_b200 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ctx():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import paraexastolog_b200 as E
    return E.Context(0, torch.cuda.Stream())


@pytest.mark.parametrize("n", [1, 4, 5, 10, 11, 16, 18])
@pytest.mark.parametrize("family", ["random", "canalizing"])
def test_graph_sizes(ctx, n, family):
    import paraexastolog_b200 as esl
    rng = np.random.default_rng(7 * n + len(family))
    if family == "random":
        net_g = synth.random_table_network(rng, n, [min(2, n)], 0.5)
    else:
        net_g = synth.nested_canalizing_network(rng, n, min(3, n))
    rates = synth.log_uniform_rates(rng, n, 2)
    rates[1, rng.integers(0, 2 * n)] = 0.0
    for r in rates:
        net = esl.Net.build(ctx, esl.Model.parse(net_g.bnet), r)
        sym = O.Model(text=net_g.bnet).analyse(r)
        order, offsets, levels, labels = [t.cpu().numpy() for t in net.export()]
        assert np.array_equal(order, sym.order)
        assert np.array_equal(offsets, sym.offsets)
        first = np.minimum.reduceat(order, offsets[:-1])
        assert np.array_equal(labels[order], np.repeat(first, np.diff(offsets)))
        assert np.array_equal(levels, sym.levels)
