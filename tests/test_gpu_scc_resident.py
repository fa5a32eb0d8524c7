"""The SCC-resident solver (`k_sw_scc`) at the edges of its thread and row splits.

The network is a d-cube that flips freely (x_i, !x_i) behind two exits, e and f, taken on
different faces of the cube: one transient SCC of 2^d states and three terminal ones (e, f
or both set).  The split of the mass between them needs the transient solve, their kernels
the deflated one (dense up to 128 states).  2^(d-1) rows of each
parity: d = 2 (a warp), 8 and 9 (several systems per CTA, one), 11 (one row per thread,
1,024 threads), 12 and 13 (several rows per thread, the largest resident SCC), 14 (above
it: the cooperative grid for few systems, clusters of two CTAs for more), 15 (of four) and 16
(the row kernels).
Batches: one system, a ragged tile, one more than a warp's lanes.

Tolerance: the solver stops at a relative residual of 1e-10 and the tests of the other
paths hold it to L1 <= 1e-9 against the oracle; the same here.
"""
import numpy as np
import pytest

import oracle as O
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


_oracle = {}


def cube_with_exits(d):
    lines = [f"x{i:02d}, !x{i:02d}" for i in range(d)]
    lines += ["e, e | (x00 & x01 & !f)", "f, f | (!x00 & x01 & !e)"]
    return "targets, factors\n" + "\n".join(lines) + "\n"


@pytest.mark.parametrize("d,B,R", [(2, 1, 1), (2, 33, 1), (8, 5, 1), (9, 3, 2), (11, 1, 1), (11, 33, 1), (12, 2, 1),
                                   (13, 1, 1), (13, 3, 1), (14, 1, 1),
                                   (14, 9, 2), (14, 33, 1), (15, 8, 1), (16, 33, 1)])
@pytest.mark.parametrize("method", ["direct", "mixed"])
def test_cube_with_exits(esl, d, B, R, method):
    n = d + 2
    text = cube_with_exits(d)
    rng = np.random.default_rng(100 * d + B)
    rates = synth.log_uniform_rates(rng, n, B)
    x0 = np.stack([synth.dirichlet_subspace_x0(rng, n, rng.choice(n, min(n, 5), replace=False)) for _ in range(R)])
    ctx = esl.Context(0, torch.cuda.Stream())
    net = esl.Net.build(ctx, esl.Model.parse(text), rates[0])
    assert net.T == 3
    m = {"direct": esl.METHOD_DIRECT, "mixed": esl.METHOD_MIXED}[method]
    torch.cuda.synchronize()
    res = esl.solve_batch(ctx, net, rates, x0, method=m)
    assert res.report.converged == 1 and res.report.fallback_systems == 0
    if (d, B) not in _oracle:  # the last system: its tile is the ragged one
        _oracle[d, B] = O.Model(text=text).analyse(rates[0]).solve(x0[-1], rates[-1])
    ox, om = _oracle[d, B]
    assert np.abs(res.x_inf[-1, -1].cpu().numpy() - ox).sum() <= 1e-9
    np.testing.assert_allclose(res.marginals[-1, -1].cpu().numpy(), om, atol=1e-9, rtol=0)
    # every system's distribution sums to 1
    np.testing.assert_allclose(res.x_inf.sum(2).cpu().numpy(), 1.0, atol=1e-9, rtol=0)
