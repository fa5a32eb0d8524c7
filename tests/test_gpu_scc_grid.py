"""The cooperative-grid solver (`k_sw_scc<kSccGrid>`) on an SCC with more even than odd rows.

A free 16-cube behind two exits, without two states of odd parity: no flip enters them, so
65,534 states form the transient SCC (32,768 even rows, 32,766 odd ones), beyond a cluster.
Few systems run on the cooperative grid; 16, 17 and 32 of them use half of a row's padding,
and all of it.  Checked against the oracle, L1 <= 1e-9 as the other paths.
"""
import numpy as np
import pytest

import oracle as O
from paraexastolog_b200 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def cube_without(d, removed):
    """Rules of a free d-cube whose flips into the states `removed` are blocked."""
    lines = []
    for i in range(d):
        me = f"x{i:02d}"
        lit = [[("" if (s >> j) & 1 else "!") + f"x{j:02d}" for j in range(d)] for s in removed]
        neg = [[("!" if (s >> j) & 1 else "") + f"x{j:02d}" for j in range(d)] for s in removed]
        # up: !x_i and, for every removed state with bit i set, another bit that differs
        up = [[f"!{me}"]]
        # stay up: x_i and the other bits of a removed state with bit i clear
        terms = []
        for s, t, u in zip(removed, lit, neg):
            if (s >> i) & 1:
                up = [c + [u[j]] for c in up for j in range(d) if j != i]
            else:
                terms.append([me] + [t[j] for j in range(d) if j != i])
        terms += up
        lines.append(f"{me}, " + " | ".join("(" + " & ".join(dict.fromkeys(c)) + ")" for c in terms))
    lines += ["e, e | (x00 & x01 & !f)", "f, f | (!x00 & x01 & !e)"]
    return "targets, factors\n" + "\n".join(lines) + "\n"


@pytest.mark.parametrize("B", [3, 16, 17, 32])
def test_more_even_than_odd_rows(B):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import paraexastolog_b200 as esl
    d, n = 16, 18
    removed = [0b0000000000000001, 0b0111111111111111]
    text = cube_without(d, removed)
    rng = np.random.default_rng(16)
    rates = synth.log_uniform_rates(rng, n, 32)[:B]
    x0 = synth.dirichlet_subspace_x0(rng, n, np.arange(4))
    ctx = esl.Context(0, torch.cuda.Stream())
    net = esl.Net.build(ctx, esl.Model.parse(text), rates[0])
    offsets = net.export()[1].cpu().numpy()
    assert np.diff(offsets).max() == (1 << d) - len(removed)
    torch.cuda.synchronize()
    res = esl.solve_batch(ctx, net, rates, x0[None], method=esl.METHOD_DIRECT)
    assert res.report.converged == 1 and res.report.fallback_systems == 0
    xi = res.x_inf[:, 0].cpu().numpy()
    np.testing.assert_allclose(xi.sum(1), 1.0, atol=1e-9, rtol=0)
    ox, _ = O.Model(text=text).analyse(rates[0]).solve(x0, rates[-1])
    assert np.abs(xi[-1] - ox).sum() <= 1e-9
