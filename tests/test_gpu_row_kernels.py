"""The row kernels of the level sweep: an SCC beyond a cluster with more than 32 systems.

The graph (n = 17) has one SCC of 33,100 states with unequal parities, and in the same level
group SCCs of 1,113, 52 and 3 states and singletons, which `k_sw_scc` takes beside it.  Both
kernel families (paired rows, the default; ESL_SWEEP_OP=reg: one system per lane, 64- and
128-system tiles) run in a process of their own, with 33 systems (two tiles) and 160 (five:
compaction starts), the latter without compaction too.  The profile records of the Schur
operator show that the row kernels ran.  Every solve is checked by its own equations (relative
residual and L1 error of the masses <= 1e-9), and families against one another (L1 <= 1e-9).
"""
import os
import subprocess
import sys

import numpy as np
import pytest

import hypercube as H
from paraexastolog_b200 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

HERE = os.path.dirname(os.path.abspath(__file__))
N_NODES = 17


def graph():
    rng = np.random.default_rng(11)
    parts = [H.random_part(rng, 16, 16700, 16400), H.random_part(rng, 13, 600, 513) | 1 << 16,
             H.random_part(rng, 7, 32, 20) | 1 << 16 | 1 << 14, H.random_part(rng, 7, 1, 2) | 1 << 16 | 1 << 15]
    return H.masks(rng, N_NODES, parts, singles=True)


def inputs(B):
    rng = np.random.default_rng(B)
    return synth.log_uniform_rates(rng, N_NODES, B), rng.dirichlet(np.ones(1 << N_NODES))


def solve(esl, F, B, **options):
    rates, x0 = inputs(B)
    ctx = esl.Context(0)
    net = esl.Net.from_csc(ctx, N_NODES, *(torch.as_tensor(a, device="cuda") for a in H.csc(F)))
    occ = torch.empty((B, F.size), dtype=torch.float64, device="cuda")
    ctx.set_profiling(True)
    res = esl.solve_batch(ctx, net, rates, x0[None], occupation=occ, marginals=False, **options)
    assert res.report.converged == 1 and res.report.fallback_systems == 0
    assert sum(name == "schur_operator" for name, _, _ in ctx.profile_entries()) > 0
    return res.x_inf[:, 0].cpu().numpy(), occ


def check(F, B, x_inf, occ):
    rates, x0 = inputs(B)
    for b in (0, B // 2, B - 1):
        H.check(F, rates[b], x0, occ[b].cpu().numpy(), x_inf[b])


CHILD = r"""
import sys
import numpy as np
sys.path[:0] = [sys.argv[1], sys.argv[2]]
import paraexastolog_b200 as esl
import test_gpu_row_kernels as T
F, B = T.graph(), int(sys.argv[3])
x_inf, occ = T.solve(esl, F, B, method=esl.METHOD_DIRECT)
T.check(F, B, x_inf, occ)
np.save(sys.argv[4], x_inf)
"""


@pytest.mark.parametrize("B", [33, 160])
def test_kernel_families_agree(tmp_path, B):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    got = []
    for k, env in enumerate([{}, {"ESL_SWEEP_OP": "reg"}, {"ESL_SWEEP_COMPACT": "0"}][:2 if B == 33 else 3]):
        out = tmp_path / f"{k}.npy"
        subprocess.run([sys.executable, "-c", CHILD, os.path.dirname(HERE), HERE, str(B), str(out)],
                       env=dict(os.environ, **env), check=True, timeout=600)
        got.append(np.load(out))
    for other in got[1:]:
        assert np.abs(other - got[0]).sum(1).max() <= 1e-9


@pytest.mark.parametrize("warm", [False, True])
def test_mixed_precision(warm):
    """FP32 inner solves in the row kernels, cold and from a warm start (a noisy solution)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import paraexastolog_b200 as esl
    F, B = graph(), 40
    options = {}
    if warm:
        _, occ = solve(esl, F, B, method=esl.METHOD_DIRECT)
        g = torch.Generator(device="cuda").manual_seed(1)
        options["warm"] = occ * torch.exp(0.3 * torch.randn(occ.shape, generator=g, device="cuda", dtype=torch.float64))
    x_inf, occ = solve(esl, F, B, method=esl.METHOD_MIXED, **options)
    check(F, B, x_inf, occ)
