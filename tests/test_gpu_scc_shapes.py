"""`k_sw_scc` on SCCs of unequal parities and odd sizes, on graphs made for it.

The graphs come in as tables (`Net.from_csc`); a solve is checked by its own equations
(`tests/hypercube.py`): relative residual and L1 error of the masses <= 1e-9.
"""
import numpy as np
import pytest

import hypercube as H
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


def solve_and_check(esl, F, sizes, B, seed, method=None, systems=3):
    """One batch on the graph F, whose largest SCCs have `sizes` states; the first and last
    systems and one between them are checked."""
    n = int(np.log2(F.size))
    rng = np.random.default_rng(seed)
    rates = synth.log_uniform_rates(rng, n, B)
    x0 = rng.dirichlet(np.ones(F.size))
    ctx = esl.Context(0, torch.cuda.Stream())
    indptr, rows = (torch.as_tensor(a, device="cuda") for a in H.csc(F))
    net = esl.Net.from_csc(ctx, n, indptr, rows)
    offsets = net.export()[1].cpu().numpy()
    assert np.array_equal(np.sort(np.diff(offsets))[::-1][:len(sizes)], np.sort(sizes)[::-1])
    occ = torch.empty((B, F.size), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    res = esl.solve_batch(ctx, net, rates, x0[None], method=esl.METHOD_DIRECT if method is None else method,
                          occupation=occ)
    assert res.report.converged == 1 and res.report.fallback_systems == 0
    for b in np.unique(np.linspace(0, B - 1, systems).astype(int)):
        H.check(F, rates[b], x0, occ[b].cpu().numpy(), res.x_inf[b, 0].cpu().numpy())
    return res


def test_two_sccs_whose_footprints_grow(esl):
    """The second SCC has fewer rows of its larger parity and the larger footprint: two systems
    of the first fit a CTA, of the second one does."""
    rng = np.random.default_rng(1)
    parts = [H.random_part(rng, 13, 2400, 1760), H.random_part(rng, 13, 2100, 2100) | (1 << 13)]
    solve_and_check(esl, H.masks(rng, 14, parts), [4160, 4200], 148, 2)


# (even, odd) rows and systems: both sides of one row per thread (512), unequal parities, a CTA;
# clusters of two to four CTAs (from 8 systems) whose last CTA has few rows, a partial slice of
# 32, or none of one parity, and their cooperative grid (fewer systems); beyond a cluster
SHAPES = [(512, 512, 3), (511, 512, 33), (513, 200, 5), (513, 513, 1), (4096, 900, 2), (900, 4096, 150), (4096, 4095, 1),
          (4097, 900, 8), (4097, 4096, 3), (5000, 8192, 9), (8300, 8200, 8), (9000, 4000, 9), (4000, 9000, 34),
          (12289, 12300, 8), (16384, 13000, 10), (16385, 16000, 17)]


def cube_of(even, odd):
    """A cube with room for the part: one more dimension where one parity has few rows."""
    return int(np.ceil(np.log2(2 * max(even, odd)))) + (3 * min(even, odd) < 2 * max(even, odd))


@pytest.mark.parametrize("even,odd,B", SHAPES)
def test_transient_shapes(esl, even, odd, B):
    rng = np.random.default_rng(even + odd)
    d = cube_of(even, odd)
    solve_and_check(esl, H.masks(rng, d + 1, [H.random_part(rng, d, even, odd)]), [even + odd], B, odd)


@pytest.mark.parametrize("even,odd,B", SHAPES)
def test_terminal_shapes(esl, even, odd, B):
    """The same parts without exits: the deflated solves."""
    rng = np.random.default_rng(even + odd)
    d = cube_of(even, odd)
    part = H.random_part(rng, d, even, odd)
    v = np.arange(1 << d)
    inside = np.isin(v, part)
    F = np.zeros(1 << d, np.uint32)
    for i in range(d):
        F[inside & inside[v ^ (1 << i)]] |= np.uint32(1 << i)
    rates = synth.log_uniform_rates(rng, d, B)
    x0 = np.where(inside, 1.0 / len(part), 0.0)
    ctx = esl.Context(0, torch.cuda.Stream())
    net = esl.Net.from_csc(ctx, d, *(torch.as_tensor(a, device="cuda") for a in H.csc(F)))
    assert np.diff(net.export()[1].cpu().numpy()).max() == even + odd
    torch.cuda.synchronize()
    res = esl.solve_batch(ctx, net, rates, x0[None], method=esl.METHOD_DIRECT)
    for b in np.unique([0, B // 2, B - 1]):
        H.check_stationary(F, rates[b], part, res.x_inf[b, 0].cpu().numpy())


def tiny_sccs(n):
    """One free node (bit 0) beside nodes that only decay: 2^(n-1) - 1 SCCs of two states, and
    two terminal states without edges."""
    v = np.arange(1 << n, dtype=np.int64)
    return np.where(v > 1, v | 1, 0).astype(np.uint32)


@pytest.mark.parametrize("n,B", [(4, 3), (11, 1), (12, 40), (17, 2)])
def test_many_tiny_sccs(esl, n, B):
    solve_and_check(esl, tiny_sccs(n), [2] * ((1 << (n - 1)) - 1), B, n)


def test_many_tiny_sccs_take_little_memory(esl):
    """Network, plan and workspace of a solve with 524,287 SCCs: under 700 bytes per state (the
    padded vectors of one system are 256 of them)."""
    n = 20
    rng = np.random.default_rng(3)
    rates = synth.log_uniform_rates(rng, n, 1)
    x0 = torch.as_tensor(rng.dirichlet(np.ones(1 << n))[None], device="cuda")
    indptr, rows = (torch.as_tensor(a, device="cuda") for a in H.csc(tiny_sccs(n)))
    out = torch.empty((1, 1, 1 << n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    esl.lib().esl_trim_cache()
    before = torch.cuda.mem_get_info()[0]
    ctx = esl.Context(0)
    net = esl.Net.from_csc(ctx, n, indptr, rows)
    res = esl.solve_batch(ctx, net, rates, x0, method=esl.METHOD_DIRECT, out=out)
    assert res.report.converged == 1
    torch.cuda.synchronize()
    esl.lib().esl_trim_cache()
    assert before - torch.cuda.mem_get_info()[0] < 700 << n


def mixed_sizes(rng):
    """n = 17: SCCs beyond a cluster, of three CTAs, of one, of one row per thread, and of the
    sizes around the narrow ones, all in one level group."""
    parts = [H.random_part(rng, 16, 16500, 16390)]
    for k, (even, odd) in enumerate([(5000, 4990), (4097, 900), (4096, 4000), (600, 513)]):
        parts.append(H.random_part(rng, 13 if even <= 4096 else 14, even, odd) | (4 + k) << 14)
    small = [(512, 500), (33, 32), (32, 20), (9, 7), (8, 8), (8, 3), (1, 1), (1, 2), (17, 16)]
    for k, (even, odd) in enumerate(small):
        # in the other half of the last region
        at = 7 << 14 | 1 << 13 | (0 if k == 0 else (7 + k) << 7)
        parts.append(H.random_part(rng, 10 if k == 0 else 7, even, odd) | at)
    return parts


@pytest.mark.parametrize("which", ["tiny", "mixed"])
def test_device_plan_equals_host_plan(esl, which):
    """8,191 SCCs of two states, whose list is sorted on the device, and every other kind."""
    F = tiny_sccs(14) if which == "tiny" else H.masks(np.random.default_rng(7), 17, mixed_sizes(np.random.default_rng(6)))
    ctx = esl.Context(0)
    net = esl.Net.from_csc(ctx, int(np.log2(F.size)), *(torch.as_tensor(a, device="cuda") for a in H.csc(F)))
    assert np.array_equal(net.plan_checksums(host_builder=False), net.plan_checksums(host_builder=True))
