"""Host rules of the SCC-resident solver (`csrc/scc_plan.h`), compiled here without CUDA."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "scc_plan.h"
using namespace esl;
extern "C" {
uint32_t own_rows(int j, uint32_t even, uint32_t odd) { return scc_own_rows(j, even, odd); }
int own_a() { return kOwnA; }
int own_w() { return kOwnW; }
int own_iq() { return kOwnIQ; }
int own_count() { return kOwnCount; }
// out: nb, CTAs, threads, shared memory, then per bucket (cta0, items, scc0, stride, lks, lteam, teams)
int plan(const SccShape* shapes, int count, int big, int defl, int K, int n, int max_iters, int64_t* out) {
    SccLaunch L;
    if (!plan_scc_launch(shapes, count, 0, big, defl, K, n, max_iters, 148, L)) return 0;
    *out++ = L.nb, *out++ = L.ctas, *out++ = L.threads, *out++ = (int64_t)L.smem;
    for (int j = 0; j < L.nb; j++) {
        const SccBucket& b = L.b[j];
        for (int64_t v : {(int64_t)b.cta0, (int64_t)b.items, (int64_t)b.scc0, (int64_t)b.stride, (int64_t)b.lks,
                          (int64_t)b.lteam, (int64_t)b.teams})
            *out++ = v;
    }
    return 1;
}
int64_t smem_doubles(int big, int dense, int n, int se, int so, int lks, int nact) {
    return (int64_t)scc_smem_doubles(big, dense, n, se, so, lks, nact);
}
int dense(int so, int max_iters) { return scc_dense(so, max_iters); }
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("scc_plan")
    src, lib = d / "plan.cpp", d / "plan.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(REPO, "paraexastolog_b200", "csrc"),
                    str(src), "-o", str(lib)], check=True)
    return C.CDLL(str(lib))


@pytest.mark.parametrize("even,odd", [(158272, 158269), (24577, 24576), (3, 10), (1, 0), (0, 1)])
def test_vectors_hold_every_row_that_indexes_them(plan, even, odd):
    # the operator's input is indexed by odd rows and, in the setup, by even rows
    for j in range(plan.own_count()):
        rows = plan.own_rows(j, even, odd)
        need = even if j in (plan.own_w(), plan.own_iq()) else max(even, odd) if j == plan.own_a() else odd
        assert rows >= max(need, 1), j


MAX_SMEM, MAX_ROWS, THREADS, THREADS_BIG, BUCKETS = 227 * 1024, 4096, 512, 1024, 16


def check_plan(plan, shapes, big, defl, K, n, max_iters):
    """Every SCC fits its bucket's shared memory and team, and every (SCC, tile) has a CTA."""
    a = np.ascontiguousarray(shapes, np.uint32)
    out = np.zeros(4 + 7 * BUCKETS, np.int64)
    assert plan.plan(a.ctypes.data_as(C.c_void_p), len(a), int(big), int(defl), K, n, max_iters,
                     out.ctypes.data_as(C.c_void_p)) == 1
    nb, ctas, threads, smem = out[:4]
    assert 1 <= nb <= BUCKETS and smem <= MAX_SMEM
    assert threads <= (THREADS_BIG if big else THREADS)
    plan.smem_doubles.restype = C.c_int64
    buckets = out[4:4 + 7 * nb].reshape(nb, 7)
    first = np.concatenate(([0], np.cumsum(a[:, 2])))
    next_cta = 0
    for j, (cta0, items, scc0, stride, lks, lteam, teams) in enumerate(buckets):
        end = buckets[j + 1][2] if j + 1 < nb else first[-1]
        assert cta0 == next_cta and scc0 in first and 1 <= teams <= 16 and (teams << lteam) <= threads
        assert teams * stride * 8 <= smem and (1 << lks) <= max(1, 2 * K - 1) and lks <= 5
        next_cta += -(-items // teams)
        mine = a[(first[:-1] >= scc0) & (first[:-1] < end)]
        assert items == mine[:, 2].sum() * -(-K // (1 << lks))
        for even, odd, _ in mine.tolist():
            dense = int(not big and not defl and plan.dense(odd, max_iters))
            assert plan.smem_doubles(int(big), dense, n, even, odd, int(lks), 1 << int(lteam)) <= stride
            if big:
                assert lteam == 10
            else:
                assert max(even, odd) << lks <= 1 << lteam
    assert next_cta == ctas
    return buckets


def _sorted(shapes):
    return sorted(shapes, key=lambda s: -max(s[0], s[1]))


@pytest.mark.parametrize("K", [1, 2, 31, 37, 148, 512])
def test_launch_plans_of_random_lists(plan, K):
    rng = np.random.default_rng(K)
    for trial in range(300):
        n = int(rng.integers(2, 27))
        big = bool(trial % 2)
        lo, hi = (THREADS + 1, MAX_ROWS) if big else (1, THREADS)
        shapes = []
        for _ in range(int(rng.integers(1, 60))):
            m = int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))
            other = int(rng.integers(1, m + 1)) if rng.random() < 0.7 else m
            even, odd = (m, other) if rng.random() < 0.5 else (other, m)
            shapes.append((even, odd, int(rng.integers(1, 40))))
        check_plan(plan, _sorted(shapes), big, bool(rng.random() < 0.3), K, n, int(rng.choice([1, 5, 600])))


@pytest.mark.parametrize("K,n,shapes", [
    (148, 22, [(2400, 1760, 1), (2100, 2100, 1)]),
    (148, 14, [(2400, 1760, 1), (2100, 2100, 1)]),
    (512, 14, [(1010, 990, 1), (1005, 1005, 1)]),
    (512, 20, [(4096, 400, 30), (4000, 4000, 1), (3990, 200, 9)]),
])
def test_a_smaller_scc_with_a_larger_footprint(plan, K, n, shapes):
    check_plan(plan, shapes, True, False, K, n, 600)


def test_more_alternations_than_buckets(plan):
    shapes = [s for j in range(40) for s in ((2400 - 2 * j, 1000, 1), (2399 - 2 * j, 2399 - 2 * j, 1))]
    buckets = check_plan(plan, shapes, True, False, 512, 20, 600)
    assert len(buckets) == BUCKETS
