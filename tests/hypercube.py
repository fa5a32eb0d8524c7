"""Transition graphs with SCCs of chosen sizes, and a check of a solve without an oracle.

A graph is its flip masks (bit i of F[s]: edge s -> s ^ (1 << i)).  The answer is checked
through what defines it: the occupation z solves q z - inflow(z) = x0 on the transient states,
and a state without edges ends with x0 plus its inflow.
"""
import numpy as np
from scipy.sparse import csr_matrix
from scipy.sparse.csgraph import connected_components


def parity(s):
    s = np.asarray(s, np.int64).copy()
    for k in (16, 8, 4, 2, 1):
        s ^= s >> k
    return s & 1


def random_part(rng, d, even, odd):
    """States of a connected part of the d-cube with `even` and `odd` states of each parity."""
    want = (even, odd)
    N = 1 << d
    par = parity(np.arange(N))
    inside = np.zeros(N, bool)
    for _ in range(500):
        for p in (0, 1):
            need = want[p] - int((inside & (par == p)).sum())
            free = ~inside & (par == p)
            near = free & np.any([inside[np.arange(N) ^ (1 << i)] for i in range(d)], axis=0)
            if need <= near.sum():  # next to what there is, once there is enough of it
                free = near
            inside[rng.choice(np.flatnonzero(free), need, replace=False)] = True
        v = np.flatnonzero(inside)
        src, dst = [], []
        for i in range(d):
            w = v ^ (1 << i)
            m = inside[w]
            src.append(v[m])
            dst.append(w[m])
        src, dst = np.concatenate(src), np.concatenate(dst)
        _, lab = connected_components(csr_matrix((np.ones(src.size, np.int8), (src, dst)), shape=(N, N)), directed=False)
        main = np.bincount(lab[v]).argmax()
        if (lab[v] == main).all():
            return v
        inside[v[lab[v] != main]] = False
    raise ValueError("no connected part found")


def masks(rng, n, parts, exits=0.2, singles=False):
    """Flip masks of a graph in which each part (an array of states) is an SCC of its own, with
    edges to states outside all parts from about `exits` of its states.  singles: odd states
    outside the parts flow into even ones, which keep no edges, and so do the parts, from their
    odd states: all of them are one level group."""
    N = 1 << n
    part_of = np.full(N, -1, np.int64)
    for j, p in enumerate(parts):
        part_of[p] = j
    F = np.zeros(N, np.uint32)
    for j, p in enumerate(parts):
        may = parity(p) == 1 if singles else np.ones(len(p), bool)
        out = np.zeros(len(p), bool)
        for i in range(n):
            t = part_of[p ^ (1 << i)]
            leave = may & (t < 0) & (rng.random(len(p)) < exits / n * 4)
            out |= leave
            F[p[(t == j) | leave]] |= np.uint32(1 << i)
        if not out.any():  # one exit at least
            s, i = next((s, i) for s in p[may] for i in range(n) if part_of[s ^ (1 << i)] < 0)
            F[s] |= np.uint32(1 << i)
    if singles:
        v = np.flatnonzero((part_of < 0) & (parity(np.arange(N)) == 1))
        for i in range(n):
            F[v[(part_of[v ^ (1 << i)] < 0) & (rng.random(len(v)) < 0.3)]] |= np.uint32(1 << i)
    return F


def csc(F):
    """(indptr, rows) of the table, destinations ascending within a column."""
    n = int(np.log2(F.size))
    s = np.arange(F.size, dtype=np.int64)
    src, dst = [], []
    for i in range(n):
        m = (F >> np.uint32(i)) & 1 == 1
        src.append(s[m])
        dst.append(s[m] ^ (1 << i))
    src, dst = np.concatenate(src), np.concatenate(dst)
    o = np.lexsort((dst, src))
    indptr = np.zeros(F.size + 1, np.int32)
    indptr[1:] = np.cumsum(np.bincount(src, minlength=F.size))
    return indptr, dst[o].astype(np.int32)


def flows(F, rates, z):
    """(out-rate sums, inflow of z) of every state."""
    s = np.arange(F.size, dtype=np.int64)
    q, inflow = np.zeros(F.size), np.zeros(F.size)
    for i in range(int(np.log2(F.size))):
        r = np.where((F >> np.uint32(i)) & 1, rates[2 * i + ((s >> i) & 1)], 0.0)
        q += r
        inflow += (r * z)[s ^ (1 << i)]
    return q, inflow


def check(F, rates, x0, z, x_inf, tol=1e-9):
    """z and x_inf of one system on a graph whose terminal states have no edges: the relative
    residual and the L1 error of the masses are within tol."""
    q, inflow = flows(F, rates, z)
    transient = F != 0
    res = np.abs(q * z - inflow - x0)[transient].sum()
    assert res <= tol * np.abs(x0).sum(), res
    want = np.where(transient, 0.0, x0 + inflow)
    assert np.abs(x_inf - want).sum() <= tol, np.abs(x_inf - want).sum()
    assert abs(x_inf.sum() - x0.sum()) <= tol


def check_stationary(F, rates, part, x_inf, tol=1e-9):
    """x_inf of one system is the stationary distribution of a part without exits: the relative
    L1 residual of the balance equations is within tol, and nothing is left outside."""
    q, inflow = flows(F, rates, x_inf)
    assert np.abs(q * x_inf - inflow).sum() <= tol * (q * x_inf).sum()
    assert abs(x_inf[part].sum() - 1.0) <= tol and abs(x_inf.sum() - 1.0) <= tol
    assert x_inf.min() >= -tol
