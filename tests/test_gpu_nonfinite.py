"""Infinities and NaN in the state: what one node's value reaches in a
right-hand side, in every stage kernel (node per thread, packed, matrix
instruction).

The derivative at a node of a line is sum_m D[i, m] x[m] over the line's own
N + 1 values, so an infinite x[m] gives the interior nodes of the line (those
without a face flux) infinities of the sign of D[i, m], or NaN where D[i, m] is
zero, and leaves every node off its three lines as it was, bit for bit, but for
the faces it lies on where they hang and the neighbours across them.  A coarse face's infinite trace gives
the fine side's mortar nodes infinities (the interpolation is a sum of finite
multiples).  No tolerances: values are compared by class and by bits."""
from __future__ import annotations

import numpy as np
import pytest

import bfam_b200 as bf

pytestmark = pytest.mark.gpu

# dim 3 orders; conforming and with hanging faces
ORDERS = [1, 2, 3, 4, 5, 6, 7]
PREC = [bf.PRECISION_FP64, bf.PRECISION_FP32]


def _domain(N, prec, p, n=(2, 2, 2), seed=2):
    m = bf.Mesh(3, N, n, refine_prob=p, seed=seed)
    rho, lam, mu = bf.material_random(m.K, 1)
    q = np.random.default_rng(0).standard_normal((m.nfields, m.K * m.Np))
    return m, bf.GpuDomain(m, rho, lam, mu, precision=prec), q


def _class(x):
    return np.where(np.isnan(x), 2, np.where(np.isposinf(x), 1, np.where(np.isneginf(x), -1, 0)))


@pytest.mark.parametrize("N", [3, 4, 5, 6, 7])
@pytest.mark.parametrize("p", [0.0, 0.5])
@pytest.mark.parametrize("prec", PREC, ids=["fp64", "fp32"])
@pytest.mark.parametrize("val", [np.inf, -np.inf])
def test_infinity_on_a_line(N, p, prec, val):
    m, d, q = _domain(N, prec, p)
    D = np.asarray(bf.lgl_operators(N)[3]).reshape(N + 1, N + 1, order="F")
    Nq = N + 1
    inner = np.arange(1, N)
    for e in (0, m.K - 1):
        for ax in range(3):
            for at in (0, N // 2, N):
                pos = [1, N - 1, 1]
                pos[ax] = at
                x = q.copy()
                x[ax, e * m.Np + pos[0] + Nq * (pos[1] + Nq * pos[2])] = val
                d.set_fields(x)
                # the normal stress along the velocity's own axis
                r = d.rhs()[3 + ax, e * m.Np:(e + 1) * m.Np].reshape(Nq, Nq, Nq)
                line = [pos[2], pos[1], pos[0]]
                line[2 - ax] = slice(None)
                with np.errstate(invalid="ignore"):
                    want = _class(D[:, at] * val)
                got = _class(r[tuple(line)])
                assert np.array_equal(got[inner], want[inner]), (e, ax, at, got, want)


@pytest.mark.parametrize("N", ORDERS)
@pytest.mark.parametrize("p", [0.0, 0.5])
@pytest.mark.parametrize("prec", PREC, ids=["fp64", "fp32"])
@pytest.mark.parametrize("val", [np.inf, np.nan])
def test_reach_of_a_value(N, p, prec, val):
    m, d, q = _domain(N, prec, p)
    Nq = N + 1
    d.set_fields(q)
    base = d.rhs().reshape(m.nfields, m.K, Nq, Nq, Nq)
    for e in (0, m.K // 2, m.K - 1):
        # not the element's first node, which the precision form subtracts
        for pos in ((N, N, N), (N, 0, 0), (0, N // 2, N), (N // 2, N, 1 if N > 1 else 0)):
            for f in (0, 4, 8):
                x = q.copy()
                x[f, e * m.Np + pos[0] + Nq * (pos[1] + Nq * pos[2])] = val
                d.set_fields(x)
                r = d.rhs().reshape(base.shape)
                same = ((r == base) | (np.isnan(r) & np.isnan(base))).all(axis=0)
                own = np.zeros((Nq, Nq, Nq), bool)
                own[pos[2], pos[1], :] = own[pos[2], :, pos[0]] = own[:, pos[1], pos[0]] = True
                if p:  # a hanging face's jumps are projected onto the whole face
                    for k, i in enumerate(pos[::-1]):
                        if i in (0, N):
                            own[(slice(None),) * k + (i,)] = True
                assert same[e][~own].all(), (e, pos, f)
                # other elements: only nodes of faces
                other = np.ones(m.K, bool)
                other[e] = False
                assert same[other][:, 1:N, 1:N, 1:N].all(), (e, pos, f)


@pytest.mark.parametrize("N", [3, 4, 5, 6, 7])
@pytest.mark.parametrize("prec", PREC, ids=["fp64", "fp32"])
def test_infinite_coarse_trace(N, prec):
    """an infinite tangential velocity in the last node of a coarse x face: on
    the fine side the traction is infinite, and so is dv_y/dt at the nodes
    inside the face"""
    m, d, q = _domain(N, prec, 0.3, n=(3, 2, 2), seed=1)
    h = m.h[:, 0]
    Nq = N + 1
    x0 = m.x0
    pairs = []
    for e in range(m.K):
        for c in range(m.K):
            # c is twice as large and e touches its upper x face
            if (abs(h[c] - 2 * h[e]) < 1e-12 and abs(x0[c, 0] + h[c] - x0[e, 0]) < 1e-12
                    and all(-1e-12 <= x0[e, a] - x0[c, a] <= m.h[c, a] - m.h[e, a] + 1e-12
                            for a in (1, 2))):
                pairs.append((c, e))
    assert pairs
    d.set_fields(q)
    base = d.rhs()
    for c, e in pairs[:6]:
        x = q.copy()
        x[1, c * m.Np + N + Nq * (N + Nq * N)] = np.inf
        d.set_fields(x)
        r = d.rhs()[1, e * m.Np:(e + 1) * m.Np].reshape(Nq, Nq, Nq)[1:N, 1:N, 0]
        assert np.isinf(r).all(), (c, e, r)
    d.set_fields(q)
    assert np.array_equal(d.rhs(), base)
