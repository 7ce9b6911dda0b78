"""The batch forms of the matrix-instruction and packed kernels, which groups of
several domains run (a group of one domain runs the single-domain form): each
domain bitwise as alone and against the oracle, where the domains of a group
differ in mesh, material, data and time step, and where a CTA takes elements of
two of them.

Bar: FP64 1e-12 relative L2 per field against the oracle, the precision form
1e-6 (as everywhere); in a batch bitwise as alone."""
from __future__ import annotations

import numpy as np
import pytest

import bfam_b200 as bf
from bfam_b200 import configs
from oracle import oracle as orc
from conftest import relerr

pytestmark = pytest.mark.gpu

SRC = ((0.4, 0.3, 0.6), (1.0, -0.5, 0.25), 10.0, 0.01)
PREC = [(bf.PRECISION_FP64, 1e-12), (bf.PRECISION_FP32, 1e-6)]
IDS = ["fp64", "fp32"]


def _problem(dim, N, n, p, seed, bounded=False):
    m = bf.Mesh(dim, N, n[:dim], refine_prob=p, seed=seed, periodic=(not bounded,) * 3)
    rho, lam, mu = bf.material_random(m.K, seed + 3)
    q = np.random.default_rng(seed).standard_normal((m.nfields, m.K * m.Np))
    return m, rho, lam, mu, q, configs.stable_dt(m, rho, lam, mu, 0.2 + 0.02 * (seed % 5))


def _bc(dim):
    return (bf.BC_ABSORBING, bf.BC_FREE_SURFACE) * dim


def _domain(prob, prec, source=False):
    m, rho, lam, mu, q, dt = prob
    d = bf.GpuDomain(m, rho, lam, mu, precision=prec, bc=_bc(m.dim))
    d.set_fields(q)
    if source:
        d.set_source(*SRC)
        d.set_receivers(np.array([[0.2, 0.7, 0.1]]), 4)
    return d


def _alone(probs, prec, steps, source=False):
    out = []
    for prob in probs:
        d = _domain(prob, prec, source)
        bf.LSRK(d).step(prob[5], steps, use_graph=True)
        out.append((d.get_fields(), d.seismograms() if source else None))
    return out


def _oracle(prob, steps, source=False):
    m, rho, lam, mu, q, dt = prob
    o = orc.Oracle.from_mesh(m, rho, lam, mu, 0, bc=_bc(m.dim))
    if source:
        o.set_source(*SRC)
        return o.seismograms(q, 0.0, dt, steps, np.array([[0.2, 0.7, 0.1]]))[0]
    return o.lsrk(q, dt, steps)


# odd and even element counts, so that the rows of an odd number of nodes start
# on either side of a 16-byte boundary, and the last row of an odd-sized state
CONFORMING = [((1, 1, 1), 0.0, 0), ((2, 1, 1), 0.0, 1), ((3, 1, 1), 0.0, 2), ((2, 2, 2), 0.0, 3)]
HANGING = [((2, 2, 1), 0.5, 4), ((2, 2, 2), 0.4, 5), ((3, 2, 1), 0.4, 6)]


@pytest.mark.parametrize("N", [5, 6, 7])
@pytest.mark.parametrize("prec,tol", PREC, ids=IDS)
@pytest.mark.parametrize("meshes", [CONFORMING, HANGING], ids=["conforming", "hanging"])
def test_high_orders_under_every_tile(N, prec, tol, meshes):
    probs = [_problem(3, N, n, p, s, bounded=s % 2 == 1) for n, p, s in meshes]
    assert {m[0].K % 2 for m in probs} == {0, 1}
    alone = _alone(probs, prec, 3, source=True)
    hanging = meshes is HANGING
    kernels = bf.tile_kernels(3, N, prec, hanging)
    assert kernels[0][0] == ("mma" if prec == 0 and (N > 5 or hanging) else "node")
    for tile in range(len(kernels)):
        doms = [_domain(p, prec, source=True) for p in probs]
        b = bf.Batch(doms, t0=0.0)
        assert len(b.groups()) == 1 and b.groups()[0]["hanging"] == hanging
        b.set_tile(0, tile, 0)
        b.step([p[5] for p in probs], 3)
        for i, d in enumerate(doms):
            assert np.array_equal(d.get_fields(), alone[i][0]), (tile, i)
            assert np.array_equal(d.seismograms(), alone[i][1]), (tile, i)
        b.free()
    for (q, _), prob in zip(alone, probs):
        assert relerr(q, _oracle(prob, 3, source=True)).max() < tol


# three uneven domains of one group, whose CTAs straddle their ends: enough
# elements that a CTA takes more than one (orders 1 and 2) and that the launch is
# not left to the node-per-thread kernel (elements per SM: the last number)
F64, F32 = PREC
STRADDLE = [(2, 1, [((29, 23), 0.3), ((31, 17), 0.4), ((7, 5), 0.5)], PREC, 8),
            (2, 2, [((27, 23), 0.4), ((19, 31), 0.3), ((3, 5), 0.4)], PREC, 8),
            (2, 3, [((5, 3), 0.4), ((4, 7), 0.5), ((3, 3), 0.4)], PREC, 0),
            (2, 6, [((59, 53), 0.4), ((7, 3), 0.5), ((13, 13), 0.4)], PREC, 32),
            (2, 7, [((83, 79), 0.4), ((7, 3), 0.5), ((13, 13), 0.4)], [F64], 60),
            (2, 8, [((43, 47), 0.4), ((5, 3), 0.5), ((11, 13), 0.4)], [F32], 22),
            (2, 6, [((37, 41), 0.0), ((7, 3), 0.0), ((5, 5), 0.0)], PREC, 10),
            (3, 1, [((8, 7, 7), 0.4), ((7, 5, 6), 0.3), ((3, 2, 3), 0.4)], PREC, 8),
            (3, 2, [((39, 37, 41), 0.0), ((13, 9, 10), 0.0), ((3, 5, 1), 0.0)], [F32], 400)]


@pytest.mark.parametrize("dim,N,meshes,prec,tol,per_sm",
                         [c[:3] + pt + c[4:] for c in STRADDLE for pt in c[3]], ids=str)
def test_different_domains_inside_a_cta(dim, N, meshes, prec, tol, per_sm):
    probs = [_problem(dim, N, n, p, 7 + k, bounded=k == 1) for k, (n, p) in enumerate(meshes)]
    hanging = meshes[0][1] > 0
    kernel, _, _, per = bf.tile_kernels(dim, N, prec, hanging)[0]
    assert kernel == "pack" and per > 1
    # of a mesh with hanging faces at least 0.7 are in the first launch
    assert (0.7 if hanging else 1.0) * sum(p[0].K for p in probs) > per_sm * 148
    alone = _alone(probs, prec, 2)
    for (q, _), prob in zip(alone, probs):
        assert relerr(q, _oracle(prob, 2)).max() < tol
    doms = [_domain(p, prec) for p in probs]
    b = bf.Batch(doms, t0=0.0)
    assert len(b.groups()) == 1
    b.step([p[5] for p in probs], 2)
    for d, (q, _) in zip(doms, alone):
        assert np.array_equal(d.get_fields(), q)
    b.free()


# one mesh per shape above the sizes below which other kernels or one element
# per CTA serve it: right-hand side, boundary faces, hanging faces, point source
LARGE = [(2, 1, (29, 27), 0.4, PREC), (2, 2, (31, 23), 0.4, PREC), (2, 6, (47, 43), 0.4, PREC),
         (2, 7, (53, 51), 0.4, [F64]), (2, 8, (47, 43), 0.4, [F32]), (3, 1, (9, 8, 8), 0.4, PREC),
         (3, 2, (40, 39, 39), 0.0, [F64]), (3, 2, (13, 12, 12), 0.0, [F32]),
         (3, 2, (16, 14, 15), 0.35, PREC)]


@pytest.mark.parametrize("dim,N,n,p,prec,tol", [c[:4] + pt for c in LARGE for pt in c[4]], ids=str)
def test_packed_kernel_on_large_meshes(dim, N, n, p, prec, tol):
    prob = _problem(dim, N, n, p, 2, bounded=True)
    m, rho, lam, mu, q, dt = prob
    d = _domain(prob, prec)
    assert d.kernel_names()[0] == "dg_pack_kernel"
    o = orc.Oracle.from_mesh(m, rho, lam, mu, 0, bc=_bc(dim))
    # one FP32 evaluation, before the update damps it by dt: 1e-4
    assert relerr(d.rhs(), o.rhs(q)).max() < (1e-12 if prec == bf.PRECISION_FP64 else 1e-4)
    d.set_source(*SRC)
    d.set_receivers(np.array([[0.2, 0.7, 0.1]]), 2)
    bf.LSRK(d).step(dt, 2, use_graph=True)
    assert relerr(d.get_fields(), _oracle(prob, 2, source=True)).max() < tol
