"""The packed stage kernel (2D, 3D orders 1 and 2) where its packing can go
wrong: element counts around the elements of a CTA (a partly empty last CTA, a
single element), CTAs whose elements mix fine, coarse, conforming and boundary
faces, domains of a batch meeting inside a CTA, and the point source.

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


def _problem(dim, N, n, p, seed, bounded):
    m = bf.Mesh(dim, N, n, refine_prob=p, seed=seed, periodic=(not bounded,) * 3)
    rho, lam, mu = bf.material_random(m.K, seed + 3)
    q = np.random.default_rng(seed).standard_normal((m.nfields, m.K * m.Np))
    return m, rho, lam, mu, q, configs.stable_dt(m, rho, lam, mu, 0.3)


ORDERS = [(2, N) for N in range(1, 9)] + [(3, 1), (3, 2)]
MESHES = [((1, 1, 1), 0.0, False), ((3, 2, 1), 0.0, True), ((3, 3, 2), 0.4, False),
          ((5, 4, 2), 0.5, True)]


@pytest.mark.parametrize("dim,N", ORDERS)
@pytest.mark.parametrize("mesh", MESHES, ids=lambda c: f"{c[0]}-p{c[1]}-b{int(c[2])}")
def test_packed_kernel_against_the_oracle(dim, N, mesh):
    n, p, bounded = mesh
    m, rho, lam, mu, q, dt = _problem(dim, N, n[:dim], p, N, bounded)
    bc = (bf.BC_ABSORBING, bf.BC_FREE_SURFACE) * dim
    o = orc.Oracle.from_mesh(m, rho, lam, mu, 0, bc=bc if bounded else 0)
    ref = o.lsrk(q, dt, 2)
    for prec, tol in ((bf.PRECISION_FP64, 1e-12), (bf.PRECISION_FP32, 1e-6)):
        d = bf.GpuDomain(m, rho, lam, mu, precision=prec, bc=bc)
        d.set_fields(q)
        if prec == bf.PRECISION_FP64:
            assert relerr(d.rhs(), o.rhs(q)).max() < tol
        bf.LSRK(d).step(dt, 2, use_graph=True)
        assert relerr(d.get_fields(), ref).max() < tol


@pytest.mark.parametrize("dim,N", [(2, 1), (2, 3), (2, 4), (2, 8), (3, 1), (3, 2)])
@pytest.mark.parametrize("prec", [bf.PRECISION_FP64, bf.PRECISION_FP32], ids=["fp64", "fp32"])
def test_domains_meeting_inside_a_cta(dim, N, prec):
    probs = [_problem(dim, N, n[:dim], p, s, False)
             for s, (n, p) in enumerate([((1, 1, 1), 0.0), ((3, 2, 1), 0.5), ((2, 2, 2), 0.0),
                                         ((2, 3, 2), 0.4)])]
    alone, doms = [], []
    for m, rho, lam, mu, q, dt in probs:
        for keep in (False, True):
            d = bf.GpuDomain(m, rho, lam, mu, precision=prec)
            d.set_fields(q)
            d.set_source((0.4, 0.3, 0.6), (1.0, -0.5, 0.25), 10.0, 0.01)
            d.set_receivers(np.array([[0.2, 0.7, 0.1]]), 3)
            if keep:
                doms.append(d)
            else:
                bf.LSRK(d).step(dt, 3, use_graph=True)
                alone.append((d.get_fields(), d.seismograms()))
    b = bf.Batch(doms, t0=0.0)
    b.step([p[5] for p in probs], 3)
    for d, (q, s) in zip(doms, alone):
        assert np.array_equal(d.get_fields(), q)
        assert np.array_equal(d.seismograms(), s)
    b.free()


# Meshes whose launches give a CTA two, several or all of the elements that it
# can hold, with a partly empty last CTA, and (3D order 2) launches on either
# side of the size from which the packed kernel serves them.  The counts are of
# the finest level's order: 4 x 148 CTAs before a second element per CTA.
SPREAD = [(2, 1, (29, 23), 0.0), (2, 1, (51, 37), 0.4), (2, 1, (140, 137), 0.0),
          (2, 2, (27, 23), 0.0), (2, 2, (43, 31), 0.4), (2, 2, (97, 89), 0.3),
          (3, 1, (9, 10, 7), 0.0), (3, 1, (9, 8, 7), 0.4), (3, 1, (23, 21, 20), 0.2),
          (3, 2, (11, 12, 13), 0.0), (3, 2, (13, 12, 12), 0.0), (3, 2, (8, 7, 7), 0.4),
          (3, 2, (16, 14, 15), 0.3)]


@pytest.mark.parametrize("dim,N,n,p", SPREAD, ids=str)
@pytest.mark.parametrize("prec,tol", [(bf.PRECISION_FP64, 1e-12), (bf.PRECISION_FP32, 1e-6)],
                         ids=["fp64", "fp32"])
def test_elements_per_cta(dim, N, n, p, prec, tol):
    m, rho, lam, mu, q, dt = _problem(dim, N, n, p, N, False)
    o = orc.Oracle.from_mesh(m, rho, lam, mu, 0)
    ref = o.lsrk(q, dt, 1)
    doms = []
    for _ in range(3):
        d = bf.GpuDomain(m, rho, lam, mu, precision=prec)
        d.set_fields(q)
        doms.append(d)
    bf.LSRK(doms[0]).step(dt, 1)
    alone = doms[0].get_fields()
    assert relerr(alone, ref).max() < tol
    bf.Batch(doms[1:]).step([dt, dt], 1)
    for d in doms[1:]:
        assert np.array_equal(d.get_fields(), alone)
