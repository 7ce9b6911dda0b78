"""Element rows of an odd number of nodes (3D orders 2, 4, 6) in the
one-element kernel: bulk copies from the 16-byte boundary below a row, for even
and odd element counts, and the last row of an odd-sized state, which has
nothing after it.

Bar: 1e-12 (FP64) and 1e-6 (precision form) relative L2 per field against the
oracle, as everywhere."""
from __future__ import annotations

import numpy as np
import pytest

import bfam_b200 as bf
from bfam_b200 import configs
from oracle import oracle as orc
from conftest import relerr

pytestmark = pytest.mark.gpu

MESHES = [((1, 1, 1), 0.0), ((2, 1, 1), 0.0), ((3, 1, 1), 0.0), ((2, 2, 2), 0.4),
          ((2, 3, 1), 0.5)]


@pytest.mark.parametrize("N,prec", [(4, 0), (4, 1), (6, 1)])
@pytest.mark.parametrize("n,p", MESHES, ids=lambda v: str(v))
def test_odd_rows_against_the_oracle(N, prec, n, p):
    m = bf.Mesh(3, N, n, refine_prob=p, seed=N)
    rho, lam, mu = bf.material_random(m.K, N)
    q = np.random.default_rng(N).standard_normal((m.nfields, m.K * m.Np))
    d = bf.GpuDomain(m, rho, lam, mu, precision=prec)
    d.set_fields(q)
    o = orc.Oracle.from_mesh(m, rho, lam, mu)
    tol = 1e-6 if prec else 1e-12
    if not prec:
        assert relerr(d.rhs(), o.rhs(q)).max() < tol
    dt = configs.stable_dt(m, rho, lam, mu, 0.3)
    bf.LSRK(d).step(dt, 3, use_graph=True)
    assert relerr(d.get_fields(), o.lsrk(q, dt, 3)).max() < tol


@pytest.mark.parametrize("n", [(1, 1, 1), (2, 2, 1), (3, 3, 1)])
def test_odd_rows_several_elements_per_cta(n):
    m = bf.Mesh(3, 2, n)
    rho, lam, mu = bf.material_random(m.K, 1)
    q = np.random.default_rng(1).standard_normal((m.nfields, m.K * m.Np))
    dt = configs.stable_dt(m, rho, lam, mu, 0.3)
    ref = orc.Oracle.from_mesh(m, rho, lam, mu).lsrk(q, dt, 2)
    for tile in range(len(bf.tile_shapes(3, 2))):
        d = bf.GpuDomain(m, rho, lam, mu)
        d.set_fields(q)
        b = bf.Batch([d], t0=0.0)
        b.set_tile(0, tile, 0)
        b.step(dt, 2)
        assert relerr(d.get_fields(), ref).max() < 1e-12, tile
        b.free()
