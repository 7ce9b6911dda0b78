"""The matrix-instruction stage kernel (plain form, 3D orders 6 and 7, and
order 5 on meshes with hanging faces) at the
sizes where its copies and its layout can go wrong, against the oracle: a
single element that is its own neighbour, odd and even element counts (rows
of an odd number of nodes start off the 16-byte boundary in alternation, and
the last row of an odd-sized state has nothing after it), hanging faces of
every piece, boundary faces, and a point source.

Bar: 1e-12 relative L2 per field, as for every FP64 form; the two orders of
summation differ by a few ulp (1e-16) per term over at most 3 x 8 terms."""
from __future__ import annotations

import numpy as np
import pytest

import bfam_b200 as bf
from bfam_b200 import configs
from oracle import oracle as orc
from conftest import relerr

pytestmark = pytest.mark.gpu

CASES = [
    # base cells, refine prob, seed, bounded
    ((1, 1, 1), 0.0, 0, False),
    ((1, 1, 2), 0.0, 0, False),
    ((3, 1, 1), 0.0, 1, True),
    ((2, 2, 2), 0.5, 2, False),
    ((2, 3, 2), 0.4, 3, True),
]


@pytest.mark.parametrize("N", [5, 6, 7])
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}-p{c[1]}-b{int(c[3])}")
@pytest.mark.parametrize("flux", [bf.FLUX_UPWIND, bf.FLUX_CENTRAL], ids=["upwind", "central"])
def test_mma_kernel_against_the_oracle(N, case, flux):
    n, p, seed, bounded = case
    m = bf.Mesh(3, N, n, refine_prob=p, seed=seed, periodic=(not bounded,) * 3)
    rho, lam, mu = bf.material_random(m.K, seed + 3)
    bc = (bf.BC_ABSORBING, bf.BC_FREE_SURFACE) * 3
    q = np.random.default_rng(seed).standard_normal((m.nfields, m.K * m.Np))
    dom = bf.GpuDomain(m, rho, lam, mu, flux=flux, bc=bc)
    o = orc.Oracle.from_mesh(m, rho, lam, mu, flux, bc=bc if bounded else 0)
    dom.set_fields(q)
    assert relerr(dom.rhs(), o.rhs(q)).max() < 1e-12
    dt = configs.stable_dt(m, rho, lam, mu, 0.3)
    bf.LSRK(dom).step(dt, 3, use_graph=True)
    got = dom.get_fields()
    assert relerr(got, o.lsrk(q, dt, 3)).max() < 1e-12
    # in a batch: the same arithmetic
    dom.set_fields(q)
    b = bf.Batch([dom], t0=0.0)
    b.step(dt, 3)
    assert np.array_equal(dom.get_fields(), got)
    b.free()


@pytest.mark.parametrize("N", [5, 6, 7])
def test_mma_kernel_point_source(N):
    m = bf.Mesh(3, N, (2, 2, 1), refine_prob=0.5, seed=4)
    rho, lam, mu = bf.material_random(m.K, 4)
    recv = np.random.default_rng(1).uniform(0.05, 0.95, (5, 3))
    src = ((0.41, 0.57, 0.33), (0.3, -0.2, 1.0), 10.0, 0.02)
    dt = configs.stable_dt(m, rho, lam, mu, 0.5)
    dom = bf.GpuDomain(m, rho, lam, mu)
    dom.set_source(*src)
    dom.set_receivers(recv, 12)
    bf.LSRK(dom).step(dt, 12, use_graph=True)
    o = orc.Oracle.from_mesh(m, rho, lam, mu)
    o.set_source(*src)
    qr, sr = o.seismograms(m.empty_fields(), 0.0, dt, 12, recv)
    assert relerr(dom.get_fields(), qr).max() < 1e-12
    s = dom.seismograms()
    assert np.abs(s - sr).max() <= 1e-12 * np.abs(sr).max()
