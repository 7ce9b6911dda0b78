"""What creating a domain or a batch sets up: the stage kernels that its mesh
launches (each is loaded by its set-up) and no others, and the right-hand
side's kernel at its first call.  Counts are exact."""
from __future__ import annotations

import numpy as np
import pytest

import bfam_b200 as bf
from bfam_b200 import configs

pytestmark = pytest.mark.gpu


def _domain(dim, N, n, p, prec=bf.PRECISION_FP64):
    m = bf.Mesh(dim, N, n, refine_prob=p, seed=3)
    rho, lam, mu = bf.material_random(m.K, 1)
    return m, bf.GpuDomain(m, rho, lam, mu, precision=prec), configs.stable_dt(m, rho, lam, mu, 0.3)


# 3D order 2: both sides of the size from which the packed kernel serves it
@pytest.mark.parametrize("dim,N,n", [(2, 4, (6, 5)), (3, 1, (3, 3, 3)), (3, 2, (3, 3, 3)),
                                     (3, 2, (13, 12, 12)), (3, 3, (3, 3, 3)), (3, 5, (3, 3, 2)),
                                     (3, 6, (2, 2, 2)), (3, 7, (2, 2, 2))], ids=str)
@pytest.mark.parametrize("p", [0.0, 0.4])
@pytest.mark.parametrize("prec", [bf.PRECISION_FP64, bf.PRECISION_FP32], ids=["fp64", "fp32"])
def test_a_domain_sets_up_what_it_launches(dim, N, n, p, prec):
    c0 = bf.prepare_count()
    m, d, dt = _domain(dim, N, n, p, prec)
    levels = d.launch_levels()
    assert levels == (2 if p else 1)
    # a kernel per launch level (level 0 has no coarse-side faces)
    assert bf.prepare_count() - c0 == levels
    d.set_fields(np.random.default_rng(0).standard_normal((m.nfields, m.K * m.Np)))
    bf.LSRK(d).step(dt, 2, use_graph=True)
    assert bf.prepare_count() - c0 == levels
    a = d.rhs()
    one = bf.prepare_count() - c0 - levels
    assert 1 <= one <= levels  # by size the levels may differ in kernel
    assert np.array_equal(d.rhs(), a)
    assert bf.prepare_count() - c0 == levels + one
    # alone in a batch: the domain's kernels
    b = bf.Batch([d])
    b.step([dt], 2)
    assert bf.prepare_count() - c0 == levels + one
    b.free()


@pytest.mark.parametrize("p", [0.0, 0.4])
def test_a_batch_sets_up_what_it_launches(p):
    pair = [_domain(3, 3, (3, 3, 3), p), _domain(3, 3, (2, 3, 2), p)]
    c0 = bf.prepare_count()
    b = bf.Batch([x[1] for x in pair])
    assert len(b.groups()) == 1
    assert bf.prepare_count() - c0 == (2 if p else 1)
    b.step([x[2] for x in pair], 2)
    assert bf.prepare_count() - c0 == (2 if p else 1)
    b.free()
