"""Receiver sampling spread over CTAs: counts around the number of receiver
CTAs of a domain (64), alone and in a batch beside domains with fewer or no
receivers; groups of one domain run the single-domain kernel in a batch.

Bar: samples to 1e-12 of the largest against the oracle (as elsewhere), and
bitwise equal alone and in the batch; clocks advance once per step."""
from __future__ import annotations

import numpy as np
import pytest

import bfam_b200 as bf
from bfam_b200 import configs
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _problem(dim, N, n, seed):
    m = bf.Mesh(dim, N, n, refine_prob=0.4, seed=seed)
    rho, lam, mu = bf.material_random(m.K, seed)
    q0 = np.random.default_rng(seed).standard_normal((m.nfields, m.K * m.Np))
    return m, rho, lam, mu, q0, configs.stable_dt(m, rho, lam, mu, 0.4)


@pytest.mark.parametrize("nrecv", [1, 63, 64, 65, 131])
def test_receiver_counts(nrecv):
    steps = 4
    probs = [_problem(3, 2, (2, 2, 2), 1), _problem(2, 3, (3, 4), 2), _problem(3, 2, (1, 2, 2), 3)]
    recvs = [np.random.default_rng(9).uniform(0.02, 0.98, (nrecv, 3)),
             np.random.default_rng(8).uniform(0.02, 0.98, (3, 3)), None]
    alone, doms = [], []
    for (m, rho, lam, mu, q0, dt), rc in zip(probs, recvs):
        for keep in (False, True):
            d = bf.GpuDomain(m, rho, lam, mu)
            d.set_fields(q0)
            if rc is not None:
                d.set_receivers(rc, steps)
            if keep:
                doms.append(d)
            else:
                bf.LSRK(d).step(dt, steps, use_graph=True)
                alone.append((d.get_fields(), d.seismograms() if rc is not None else None))
    m, rho, lam, mu, q0, dt = probs[0]
    _, ref = orc.Oracle.from_mesh(m, rho, lam, mu).seismograms(q0, 0.0, dt, steps, recvs[0])
    assert alone[0][1].shape == (steps, nrecv, 9)
    assert np.abs(alone[0][1] - ref).max() <= 1e-12 * np.abs(ref).max()
    b = bf.Batch(doms, t0=0.0)
    b.step([p[5] for p in probs], steps)
    for i, d in enumerate(doms):
        assert np.array_equal(d.get_fields(), alone[i][0])
        if recvs[i] is not None:
            assert np.array_equal(d.seismograms(), alone[i][1])
        assert abs(b.time(i) - steps * probs[i][5]) < 1e-14
    b.free()
    # the device clocks kept the same time
    b = bf.Batch(doms)
    for i, p in enumerate(probs):
        assert abs(b.time(i) - steps * p[5]) < 1e-14
    b.free()
