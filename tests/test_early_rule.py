"""Which stages let the next launch's CTAs in before their end: on the host the
rule's ranges (as fractions of a wave of resident CTAs, and never on at most a
CTA per SM), on the GPU the same bits whichever way."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import bfam_b200 as bf
from bfam_b200 import configs
from bfam_b200.build import NVCC_ARCH, _nvcc

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.skipif(not (shutil.which("nvcc") or Path("/usr/local/cuda/bin/nvcc").exists()),
                    reason="no nvcc")
def test_ranges(tmp_path):
    exe = tmp_path / "early"
    subprocess.run([_nvcc(), *NVCC_ARCH, "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", str(ROOT / "include"), "-I", str(ROOT / "bfam_b200" / "csrc"),
                    "-o", str(exe), str(ROOT / "tests" / "c" / "early_check.cu")], check=True)
    out = {r.split()[0]: tuple(map(int, r.split()[1:])) for r in
           subprocess.run([str(exe)], check=True, capture_output=True,
                          text=True).stdout.splitlines()}
    # per cent of a wave from which the next launch waits; none: never
    want = {"node-3-fp64": None, "node-4-fp64": 50, "node-5-fp64": 50, "node-5-fp32": 42,
            "node-2d-7": None, "mma-5": 34, "mma-6": 42, "mma-7": None,
            "node-7-fp32": None}
    assert set(out) == set(want)
    for name, lo in want.items():
        slots, first, last, holes = out[name]
        if lo is None:
            assert (first, last) == (0, 0), name
            continue
        ctas = np.arange(1, 2 * slots + 1)
        late = ctas[(ctas > 148) & (100 * ctas > lo * slots) & (100 * ctas < 85 * slots)]
        assert (first, last, holes) == (late[0], late[-1], 0), name


# sizes inside the ranges
@pytest.mark.gpu
@pytest.mark.parametrize("N,n,p,prec", [(4, (8, 8, 8), 0.0, bf.PRECISION_FP64),
                                        (5, (8, 8, 8), 0.0, bf.PRECISION_FP64),
                                        (5, (6, 5, 4), 0.4, bf.PRECISION_FP64),
                                        (5, (7, 6, 6), 0.0, bf.PRECISION_FP32),
                                        (6, (7, 6, 6), 0.0, bf.PRECISION_FP64),
                                        (6, (4, 4, 4), 0.5, bf.PRECISION_FP64)])
def test_same_bits(N, n, p, prec):
    m = bf.Mesh(3, N, n, refine_prob=p, seed=1)
    rho, lam, mu = bf.material_random(m.K, 2)
    q = np.random.default_rng(3).standard_normal((m.nfields, m.K * m.Np))
    dt = configs.stable_dt(m, rho, lam, mu, 0.3)
    out = []
    for graph in (False, True):
        d = bf.GpuDomain(m, rho, lam, mu, precision=prec)
        d.set_fields(q)
        bf.LSRK(d).step(dt, 6, use_graph=graph)
        out.append(d.get_fields())
    # beside a domain of another order the launches do not overlap at all
    d = bf.GpuDomain(m, rho, lam, mu, precision=prec)
    d.set_fields(q)
    m2 = bf.Mesh(3, 1, (2, 2, 2))
    other = bf.GpuDomain(m2, *bf.material_random(m2.K, 0))
    other.set_fields(m2.empty_fields())
    b = bf.Batch([d, other])
    b.step([dt, dt], 6)
    out.append(d.get_fields())
    b.free()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
