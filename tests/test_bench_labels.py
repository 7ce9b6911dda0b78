"""The bench line's kernel name and DRAM traffic are those of the kernels that
ran: names from the library's dispatch, traffic only where that problem, size,
form and kernel were captured."""
from __future__ import annotations

import importlib.util
from pathlib import Path

import pytest

import bfam_b200 as bf

ROOT = Path(__file__).resolve().parent.parent


def _bench():
    spec = importlib.util.spec_from_file_location("bench_module", ROOT / "bench.py")
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def test_traffic_is_of_what_was_captured():
    b = _bench()
    mma = ["dg_mma_kernel"] * 2
    assert b.profiled_traffic(b.stage_key("cfg1", 32, False, mma)) == pytest.approx(6.783e9)
    for other in (("cfg1", 32, True, ["dg_stage_kernel"]), ("cfg1", 24, False, mma),
                  ("cfg1", 32, False, ["dg_stage_kernel"]), ("cfg2", 32, False, mma)):
        assert b.profiled_traffic(b.stage_key(*other)) is None


def test_group_kernels():
    b = _bench()
    g = {"dim": 3, "N": 5, "precision": 0, "hanging": True, "domains": 4, "tile": 1,
         "ctas_per_sm": 0}
    assert b.group_kernel(g) == "dg_mma_batch_kernel"
    assert b.group_kernel(dict(g, hanging=False)) == "dg_stage_batch_kernel"
    assert b.group_kernel(dict(g, domains=1, tile=0)) == "dg_mma_kernel"
    assert b.group_kernel(dict(g, precision=1, domains=1, tile=0)) == "dg_stage_kernel"
    assert b.group_kernel(dict(g, N=2, tile=0, precision=1)) == "dg_pack_batch_kernel"


@pytest.mark.gpu
@pytest.mark.parametrize("dim,N,n,p,prec,names", [
    (2, 4, (4, 4), 0.0, 0, ["pack"]), (2, 7, (4, 4), 0.0, 1, ["stage"]),
    (3, 1, (3, 3, 3), 0.4, 0, ["pack", "pack"]), (3, 2, (3, 3, 3), 0.4, 0, ["stage", "stage"]),
    (3, 2, (40, 39, 39), 0.0, 0, ["pack"]), (3, 2, (13, 12, 12), 0.0, 1, ["pack"]),
    (3, 2, (13, 12, 12), 0.0, 0, ["stage"]), (2, 8, (4, 4), 0.4, 0, ["stage", "stage"]),
    (2, 6, (4, 4), 0.4, 0, ["pack", "pack"]), (3, 2, (16, 14, 15), 0.3, 0, ["pack", "stage"]),
    (3, 3, (3, 3, 3), 0.4, 0, ["stage"] * 2), (3, 5, (2, 2, 2), 0.5, 0, ["mma"] * 2),
    (3, 5, (2, 2, 2), 0.0, 0, ["stage"]), (3, 5, (2, 2, 2), 0.5, 1, ["stage"] * 2),
    (3, 6, (2, 2, 2), 0.0, 0, ["mma"]), (3, 7, (2, 2, 2), 0.5, 0, ["mma"] * 2),
    (3, 7, (2, 2, 2), 0.0, 1, ["stage"])], ids=str)
def test_kernel_names(dim, N, n, p, prec, names):
    m = bf.Mesh(dim, N, n, refine_prob=p, seed=2)
    d = bf.GpuDomain(m, *bf.material_random(m.K, 1), precision=prec)
    assert d.kernel_names() == [f"dg_{k}_kernel" for k in names]
