"""The tuner times the kernels that the tuned group runs: one domain or
several, conforming or with hanging faces, each under its own cache entry."""
from __future__ import annotations

import pytest

import bfam_b200 as bf
from bfam_b200 import autotune


class _FakeBatch:
    def __init__(self, groups):
        self._groups, self.tiles = groups, {}

    def groups(self):
        return self._groups

    def set_tile(self, g, tile, cps):
        self.tiles[g] = (tile, cps)


def _info(N, precision, domains, hanging):
    return {"dim": 3, "N": N, "precision": precision, "elements": 500, "domains": domains,
            "hanging": hanging}


def test_groups_are_tuned_by_kind(monkeypatch):
    import torch
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda d=0: "GPU")
    calls = []

    def tune(dim, N, precision, elements, device=0, hanging=True, domains=1):
        calls.append((N, precision, hanging, domains == 1))
        return {"best": {"tile": len(calls), "ctas_per_sm": 0}, "table": []}

    monkeypatch.setattr(autotune, "tune_group", tune)
    kinds = [_info(5, 0, 1, True), _info(5, 0, 1, False), _info(5, 0, 4, True),
             _info(5, 0, 4, False), _info(5, 0, 9, False), _info(5, 1, 4, False)]
    b = _FakeBatch(kinds)
    cache = {}
    autotune.autotune(b, cache=cache)
    assert calls == [(5, 0, True, True), (5, 0, False, True), (5, 0, True, False),
                     (5, 0, False, False), (5, 1, False, False)]
    assert len(cache) == 5
    # several conforming domains share an entry whatever their number
    assert [b.tiles[g][0] for g in range(6)] == [1, 2, 3, 4, 4, 5]


@pytest.mark.gpu
@pytest.mark.parametrize("hanging", [False, True])
@pytest.mark.parametrize("domains", [1, 3])
def test_the_tuned_batch_is_of_the_groups_kind(monkeypatch, hanging, domains):
    """the batch that the tuner times is a group of one domain only for a group
    of one, on the same kind of mesh"""
    seen = []
    init = bf.Batch.__init__

    def spy(self, doms, *a, **k):
        init(self, doms, *a, **k)
        seen.append(self.groups())

    monkeypatch.setattr(bf.Batch, "__init__", spy)
    t = autotune.tune_group(3, 5, bf.PRECISION_FP64, 200, steps=1, hanging=hanging,
                            domains=domains)
    (groups,) = seen
    assert len(groups) == 1
    assert (groups[0]["domains"] == 1) == (domains == 1)
    assert groups[0]["hanging"] == hanging
    assert groups[0]["elements"] == t["elements"]
    assert {r["tile"] for r in t["table"]} >= {0, 1}


@pytest.mark.gpu
def test_no_capture_is_timed(monkeypatch):
    """a step is captured once per state parity; both are before the timed steps"""
    calls, tiles = [], []
    step, set_tile = bf.Batch.step, bf.Batch.set_tile
    monkeypatch.setattr(bf.Batch, "step", lambda self, dt, n=1, **k: (
        calls.append((len(tiles), n)), step(self, dt, n, **k))[1])
    monkeypatch.setattr(bf.Batch, "set_tile", lambda self, *a: (
        tiles.append(a), set_tile(self, *a))[1])
    t = autotune.tune_group(3, 4, bf.PRECISION_FP64, 100, steps=3, domains=2)
    assert len(t["table"]) == len(tiles)
    for k in range(1, len(tiles) + 1):
        assert [n for c, n in calls if c == k] == [2, 3]


@pytest.mark.gpu
def test_group_kinds():
    def dom(N, p):
        m = bf.Mesh(3, N, (2, 2, 2), refine_prob=p, seed=2)
        return bf.GpuDomain(m, *bf.material_random(m.K, 1))
    doms = [dom(3, 0.0), dom(3, 0.5), dom(3, 0.0), dom(5, 0.5)]
    b = bf.Batch(doms)
    assert [(g["N"], g["domains"], g["hanging"]) for g in b.groups()] == \
        [(3, 2, False), (3, 1, True), (5, 1, True)]
    b.free()


# kernels of the first tiles: what the dispatch runs
FIRST = [(2, 4, 0, 0, "pack"), (2, 4, 1, 1, "pack"), (2, 7, 0, 0, "pack"), (2, 7, 1, 0, "node"), (2, 8, 0, 0, "node"), (2, 8, 1, 0, "pack"),
         (3, 1, 0, 1, "pack"), (3, 2, 1, 0, "pack"), (3, 2, 0, 0, "node"), (3, 3, 0, 1, "node"), (3, 4, 1, 1, "node"),
         (3, 5, 0, 0, "node"), (3, 5, 0, 1, "mma"), (3, 5, 1, 1, "node"), (3, 6, 0, 0, "mma"),
         (3, 6, 1, 1, "node"), (3, 7, 0, 1, "mma"), (3, 7, 1, 0, "node")]


@pytest.mark.parametrize("dim,N,prec,hanging,kernel", FIRST)
def test_tile_kernels(dim, N, prec, hanging, kernel):
    t = bf.tile_kernels(dim, N, prec, bool(hanging))
    assert t[0][0] == kernel
    # as many as the order's shapes, and no two alike (the precision form's
    # first budget at order 5 is also one of the others)
    assert len(t) == len(bf.tile_shapes(dim, N))
    assert len(set(t)) == len(t) - ((dim, N, prec) == (3, 5, 1))
    for name, threads, minb, elements in t:
        assert threads % 32 == 0 and threads <= 1024 and minb >= 1 and elements >= 1
        assert name != "mma" or (threads == 32 * (N + 1) and elements == 1)


def test_cache_key_names_the_kernels():
    """a tile index is not reused for a group that runs other kernels under it"""
    key = lambda *a, **k: autotune._key("GPU", *a, **k)
    keys = {key(3, 5, 0, hanging=h, domains=d) for h in (False, True) for d in (1, 5)}
    assert len(keys) == 4
    assert key(3, 5, 0, domains=2) == key(3, 5, 0, domains=7)
    assert "kernels:mma." in key(3, 5, 0, hanging=True)
    assert "kernels:node." in key(3, 5, 0, hanging=False)
    assert "kernels:pack." in key(2, 4, 0) and "kernels:pack." in key(3, 2, 1)
    assert "kernels:mma." in key(3, 7, 0) and "kernels:node." in key(3, 7, 1)
