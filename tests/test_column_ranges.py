"""Contracted-mode split: where the planner says that C cuts into ranges along tile columns, every column of every tile must
lie in the range of the rank that owns the tile (planner only, no GPU; columns are numbered here from the description)."""
import numpy as np

from cases import random_contraction, to_equation
from oracle_lib import F32, Contraction


def describe(engine, c, selection=0):
    return engine.plan(to_equation(engine, c, selection)).describe()


def index_of_slowest_mode(d):
    """For each tile column and slot of it: the index of C's slowest mode the slot holds, -1 where it holds nothing."""
    u = d["umma"]
    ext = dict((m.rsplit(":", 1)[0], int(m.rsplit(":", 1)[1])) for m in d["N"])
    names, slow = list(ext), list(ext)[-1]
    w, per_tile = u["b_slab_w"], u["b_slabs"]
    if u["b_fused"]:
        slab_modes, rest = names[:2], names[2:]
        assert ext[names[0]] == u["b_fused"]
    else:
        first = d["B"][0].rsplit(":", 1)[0] if u["b_major"] == "MN" else names[0]
        slab_modes, rest = [first], [n for n in names if n != first]
    slab_ext = int(np.prod([ext[m] for m in slab_modes]))
    digits = [-(-slab_ext // w)] + [ext[m] for m in rest]
    out = np.full((u["tiles_n"], per_tile * w), -1)
    for slab in range(int(np.prod(digits))):
        rem, idx = slab, []
        for e in digits:
            idx.append(rem % e)
            rem //= e
        for i in range(w):
            at = idx[0] * w + i
            if at >= slab_ext:
                continue
            value = dict(zip(rest, idx[1:]))
            value.update(zip(slab_modes, (at % ext[slab_modes[0]], at // ext[slab_modes[0]])))
            out[slab // per_tile, slab % per_tile * w + i] = value[slow]
    return out, ext[slow]


def check(d):
    owned, extent = index_of_slowest_mode(d)
    for ranks in d["umma"]["column_ranges"]:
        assert extent % ranks == 0 and owned.shape[0] % ranks == 0, d
        per = owned.shape[0] // ranks
        for tile, row in enumerate(owned):
            assert set(row[row >= 0] // (extent // ranks)) <= {tile // per}, (ranks, tile, d)


def test_fused_columns_that_end_inside_a_slab_are_not_cut(engine, monkeypatch):
    monkeypatch.setenv("TCONT_SPLITK", "1")
    # c and d fuse into 1 008 columns in 32 slabs (31.5 used): half of C ends inside a tile column
    d = describe(engine, Contraction("acbd", "abk", "cdk", dict(a=64, b=64, c=36, d=28, k=64), F32), 1)
    assert d["kernel"] == "umma_tf32" and d["umma"]["b_fused"] == 36 and d["umma"]["tiles_n"] % 2 == 0
    assert 2 not in d["umma"]["column_ranges"]
    # the same with whole slabs per half
    d = describe(engine, Contraction("acbd", "abk", "cdk", dict(a=64, b=64, c=40, d=64, k=64), F32), 1)
    assert d["umma"]["b_fused"] == 40 and 2 in d["umma"]["column_ranges"]
    check(d)


def test_slowest_mode_that_is_the_slab_mode_is_not_cut(engine, monkeypatch):
    monkeypatch.setenv("TCONT_SPLITK", "1")
    # B's stride-1 mode d is C's slowest: its chunks are the fastest digit of the column slabs, the ranges would be c's
    d = describe(engine, Contraction("acd", "ak", "dkc", dict(a=64, c=16, d=64, k=64), F32), 1)
    assert d["kernel"] == "umma_tf32" and d["umma"]["b_major"] == "MN" and d["umma"]["column_ranges"] == []


def test_every_tile_column_has_one_owner(engine, monkeypatch):
    monkeypatch.setenv("TCONT_SPLITK", "1")
    rng = np.random.default_rng(11)
    pool = (2, 4, 6, 8, 12, 16, 20, 24, 32, 36, 40, 64, 72, 96)
    cut = fused = 0
    for _ in range(1500):
        c = random_contraction(rng, F32, max_out=3_000_000, max_macs=10**9, pool=pool)
        d = describe(engine, c)
        if d["kernel"] == "umma_tf32" and d["umma"]["column_ranges"]:
            cut += 1
            fused += d["umma"]["b_fused"] > 0
            check(d)
    assert cut > 100 and fused > 10
