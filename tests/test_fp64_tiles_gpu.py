"""Tiles and chunks of the TMA-fed FP64 kernel at the sizes where they can go wrong, against the CPU oracle.

Every output is a chain of K fused multiply-adds (in ranges with split-K), each off by at most 2^-53 of its partial sum:
|err| <= (K + splits) 2^-53 sum|ab|.
"""
import numpy as np
import pytest

from cases import to_equation
from oracle_lib import F64, Contraction
from test_contraction_gpu import run_contraction
from test_scaled_epilogues_gpu import scaled_run

pytestmark = pytest.mark.gpu


def hold(oracle, c, A, B, out, k, splits=1):
    exact, scale = oracle.contract(c, A, B), oracle.contract(c, np.abs(A), np.abs(B))
    assert (np.abs(out - exact) <= (k + splits) * 2.0**-53 * scale).all()


# chunked mode: whole chunks of 16, one k to eight past them (half a chunk is left out), more than eight past them, one
# chunk in all; alone, and as the first of two contracted modes, where a short chunk comes back every few iterations
@pytest.mark.parametrize("chunked", [16, 18, 40, 42, 48, 56, 58, 72])
@pytest.mark.parametrize("layout", ["k_k", "mn_mn", "mn_k_two", "k_mn_two"])
@pytest.mark.parametrize("splits", ["1", "3"])
def test_last_chunk_of_eight_or_fewer(engine, oracle, monkeypatch, chunked, layout, splits):
    monkeypatch.setenv("TCONT_KERNEL", "tma")
    monkeypatch.setenv("TCONT_SPLITK", splits)
    C, A_, B_, other = {"k_k": ("ab", "ka", "kb", 1), "mn_mn": ("ab", "ak", "bk", 1), "mn_k_two": ("ab", "alk", "klb", 5),
                        "k_mn_two": ("ab", "kal", "blk", 3)}[layout]
    ext = dict(a=132, b=70, k=chunked)
    if other > 1:
        ext["l"] = other
    c = Contraction(C, A_, B_, ext, F64)
    A, B = oracle.inputs(c, 29, -1.0, 1.0)
    out, desc = run_contraction(engine, c, A, B, 1)
    u = desc["umma"]
    assert desc["kernel"] == "dmma_f64_tma"
    hold(oracle, c, A, B, out, chunked * other, u["k_splits"])


# the epilogue's straight-line form (whole tiles, everything on multiples of 32 bytes) and the other one, tile by tile: ragged
# last tiles, columns on odd multiples of 16 bytes (a = 130), C itself on one, fused rows, tiles across slabs, several tiles a group
STORES = {
    "whole": ("ab", "ak", "kb", dict(a=512, b=320, k=24), 0),
    "last_tiles_ragged": ("ab", "ka", "bk", dict(a=1028, b=1060, k=16), 0),
    "odd_columns": ("ab", "ak", "kb", dict(a=130, b=640, k=24), 0),
    "odd_c": ("ab", "ak", "kb", dict(a=512, b=320, k=24), 2),
    "fused_rows": ("acb", "abk", "kc", dict(a=12, b=60, c=128, k=24), 0),
    "fused_rows_odd": ("acb", "abk", "kc", dict(a=6, b=50, c=128, k=24), 0),
    "across_slabs": ("abcd", "dbea", "ec", dict(a=24, b=9, c=64, d=48, e=24), 0),
    # one column of tiles that C fills to three quarters or less: fewer column fragments, the last one not one of a pair
    "slim_24": ("ab", "ak", "kb", dict(a=1540, b=24, k=24), 0),
    "slim_17": ("ab", "ka", "kb", dict(a=1540, b=17, k=40), 0),
    "slim_48": ("ab", "ak", "kb", dict(a=1540, b=48, k=24), 0),
    "slim_33": ("ab", "ka", "kb", dict(a=1538, b=33, k=40), 0),
    "slim_across_slabs": ("abcd", "dbea", "ec", dict(a=24, b=9, c=24, d=48, e=24), 0),
    "slim_across_slabs_48": ("abcd", "dbea", "ec", dict(a=24, b=9, c=42, d=40, e=40), 0),
    # a last column of tiles that is not filled, B along k and along its columns; pieces of two elements (C's strides 2 modulo 4),
    # with few and many k chunks; of one (odd strides)
    "columns_56": ("ab", "ak", "kb", dict(a=1540, b=56, k=24), 0),
    "columns_40_mn": ("ab", "ak", "bk", dict(a=1540, b=40, k=24), 0),
    "halves": ("ab", "ak", "bk", dict(a=1030, b=150, k=40), 0),
    "halves_many_chunks": ("ab", "ka", "kb", dict(a=1030, b=150, k=136), 0),
    "slim_halves": ("ab", "ak", "kb", dict(a=1538, b=22, k=40), 0),
    "odd_strides": ("ab", "ka", "kb", dict(a=1029, b=149, k=40), 0),
    "across_slabs_ragged": ("abcd", "dbea", "ec", dict(a=24, b=9, c=60, d=54, e=40), 0),
}


@pytest.mark.parametrize("name", list(STORES))
@pytest.mark.parametrize("beta", [0.0, -0.7])
def test_stores(engine, oracle, monkeypatch, name, beta):
    import torch
    from tcont_b200 import api
    monkeypatch.setenv("TCONT_KERNEL", "tma")
    monkeypatch.setenv("TCONT_SPLITK", "1")
    monkeypatch.setenv("TCONT_SCALE_PASSES", "1")
    C, A_, B_, ext, shift = STORES[name]
    c = Contraction(C, A_, B_, ext, F64)
    A, B = oracle.inputs(c, 31, -1.0, 1.0)
    n = c.size(C)
    C0 = np.random.default_rng(7).uniform(-4.0, 4.0, n)
    guarded = torch.full((n + 16,), 7.0, dtype=torch.float64, device="cuda")
    dC = guarded[shift:shift + n]
    dC.copy_(torch.from_numpy(C0))
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    plan = engine.plan(to_equation(engine, c, 1))
    run = api.prepare_on_device(plan, dA.data_ptr(), dB.data_ptr(), dC.data_ptr(), keep=(dA, dB, guarded))
    run.set_scalars(1.0, beta)
    engine.launch(run)
    torch.cuda.synchronize()
    u = plan.describe()["umma"]
    assert plan.describe()["kernel"] == "dmma_f64_tma" and u["slim"] == name.startswith("slim") and run.device_status() == 0
    outside = torch.cat([guarded[:shift], guarded[shift + n:]])
    assert bool((outside == 7.0).all())
    exact, scale = oracle.contract(c, A, B) + beta * C0, oracle.contract(c, np.abs(A), np.abs(B)) + abs(beta * C0)
    k = ext.get("k", ext.get("e"))
    assert (np.abs(dC.cpu().numpy() - exact) <= (k + 4) * 2.0**-53 * scale).all()


@pytest.mark.parametrize("rows", [128, 130, 131])
def test_rows_of_a_view(engine, oracle, monkeypatch, rows):
    """C's columns lie on multiples of 32 bytes whatever their extent: pieces that C ends in are not stored whole."""
    import torch
    from tcont_b200 import api
    monkeypatch.setenv("TCONT_KERNEL", "tma")
    c = Contraction("ab", "ka", "kb", dict(a=rows, b=70, k=40), F64)
    A, B = oracle.inputs(c, 37, -1.0, 1.0)
    big = torch.full((70, 136), 7.0, dtype=torch.float64, device="cuda")
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    plan = api.plan_views(to_equation(engine, c, 1), parent_c=[136, 70])
    u = plan.describe()["umma"]
    assert plan.describe()["kernel"] == "dmma_f64_tma" and u["piece"] == (4 if rows % 4 == 0 else 2 if rows % 2 == 0 else 1), u
    run = api.prepare_on_device(plan, dA.data_ptr(), dB.data_ptr(), big.data_ptr(), keep=(dA, dB, big))
    engine.launch(run)
    torch.cuda.synchronize()
    hold(oracle, c, A, B, big[:, :rows].contiguous().cpu().numpy().reshape(-1), 40)
    big[:, :rows] = 7.0
    assert bool((big == 7.0).all()) and run.device_status() == 0


# odd strides: both operands copied to matrices whose strides are even, rows in one run or several, contracted modes in A's order,
# in B's or in neither's, an operand that already lies in the right order, one that needs no padding
PADDED = {
    "four_d": ("abcd", "aebf", "fdec", dict(a=61, b=5, c=7, d=9, e=13, f=23)),
    "rows_apart": ("abcd", "aecf", "bfde", dict(a=19, b=7, c=11, d=13, e=9, f=15)),
    "in_order": ("ab", "ak", "kb", dict(a=131, b=67, k=35)),
    "even_rows": ("abc", "adc", "db", dict(a=38, b=45, c=7, d=21)),
    "even_k": ("abcd", "eafd", "fbec", dict(a=21, b=13, c=9, d=15, e=6, f=11)),
    "swapped": ("abc", "db", "adc", dict(a=33, b=27, c=5, d=41)),
    "long_k": ("ab", "ac", "cb", dict(a=45, b=33, c=1001)),
}


@pytest.mark.parametrize("name", list(PADDED))
def test_padded_copies(engine, oracle, monkeypatch, name):
    monkeypatch.setenv("TCONT_PADDED_COPIES", "1")
    monkeypatch.setenv("TCONT_KERNEL", "tma")
    C, A_, B_, ext = PADDED[name]
    c = Contraction(C, A_, B_, ext, F64)
    A, B = oracle.inputs(c, 43, -1.0, 1.0)
    out, desc = run_contraction(engine, c, A, B, 2, launches=2)
    assert desc["kernel"] == "dmma_f64_tma" and desc["backend"] == "ttgt" and not desc["views"], desc
    k = 1
    for m, e in ext.items():
        k *= 1 if m in C else e
    hold(oracle, c, A, B, out, k, desc["umma"]["k_splits"])


@pytest.mark.parametrize("name", ["four_d", "in_order", "even_rows"])
def test_accumulating_behind_padded_copies(engine, oracle, monkeypatch, name):
    monkeypatch.setenv("TCONT_PADDED_COPIES", "1")
    monkeypatch.setenv("TCONT_KERNEL", "tma")
    C, A_, B_, ext = PADDED[name]
    c = Contraction(C, A_, B_, ext, F64)
    A, B = oracle.inputs(c, 43, -1.0, 1.0)
    C0 = np.random.default_rng(13).uniform(-4.0, 4.0, c.size(C))
    desc, (out,) = scaled_run(engine, c, A, B, C0, [(0.3, -0.7)], 2)
    assert desc["kernel"] == "dmma_f64_tma" and desc["backend"] == "ttgt", desc
    k = int(np.prod([e for m, e in ext.items() if m not in C]))
    want, scale = 0.3 * oracle.contract(c, A, B) - 0.7 * C0, 0.3 * oracle.contract(c, np.abs(A), np.abs(B)) + 0.7 * np.abs(C0)
    assert (np.abs(out - want) <= (k + desc["umma"]["k_splits"] + 4) * 2.0**-53 * scale).all()
