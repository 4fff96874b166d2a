"""The gather kernel's tiles and forms, and the operand layouts the tcgen05 kernel stages, at the sizes where they can go wrong.

FP64 is held to the reference's criterion, Float32 on the gather kernel to plain IEEE single precision: every output is a
chain of K fused multiply-adds, each off by at most half a unit in the last place of its partial sum, so that
|err| <= K 2^-24 sum|ab| (and twice that with the partial sums of a cluster split).
"""
import numpy as np
import pytest

from cases import to_equation
from oracle_lib import F32, F64, Contraction
from test_contraction_gpu import check, run_contraction

pytestmark = pytest.mark.gpu

# one row or column more and less than the tiles of 32, 64 and 128; contracted extents around the k tile of 16, the ring of
# four, and past the 256 entries of the k table; rows cut in two modes (A's stride-1 mode is not C's)
GATHER_SHAPES = {
    "outer_product": ("ab", "a", "b", dict(a=65, b=33)),
    "below_tiles": ("ab", "ak", "kb", dict(a=127, b=31, k=15)),
    "above_tiles": ("ab", "ka", "bk", dict(a=129, b=65, k=17)),
    "k_ring": ("abc", "adc", "db", dict(a=13, c=5, b=33, d=65)),
    "k_past_table": ("ab", "kal", "lbk", dict(a=37, b=35, k=19, l=31)),
    "k_many": ("ab", "akl", "lkb", dict(a=5, b=7, k=61, l=67)),
    "rows_cut": ("abcd", "dbea", "ec", dict(a=19, b=3, c=7, d=21, e=33)),
    "rows_cut_c_larger": ("abcde", "efba", "cfd", dict(a=31, b=3, c=9, d=7, e=29, f=5)),
    "columns_reordered": ("abcd", "aebf", "dfce", dict(a=11, b=3, c=9, d=13, e=7, f=5)),
}


@pytest.mark.parametrize("name", list(GATHER_SHAPES))
@pytest.mark.parametrize("scalar", [F32, F64], ids=["f32", "f64"])
def test_gather_kernel_forms(engine, oracle, monkeypatch, name, scalar):
    modes = GATHER_SHAPES[name]
    c = Contraction(*modes[:3], modes[3], scalar)
    A, B = oracle.inputs(c, 5, -1.0, 1.0)
    exact = oracle.contract(c, A, B, rounding=0) if scalar == F32 else oracle.contract(c, A, B)
    scale = oracle.contract(c, np.abs(A), np.abs(B), rounding=0) if scalar == F32 else oracle.contract(c, np.abs(A), np.abs(B))
    k = 1
    for m, e in modes[3].items():
        k *= 1 if m in modes[0] else e
    unit = 2.0 ** (-24 if scalar == F32 else -53)
    monkeypatch.setenv("TCONT_KERNEL", "gather" if scalar == F64 else "simt")
    forms = [(t, s, f) for t in range(3 if scalar == F64 else 4) for s, f in ((1, 0), (1, 1), (2, 0), (8, 0), (16, 0))]
    seen = set()
    for tile, cluster, flat in forms:
        monkeypatch.setenv("TCONT_GATHER_TILE", str(tile))
        monkeypatch.setenv("TCONT_GATHER_CLUSTER", str(cluster))
        monkeypatch.setenv("TCONT_GATHER_FLAT", str(flat))
        p = engine.plan(to_equation(engine, c, 1))
        d = p.describe()
        assert d["kernel"] in ("simt", "dmma_f64")
        form = (d["gather"]["tile"], d["gather"]["cluster"], d["gather"]["flat"])
        if cluster == 1 or cluster <= k // 32:     # (at least two k tiles of 16 for every CTA of a cluster)
            assert form == (tile, cluster, bool(flat) and (scalar == F64 or tile != 2)), form   # (no persistent form of the small Float32 tile)
        form += (d["gather"]["t0"], d["gather"]["rows"])
        if form in seen:
            continue   # (a cluster longer than the contracted extent: one CTA per tile instead)
        seen.add(form)
        r = engine.prepare(p, A, B)
        engine.launch(r)
        out = engine.copy_output_to_host(r)
        worst = float((np.abs(out.astype(np.float64) - exact) / (scale + 1e-300)).max())
        assert worst <= 2.0 * (k + 2) * unit, (tile, cluster, flat, worst)
        r.set_scalars(2.0, 1.0)                    # 2 A B + A B: exact multiples up to one rounding
        engine.launch(r)
        np.testing.assert_allclose(engine.copy_output_to_host(r).astype(np.float64), 3.0 * out.astype(np.float64), rtol=4 * unit, atol=0)


# both operands moved into matrices whose rows are two modes each: 72 = 2.25 slabs, fused 5 184 / 1 296 / ...
MATRICES = {
    "72_extents": ("abcd", "aedf", "fbec", dict(a=72, b=40, c=56, d=24, e=40, f=24)),
    "runs_past_the_end": ("abcd", "aecf", "fbed", dict(a=40, b=72, c=56, d=24, e=40, f=40)),
    "short_rows": ("abcd", "aecf", "fbed", dict(a=20, b=36, c=44, d=60, e=72, f=40)),
}


@pytest.mark.parametrize("name", list(MATRICES))
@pytest.mark.parametrize("pair", ["auto", "0"])
def test_float32_operands_as_matrices(engine, oracle, monkeypatch, name, pair):
    modes = MATRICES[name]
    if pair == "0":
        monkeypatch.setenv("TCONT_UMMA_PAIR", "0")
    c = Contraction(*modes[:3], modes[3], F32)
    A, B = oracle.inputs(c, 7, -1.0, 1.0)
    out, desc = run_contraction(engine, c, A, B, 2)
    assert desc["kernel"] == "umma_tf32" and desc["backend"] == "ttgt", desc
    check(oracle, c, A, B, out, desc)
