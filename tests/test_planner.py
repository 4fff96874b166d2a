"""CPU-only: the host-side planner behind TconT::plan, driven through the C ABI."""
import pytest

from cases import CONFIGS, fixture_contraction, golden_fixtures, to_equation
from oracle_lib import F32, F64, Contraction


def describe(engine, c, selection=0):
    return engine.plan(to_equation(engine, c, selection)).describe()


def test_mode_groups_and_fusion(engine):
    d = describe(engine, CONFIGS["cfg3"][0])
    assert d["A"] == ["a:48", "e:48", "ij:576"] and d["B"] == ["bc:2304", "e:48", "k:24"]
    assert d["M"] == ["a:48", "ij:576"] and d["N"] == ["bc:2304", "k:24"] and d["K"] == ["e:48"]
    assert (d["Mtot"], d["Ntot"], d["Ktot"]) == (27648, 55296, 48)
    # cfg5's (a,b) are neighbours in C but split by e in A: nothing may fuse
    d5 = describe(engine, CONFIGS["cfg5"][0])
    assert d5["C"] == ["a:128", "b:128", "c:128", "d:128"]


def test_roles_follow_position_not_names(engine):
    # C's stride-1 mode lives in the right operand: roles are exchanged (the reference keys this
    # on the letter 'a', backends/cogent/plan/tc_gen_inner_group.py:450)
    eq = engine.TCEquation("xyz", "kz", "ykx", dict(x=8, y=4, z=6, k=5))
    d = engine.plan(eq).describe()
    assert d["swapped"] is True and d["M"][0].startswith("x") and d["K"] == ["k:5"]
    eq2 = engine.TCEquation("xyz", "ykx", "kz", dict(x=8, y=4, z=6, k=5))
    assert engine.plan(eq2).describe()["swapped"] is False


def test_backend_selection_and_names(engine):
    c = CONFIGS["cfg1"][0]
    assert engine.plan(to_equation(engine, c, 1)).backend == engine.Backend.COGENT
    p = engine.plan(to_equation(engine, c, 2))
    assert p.backend == engine.Backend.TTGT_CUTT
    d = p.describe()
    # role A = A[a,e,b,f] -> [a,b | f,e] (lead = ab, K in B's order); B[f,d,e,c] is K-major on f and
    # is used where it lies; C never needs a transpose
    assert d["transpose_a"] == [0, 2, 3, 1] and d["transpose_b"] is None
    assert d["A"] == ["ab:576", "f:16", "e:16"] and d["B"] == ["f:16", "d:24", "e:16", "c:24"]


def test_configs_pick_the_intended_kernels(engine):
    d2 = describe(engine, CONFIGS["cfg2"][0])
    assert d2["backend"] == "direct" and d2["kernel"] == "umma_tf32"
    u = d2["umma"]
    # CTA pairs on 256 x 256 tiles with a k chunk of 64: three stages of 64 KB per CTA, one copy per operand and stage
    assert (u["a_major"], u["b_major"], u["BN"], u["BK"], u["k_iters"], u["pair"], u["stages"]) == ("MN", "K", 256, 64, 16, True, 3)
    assert (u["a_slabs_per_copy"], u["b_slab_w"], u["b_slabs"]) == (4, 128, 2)
    assert u["tiles_m"] * u["tiles_n"] == 2048 and u["coalesced_store"] and u["smem_bytes"] <= 227 * 1024
    d4 = describe(engine, CONFIGS["cfg4"][0])
    assert d4["backend"] == "ttgt" and d4["kernel"] == "umma_tf32" and d4["umma"]["BK"] == 8
    assert d4["transpose_a"] == [3, 2, 1, 0] and d4["A"] == ["ab:2304", "f:8", "e:48"] and d4["umma"]["pair"] is False
    # cfg5: A's contracted rows lie 8 MB apart; the cost table sends A through one transpose to
    # [a | f,e | b] so that every TMA box is one contiguous piece, and keeps B where it lies
    d5 = describe(engine, CONFIGS["cfg5"][0])
    assert d5["backend"] == "ttgt" and d5["transpose_a"] == [0, 3, 1, 2] and d5["transpose_b"] is None
    assert d5["kernel"] == "umma_tf32" and d5["umma"]["k_iters"] == 256 and d5["umma"]["kc"] == "f"
    assert d5["umma"]["pair"] is True and d5["umma"]["BK"] == 64 and d5["umma"]["b_slabs_per_copy"] == 4
    d3 = describe(engine, CONFIGS["cfg3"][0])   # TMA-fed FP64 kernel: one 128-byte row of 16 doubles per box row
    assert d3["backend"] == "direct" and d3["kernel"] == "dmma_f64_tma"
    assert (d3["umma"]["BN"], d3["umma"]["BK"], d3["umma"]["stages"], d3["umma"]["k_iters"]) == (64, 16, 8, 3)
    assert d3["umma"]["coalesced_store"] and d3["umma"]["smem_bytes"] <= 227 * 1024


def test_fp64_kernel_choice_follows_the_cost_table(engine, monkeypatch):
    F64 = 1
    # A's stride-1 mode is not C's: where C's stride-1 mode lies behind the contracted mode in A and its extent is a
    # multiple of 8, a tile takes 8 of its indices x 16 elements of A's stride-1 mode and stores across slabs
    c31 = Contraction("abcdef", "dega", "gfbc", dict(a=24, b=16, c=16, d=24, e=16, f=16, g=24), F64)
    d = describe(engine, c31)
    assert d["backend"] == "direct" and d["kernel"] == "dmma_f64_tma" and d["umma"]["store_across_slabs"]
    assert d["umma"]["a_slabs_per_copy"] == 8 and not d["umma"]["coalesced_store"]
    c1 = Contraction("abc", "bda", "dc", dict(a=312, b=312, c=24, d=312), F64)
    d = describe(engine, c1)
    assert d["backend"] == "direct" and d["kernel"] == "dmma_f64_tma" and d["umma"]["store_across_slabs"]
    # ... where it cannot (extent 30 is no multiple of 8), rows along A's stride-1 mode would be stored element by
    # element, and one transpose of A is cheaper
    c31r = Contraction("abcdef", "dega", "gfbc", dict(a=30, b=16, c=16, d=24, e=16, f=16, g=24), F64)
    d = describe(engine, c31r)
    assert d["backend"] == "ttgt" and d["kernel"] == "dmma_f64_tma" and d["umma"]["coalesced_store"] and not d["umma"]["store_across_slabs"]
    # operands that are K-major on different contracted modes cannot be described to TMA where they lie
    c28 = Contraction("abcd", "eafb", "fdec", dict(a=72, b=72, c=72, d=72, e=72, f=72), F64)
    d = describe(engine, c28)
    assert d["backend"] == "ttgt" and d["kernel"] == "dmma_f64_tma"
    monkeypatch.setenv("TCONT_KERNEL", "gather")
    assert describe(engine, c28, 1)["kernel"] == "dmma_f64"
    monkeypatch.setenv("TCONT_KERNEL", "simt")
    assert describe(engine, c28, 1)["kernel"] == "simt"
    monkeypatch.delenv("TCONT_KERNEL")
    # tiny problems stay on the CUDA-core tiles
    assert describe(engine, CONFIGS["cfg1"][0])["kernel"] in ("simt", "dmma_f64_tma")


def test_fp64_row_widths_and_split_k(engine, monkeypatch):
    F64 = 1
    # extents of 72: slabs of 8 doubles (9 x 8) instead of 16 (5 x 16, 11 % padding) for the MN-major A,
    # 8 rows per slab for the K-major B
    d = describe(engine, Contraction("abcd", "aebf", "fdec", dict(a=72, b=72, c=72, d=72, e=72, f=72), F64), 1)
    u = d["umma"]
    assert d["kernel"] == "dmma_f64_tma" and (u["a_major"], u["b_major"], u["a_slab_w"], u["b_slab_w"]) == ("MN", "K", 8, 8)
    assert u["tiles_m"] == 41 and u["tiles_n"] == 81 and u["BK"] == 16        # ceil(5184 / 128), 5184 / 64
    # a contracted extent of 24: k chunks of 8 (64-byte rows for the K-major operand) instead of 2 x 16
    d = describe(engine, Contraction("abcdef", "degc", "gfab", dict(a=24, b=16, c=16, d=24, e=16, f=16, g=24), F64), 1)
    assert d["kernel"] == "dmma_f64_tma" and d["umma"]["BK"] == 8 and d["umma"]["k_iters"] == 3
    # narrow N: 128 x 32 tiles
    d = describe(engine, Contraction("abc", "dca", "bd", dict(a=312, b=24, c=296, d=312), F64), 1)
    assert d["kernel"] == "dmma_f64_tma" and d["umma"]["BN"] == 32
    # few tiles and a long contracted extent: split-K into a count of work units that fills whole waves
    # (296 units per wave for the FP64 kernel with its two consumer groups, 148 for tcgen05)
    for st, wave in ((F64, 296), (0, 148)):
        d = describe(engine, Contraction("ab", "acd", "dbc", dict(a=312, b=296, c=296, d=312), st), 1)
        u = d["umma"]
        units = u["tiles_m"] * u["tiles_n"] * u["k_splits"]
        assert u["k_splits"] > 1 and units / (-(-units // wave) * wave) >= 0.9, u
    # a little over one wave of tiles (162 on 148 SMs) is cut as well
    d = describe(engine, Contraction("abc", "adec", "ebd", dict(a=72, b=72, c=72, d=72, e=72), 0), 1)
    assert d["umma"]["tiles_m"] * d["umma"]["tiles_n"] == 162 and d["umma"]["k_splits"] >= 3
    monkeypatch.setenv("TCONT_SPLITK", "1")
    assert describe(engine, Contraction("ab", "acd", "dbc", dict(a=312, b=296, c=296, d=312), F64), 1)["umma"]["k_splits"] == 1


def test_every_reference_pattern_plans(engine):
    for fx in golden_fixtures():
        c = fixture_contraction(fx)
        for sel in (0, 1, 2):
            d = describe(engine, c, sel)
            assert d["Mtot"] * d["Ntot"] == c.size(c.modeC)
            assert d["Mtot"] * d["Ktot"] == c.size(c.modeB if d["swapped"] else c.modeA)


def test_plan_is_deterministic(engine):
    c = CONFIGS["cfg4"][0]
    assert describe(engine, c) == describe(engine, c)


def test_error_conventions(engine):
    E = engine.TCEquation
    with pytest.raises(ValueError, match="Missing extent for mode: d"):     # std::invalid_argument, src/tcont.cpp:44
        engine.plan(E("abc", "adc", "db", dict(a=2, b=2, c=2)))
    with pytest.raises(ValueError):
        engine.plan(E("ab", "ak", "kb", dict(a=2, b=0, k=2)))
    with pytest.raises(NotImplementedError, match="batch"):
        engine.plan(E("abn", "akn", "kbn", dict(a=2, b=2, k=2, n=2)))
    with pytest.raises(NotImplementedError):
        engine.plan(E("ab", "akx", "kb", dict(a=2, b=2, k=2, x=2)))
    with pytest.raises(ValueError):
        engine.launch(None)
    with pytest.raises(ValueError, match="ExecutionPlan is empty"):
        engine.prepare(None)


def test_flop_count_is_the_reference_formula(engine):
    c = CONFIGS["cfg2"][0]
    p = engine.plan(to_equation(engine, c))
    assert p.flops == pytest.approx(2.0 * 65536 * 1024 * 1024)
    assert engine.compute_gflops(p.equation, 1.0) == pytest.approx(p.flops / 1e6)
    assert engine.compute_gflops(p.equation, 0.0) == 0.0


def test_random_descriptors_plan_consistently(engine):
    """300 random descriptors (1-3 modes per group, ragged extents, random orders, both precisions, every backend
    selection): the planner accepts each one and its GEMM view multiplies out to the descriptor's extents."""
    import numpy as np

    from cases import random_contraction
    rng = np.random.default_rng(2024)
    for i in range(300):
        c = random_contraction(rng, int(rng.integers(0, 2)))
        sel = int(rng.integers(0, 3))
        d = engine.plan(to_equation(engine, c, sel)).describe()
        assert d["Mtot"] * d["Ntot"] == c.size(c.modeC), (i, c)
        assert d["Mtot"] * d["Ktot"] in (c.size(c.modeA), c.size(c.modeB)), (i, c)
        assert d["backend"] in ("direct", "ttgt") and d["kernel"] in ("simt", "umma_tf32", "dmma_f64", "dmma_f64_tma")
        if sel == 1:
            assert d["backend"] == "direct" and d["transpose_a"] is None and d["transpose_b"] is None
        u = d["umma"]
        if d["kernel"] in ("umma_tf32", "dmma_f64_tma"):
            assert u["eligible"] and u["smem_bytes"] <= 227 * 1024
            assert u["tiles_m"] * u["BM"] >= d["Mtot"] and u["tiles_n"] * u["BN"] >= d["Ntot"]
            assert u["k_iters"] * u["BK"] >= d["Ktot"] and 1 <= u["k_splits"] <= u["k_iters"]


def test_planning_is_reentrant(engine):
    """plan() from eight threads at once (ctypes releases the GIL) gives what a single thread gets, and an error raised
    in one thread does not leak into another's tcontb_last_error (it is thread-local)."""
    import threading

    import numpy as np

    from cases import random_contraction
    rng = np.random.default_rng(5)
    eqs = [to_equation(engine, random_contraction(rng, i % 2), i % 3) for i in range(40)]
    want = [engine.plan(e).describe() for e in eqs]
    bad = engine.TCEquation("ab", "ak", "kb", dict(a=4, b=4))   # extent of k missing
    failures = []

    def worker(tid):
        try:
            for rep in range(5):
                for i, e in enumerate(eqs):
                    if (i + tid) % 7 == 0:
                        with pytest.raises(ValueError, match="k"):
                            engine.plan(bad)
                    if engine.plan(e).describe() != want[i]:
                        failures.append((tid, rep, i))
        except Exception as ex:  # noqa: BLE001
            failures.append((tid, repr(ex)))

    threads = [threading.Thread(target=worker, args=(t,)) for t in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[:3]


def test_sub_tensor_views_take_their_strides_from_the_parent(engine):
    """tcontb_plan_create_strided: modes fuse only where the view leaves no gap between them; a view whose strides
    are not multiples of 16 bytes cannot be staged by TMA; parents must cover their views."""
    c = CONFIGS["cfg3"][0]
    eq = to_equation(engine, c)
    dense = engine.plan(eq).describe()
    assert dense["views"] is False and dense["A"] == ["a:48", "e:48", "ij:576"]
    # A is a view with a gap after i (parent 26 wide in i): i and j no longer fuse anywhere; b and c still do
    d = engine.plan_views(eq, None, [48, 48, 26, 24], None).describe()
    assert d["views"] is True and d["A"] == ["a:48", "e:48", "i:24", "j:24"] and d["B"][0] == "bc:2304"
    assert d["C"] == ["a:48", "bc:2304", "i:24", "j:24", "k:24"]
    assert d["kernel"] == "dmma_f64_tma"                      # strides stay multiples of 16 bytes
    # a parent that is one element wider in the stride-1 mode: 8-byte-aligned rows only, so no TMA
    d = engine.plan_views(eq, None, [49, 48, 24, 24], None).describe()
    assert d["kernel"] in ("dmma_f64", "simt") and "16 bytes" in d["umma"]["why_not"]
    # C as a view: no split-K (there is no workspace laid out like C)
    lk = Contraction("ab", "acd", "dbc", dict(a=312, b=296, c=296, d=312), 1)
    assert engine.plan(to_equation(engine, lk, 1)).describe()["umma"]["k_splits"] > 1
    assert engine.plan_views(to_equation(engine, lk, 1), [320, 296], None, None).describe()["umma"]["k_splits"] == 1
    with pytest.raises(ValueError):
        engine.plan_views(eq, None, [40, 48, 24, 24], None)   # parent smaller than the view


def test_tcgen05_kernel_forms(engine, monkeypatch):
    """Which form of the tcgen05 kernel a plan asks for: CTA pairs with stages of 64 k and one producer warp for
    large problems; one CTA per tile with two producer warps (and an even number of stages) otherwise; k chunks of
    24 where 32 would pad an MN-major contracted mode by a quarter."""
    from oracle_lib import F32
    pair = describe(engine, CONFIGS["cfg2"][0])["umma"]
    assert pair["pair"] is True and pair["BK"] == 64 and pair["producers"] == 1 and pair["stages"] == 3
    # the 72-extent 4-D family (reference case 22): both operands MN-major, chunked mode of extent 72
    c22 = Contraction("abcd", "aecf", "bfde", dict(a=72, b=72, c=72, d=72, e=72, f=72), F32)
    one = describe(engine, c22, 1)["umma"]
    assert one["pair"] is False and one["producers"] == 2 and one["stages"] % 2 == 0 and one["BK"] == 24
    monkeypatch.setenv("TCONT_UMMA_NO_BK24", "1")
    assert describe(engine, c22, 1)["umma"]["BK"] == 32
    monkeypatch.delenv("TCONT_UMMA_NO_BK24")
    # one k iteration per tile (the low-K configuration after its transposes): a second producer has nothing to do
    low_k = describe(engine, CONFIGS["cfg4"][0])["umma"]
    assert low_k["pair"] is False and low_k["producers"] == 1
    monkeypatch.setenv("TCONT_UMMA_PRODUCERS", "1")
    assert describe(engine, c22, 1)["umma"]["producers"] == 1


@pytest.mark.parametrize("scalar", [F32, F64])
@pytest.mark.parametrize("cluster", ["16", "3"])
def test_gather_plan_without_a_candidate_covers_all_rows(engine, monkeypatch, scalar, cluster):
    """A forced cluster that the contracted extent is too short for (or that does not exist) falls back to one CTA per tile."""
    monkeypatch.setenv("TCONT_KERNEL", "gather" if scalar == F64 else "simt")
    monkeypatch.setenv("TCONT_GATHER_CLUSTER", cluster)
    g = describe(engine, Contraction("ab", "ak", "kb", dict(a=65, b=33, k=17), scalar), 1)["gather"]
    assert g["cluster"] == 1 and g["rows"] >= 65


def test_gather_plan_with_unusable_rates_covers_all_rows(engine, monkeypatch, tmp_path):
    table = tmp_path / "table.txt"
    table.write_text("".join(f"gather_f64_tflops_{t} 0\n" for t in range(3)))
    monkeypatch.setenv("TCONT_COST_TABLE", str(table))
    monkeypatch.setenv("TCONT_KERNEL", "gather")
    g = describe(engine, Contraction("ab", "ak", "kb", dict(a=65, b=33, k=17), F64), 1)["gather"]
    assert g["cluster"] == 1 and g["rows"] >= 65


@pytest.mark.parametrize("modes,ext", [
    (("abcde", "efba", "cfd"), dict(a=16, b=16, c=8, d=16, e=16, f=8)),     # rows that the TMA-fed kernel would take across slabs
    (("abcde", "efba", "cfd"), dict(a=16, b=24, c=12, d=20, e=18, f=4)),
])
def test_small_fp64_is_gathered(engine, modes, ext):
    d = describe(engine, Contraction(*modes, ext, F64))
    assert d["kernel"] in ("simt", "dmma_f64") and d["backend"] == "direct"


# 15 x 19 tiles of a permutation: moving the tensor takes longer than contracting it where it lies
@pytest.mark.parametrize("modes,ext,scalar", [
    (("abcde", "efbad", "cf"), dict(a=19, b=13, c=29, d=15, e=15, f=223), F32),
    (("abcde", "efcad", "bf"), dict(a=13, b=9, c=13, d=13, e=8, f=161), F32),
    (("abcde", "efbad", "cf"), dict(a=15, b=13, c=9, d=17, e=19, f=61), F64),
])
def test_short_permutation_tiles_count(engine, modes, ext, scalar):
    assert describe(engine, Contraction(*modes, ext, scalar))["backend"] == "direct"


def test_long_permutation_tiles_still_pay(engine):
    assert describe(engine, Contraction("abcde", "efba", "cfd", dict(a=31, b=47, c=43, d=43, e=53, f=7), F32))["backend"] == "ttgt"


@pytest.mark.parametrize("modes,ext", [
    (("ab", "cad", "dcb"), dict(a=168, b=192, c=64, d=64)),
    (("abcd", "eafb", "fdec"), dict(a=24, b=24, c=16, d=32, e=24, f=24)),
])
def test_sectors_fetched_for_one_element_count(engine, modes, ext):
    """Operands that are K-major on different modes: a transpose and the TMA-fed kernel instead of scattered gathers."""
    d = describe(engine, Contraction(*modes, ext, F64))
    assert (d["backend"], d["kernel"]) == ("ttgt", "dmma_f64_tma")


@pytest.mark.parametrize("modes,ext", [
    (("abcd", "deca", "be"), dict(a=35, b=35, c=27, d=33, e=311)),
    (("abcde", "ecbfa", "fd"), dict(a=23, b=21, c=19, d=42, e=21, f=91)),
])
def test_scattered_rows_are_not_fetched_twice(engine, modes, ext):
    """33 to 64 columns: not in 32-column tiles where every element of A comes in a sector of its own."""
    d = describe(engine, Contraction(*modes, ext, F64), 1)
    assert d["kernel"] in ("simt", "dmma_f64") and (d["gather"]["t0"] > 0 or d["gather"]["tile"] != 1)


def test_float32_tiles_across_stride_1_modes_are_taken_where_they_are_faster(engine):
    """Measured in both forms (microseconds across / behind a copy of A or where A lies)."""
    def across(eq, extents):
        C, A, B = eq.split()
        d = describe(engine, Contraction(C, A, B, dict(zip(sorted(set(C + A + B)), extents)), F32))
        assert d["umma"]["in_use"] == ("across" not in d)
        return "across" in d
    assert across("abcde efbad cf", (48, 32, 24, 32, 48, 32))             # 107 / 311
    assert across("abcd dbea ec", (72, 72, 48, 72, 72))                   # 39.5 / 100
    assert across("abcd deca be", (96, 64, 96, 96, 32))                   # 65.9 / 139
    assert across("abcdef gfbc dega", (16, 16, 16, 24, 24, 16, 24))       # 27.2 / 37.5
    assert across("abcde efba cfd", (32, 52, 36, 60, 32, 8))              # 87.0 / 91.5
    assert across("abc bda dc", (212, 256, 216, 4))                       # 16.8 / 29.9
    # rows that end in half of a chunk, that end inside a sector, A's rows off their lines or sectors, estimates that are level
    assert not across("abcdef dfga gebc", (24, 16, 16, 24, 16, 16, 24))   # 44.3 / 39.2
    assert not across("abcde efba cfd", (20, 20, 20, 40, 20, 8))          # 18.3 / 16.4
    assert not across("abcde efba cfd", (40, 28, 32, 16, 24, 72))         # 33.5 / 23.9
    assert not across("abcdef dfga gebc", (16, 20, 12, 20, 28, 16, 48))   # 71.7 / 41.9
    assert not across("abcde efba cfd", (40, 40, 32, 40, 64, 8))          # 104 / 94.3


@pytest.mark.parametrize("eq,extents,piece", [
    ("ab ak kb", (1540, 56, 24), 4), ("ab ak bk", (1540, 40, 24), 4), ("ab ak bk", (1030, 150, 40), 2), ("ab ka kb", (1029, 149, 40), 1),
    ("abcd dbea ec", (24, 9, 60, 54, 40), 4), ("acb abk kc", (12, 60, 128, 24), 4), ("acb abk kc", (6, 50, 128, 24), 2),
])
def test_fp64_pieces_follow_the_strides_of_c(engine, monkeypatch, eq, extents, piece):
    """How many neighbouring elements of C the TMA-fed FP64 kernel may store at a time."""
    monkeypatch.setenv("TCONT_KERNEL", "tma")
    C, A, B = eq.split()
    d = describe(engine, Contraction(C, A, B, dict(zip(sorted(set(C + A + B)), extents)), F64), 1)
    assert d["kernel"] == "dmma_f64_tma" and d["umma"]["piece"] == piece, d["umma"]


def test_fp64_narrow_tiles(engine, monkeypatch):
    """128 x 32 tiles for short contracted extents, unless they compute more columns, A comes in slabs of 8 rows, or k is cut."""
    F64 = 1
    narrow = lambda c: "narrow" in describe(engine, c, 1)
    rows = lambda n, k: Contraction("ab", "ak", "kb", dict(a=9216, b=n, k=k), F64)
    across = lambda k: Contraction("abcdef", "dega", "gfbc", dict(a=24, b=16, c=16, d=24, e=16, f=16, g=k), F64)
    assert narrow(rows(4096, 16)) and narrow(rows(4096, 96)) and not narrow(rows(4096, 112))
    assert narrow(rows(4096, 24)) and not narrow(rows(4096, 40))      # k chunks of 8
    assert narrow(across(24)) and narrow(across(256)) and not narrow(across(272))
    assert not narrow(rows(40, 64)) and not narrow(rows(24, 64))      # three column fragments a warp; 32 columns anyway
    assert not narrow(Contraction("abc", "akb", "kc", dict(a=24, b=400, c=4096, k=64), F64))
    d = describe(engine, rows(4096, 16), 1)
    assert not d["umma"]["in_use"] and d["narrow"]["BN"] == 32 and d["narrow"]["stages"] % 3 == 0
    monkeypatch.setenv("TCONT_DMMA_BN", "64")
    assert not narrow(rows(4096, 16)) and describe(engine, rows(4096, 16), 1)["umma"]["in_use"]


def test_fp64_ranges_where_slabs_and_k_chunks_of_8_meet(engine):
    """These stay on the tiles and ranges planned without narrow ones, whatever their size; with k chunks of 16 large ones go narrow too."""
    F64 = 1
    plan = lambda C, A, B, *extents: describe(engine, Contraction(C, A, B, dict(zip("abcdef", extents)), F64))
    for d in (plan("abcd", "aecf", "fbed", 24, 56, 40, 24, 16, 24), plan("abcd", "aebf", "fdec", 24, 32, 40, 40, 32, 40), plan("abcd", "aebf", "dfce", 40, 8, 8, 8, 64, 24)):
        assert d["kernel"] == "dmma_f64_tma" and "narrow" not in d and (d["umma"]["BK"], d["umma"]["a_slab_w"]) == (8, 8) and d["umma"]["k_splits"] > 1
    d = plan("abcd", "aebf", "dfce", 72, 16, 72, 64, 40, 64)
    assert (d["umma"]["BK"], d["umma"]["a_slab_w"], d["umma"]["k_splits"]) == (16, 8, 3) and d["narrow"]["k_splits"] == 1


def test_fp64_consumer_groups(engine, monkeypatch):
    """Two consumer groups on 128 x 32 tiles: where three would not spare a round of them, for pieces of 8 or 16 bytes, and for one or two
    k chunks of 16 along C, or across slabs into one column of a C of more than 250 MB; three where old values are read in wider pieces, across slabs, and where A's slabs and k chunks of 8 meet."""
    F64 = 1

    def groups(C, A, B, **ext):
        d = describe(engine, Contraction(C, A, B, ext, F64), 1)
        u = d.get("narrow", d["umma"])
        assert d["kernel"] == "dmma_f64_tma" and d["umma"]["in_use"] == ("narrow" not in d)
        return u["BN"], *u["groups"]
    monkeypatch.setenv("TCONT_KERNEL", "tma")
    for tiles, rounds in ((1, 2), (2, 2), (3, 3), (4, 2), (5, 3)):
        assert groups("ab", "ak", "kb", a=128 * 148 * tiles, b=32, k=96) == (32, rounds, rounds), tiles
    assert groups("ab", "ak", "kb", a=9216, b=4096, k=32) == (32, 2, 3)
    assert groups("ab", "ak", "kb", a=9216, b=4096, k=48) == (32, 3, 3)
    assert groups("ab", "ak", "kb", a=9216, b=4096, k=24) == (32, 3, 3)            # k chunks of 8
    assert groups("ab", "ka", "kb", a=9217, b=4096, k=24) == (32, 2, 2)            # columns on odd multiples of 8 bytes
    assert groups("ab", "ka", "kb", a=9218, b=4096, k=24) == (32, 2, 3)            # of 16 bytes
    assert groups("abcd", "dbka", "kc", a=24, b=42, c=1024, d=32, k=16) == (32, 3, 3)
    assert groups("abc", "akb", "kc", a=24, b=740, c=32, k=24) == (32, 3, 3) and groups("abc", "akb", "kc", a=24, b=740, c=32, k=48) == (32, 2, 2)
    assert groups("ab", "ak", "kb", a=9216, b=24, k=96) == (32, 3, 3)              # three column fragments a warp
    assert groups("ab", "ak", "kb", a=9216, b=4096, k=200) == (64, 2, 2)
    long = dict(a=48, b=32, c=24, d=32, e=48)                                      # across slabs, C of 453 MB
    for k, plain in ((16, 2), (32, 2), (24, 3), (48, 3)):
        assert groups("abcde", "ekbad", "ck", k=k, **dict(long, c=28, a=40)) == (32, plain, 3), k
    assert groups("abcde", "ekbad", "ck", k=32, **dict(long, b=16)) == (32, 3, 3)  # of 226 MB
    assert groups("abcde", "ekbad", "ck", k=32, **dict(long, c=48)) == (32, 3, 3)  # two columns of tiles
    monkeypatch.setenv("TCONT_DMMA_GROUPS", "3")
    assert groups("ab", "ak", "kb", a=9216, b=4096, k=32) == (32, 3, 3)


def test_fp64_slim_across_slabs(engine):
    """Three column fragments a warp: not across slabs where a C of more than 150 MB is stored after one, two or three k chunks of 16."""
    F64 = 1

    def slim(**ext):
        d = describe(engine, Contraction("abcd", "dbka", "kc", dict(dict(a=48, b=96, c=24, d=192), **ext), F64), 1)
        u = d.get("narrow", d["umma"])
        assert d["kernel"] == "dmma_f64_tma" and d["umma"]["store_across_slabs"] and d["umma"]["in_use"] == ("narrow" not in d)
        if "narrow" not in d:
            assert u["slim_reads"] == (u["slim"] or ext["k"] == 48)                # accumulating launches keep it with three k chunks
        return u["BN"], u["slim"], u["groups"][0]
    for k in (16, 24, 32, 40, 48, 64):
        assert slim(k=k) == (32, k not in (32, 48), 3), k                          # 170 MB
        assert slim(k=k, b=64) == (32, True, 3), k                                 # 113 MB
    assert slim(k=32, b=192) == (32, False, 2) and slim(k=48, b=192) == (32, False, 3)
    assert slim(k=48, d=24, b=800) == (32, True, 3)                                # a fourth of the rows of its tiles is padding
    assert slim(k=16, c=48) == (32, False, 3) and slim(k=16, c=48, b=32) == (64, True, 2)
    assert slim(k=24, c=48) == (64, True, 2) and slim(k=32, c=48) == (64, True, 2)


def test_fp64_wide_tiles_where_old_values_are_read(engine, monkeypatch):
    """Rows along C, a C of more than 150 MB and more than 48 k: accumulating launches on 128 x 64 tiles, plain ones on narrow ones."""
    F64 = 1

    def wide(C, A, B, **ext):
        d = describe(engine, Contraction(C, A, B, ext, F64), 1)
        assert "narrow" in d and d["kernel"] == "dmma_f64_tma"
        return d["narrow"]["wide_reads"]
    assert wide("ab", "ak", "kb", a=18432, b=1024, k=64) and not wide("ab", "ak", "kb", a=18304, b=1024, k=64)
    assert wide("ab", "ka", "bk", a=39040, b=1024, k=56) and not wide("ab", "ka", "bk", a=39040, b=1024, k=48)
    assert not wide("abcd", "dbka", "kc", a=24, b=64, c=512, d=32, k=96)
    monkeypatch.setenv("TCONT_DMMA_BN", "32")
    assert not wide("ab", "ak", "kb", a=18432, b=1024, k=64)


def test_fp64_ranges_on_narrow_tiles(engine, monkeypatch):
    """Few tiles: ranges of k on narrow tiles in the place of ranges on wide ones, and of the gather kernel above 13.5 us."""
    F64 = 1
    small = Contraction("abcd", "aebf", "fdec", dict(a=24, b=24, c=24, d=24, e=16, f=16), F64)
    d = describe(engine, small)
    assert d["kernel"] == "dmma_f64_tma" and d["narrow"]["k_splits"] > 1 and not d["umma"]["in_use"]
    monkeypatch.setenv("TCONT_KERNEL", "gather")
    assert "narrow" not in describe(engine, small)
    monkeypatch.delenv("TCONT_KERNEL")
    smaller = Contraction("ab", "ak", "kb", dict(a=128, b=104, k=496), F64)
    assert describe(engine, smaller)["kernel"] == "simt" and "narrow" not in describe(engine, smaller)
    # more than 49 152 k on the gather kernel, operands that TMA could stage: one chain of FMAs
    longer = describe(engine, Contraction("abcdef", "degb", "gfac", dict(a=4, b=16, c=12, d=24, e=16, f=12, g=62714), F64), 1)
    assert longer["kernel"] != "dmma_f64_tma" and longer["umma"]["eligible"] and "narrow" not in longer and longer["gather"]["cluster"] == 1
    long_on_tma = describe(engine, Contraction("ab", "ak", "kb", dict(a=64, b=64, k=60000), F64))
    assert long_on_tma["kernel"] == "dmma_f64_tma" and long_on_tma["narrow"]["k_splits"] > 1 and long_on_tma["narrow"]["instead_of"] == "dmma_f64_tma"
    many = describe(engine, Contraction("abcd", "aecf", "bfde", dict(a=32, b=32, c=32, d=40, e=16, f=24), F64))
    assert many["umma"]["k_splits"] == 3 and many["narrow"]["k_splits"] == 2
    monkeypatch.setenv("TCONT_SPLITK", "3")
    assert "narrow" not in describe(engine, Contraction("abcd", "aecf", "bfde", dict(a=32, b=32, c=32, d=40, e=16, f=24), F64))


@pytest.mark.parametrize("tile,cluster,a,k,form", [(3, 1, 3201, 159, "plain"), (3, 1, 3201, 160, "wide"), (3, 2, 1401, 191, "plain"), (3, 2, 1401, 192, "wide"),
                                                   (3, 4, 1801, 383, "plain"), (3, 4, 1801, 384, "wide"), (3, 8, 701, 1535, "plain"), (3, 8, 701, 1536, "wide"),
                                                   (3, 4, 700, 384, "plain"), (0, 1, 323, 47, "short"), (0, 1, 323, 48, "plain"), (0, 2, 323, 49, "plain")])
def test_forms_of_float32_tiles(engine, monkeypatch, tile, cluster, a, k, form):
    """Four wide warps from a number of k per block on and with more blocks than SMs; full lines for short ranges of k."""
    monkeypatch.setenv("TCONT_KERNEL", "simt")
    monkeypatch.setenv("TCONT_GATHER_TILE", str(tile))
    monkeypatch.setenv("TCONT_GATHER_CLUSTER", str(cluster))
    monkeypatch.setenv("TCONT_GATHER_FLAT", "0")
    g = describe(engine, Contraction("ab", "ka", "bk", dict(a=a, b=a - 1, k=k), F32), 1)["gather"]
    assert (g["tile"], g["cluster"], g["form"]) == (tile, cluster, form), g


@pytest.mark.parametrize("b,k,tile,flat", [(57, 16, 0, True), (57, 17, 0, True), (57, 27, 0, True), (57, 28, 0, False), (57, 48, 0, False), (57, 49, 0, True),
                                           (77, 32, 3, True), (77, 33, 3, True), (77, 40, 3, True), (77, 41, 3, False), (77, 64, 3, False), (131, 33, None, True)])
def test_one_column_of_float32_tiles(engine, monkeypatch, b, k, tile, flat):
    """Many rows and one column of tiles: one tile a block where a tile has a few k tiles, the last of them well filled, persistent blocks
    otherwise; whatever the last one holds where A's rows lie scattered."""
    monkeypatch.setenv("TCONT_KERNEL", "simt")
    monkeypatch.setenv("TCONT_GATHER_TILE", str(3 if tile is None else tile))
    g = describe(engine, Contraction("ab", "ka", "bk", dict(a=400003, b=b, k=k), F32), 1)["gather"]
    assert g["cluster"] == 1 and g["flat"] == flat, g
    if tile is not None:
        g = describe(engine, Contraction("abcd", "dbea", "ec", dict(a=57, b=81, c=b, d=83, e=k), F32), 1)["gather"]
        assert g["cluster"] == 1 and g["flat"] == (k <= 16 or (tile == 0 and k > 48) or (tile == 3 and k <= 32)), g
