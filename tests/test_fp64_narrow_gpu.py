"""FP64 contractions on 128 x 32 and 128 x 64 tiles: the two fragment layouts, rows of a tile along C, along k and across slabs, the ends of
tiles and slabs, contracted extents from one k chunk to more than fit the ring, old values of C staged and read in the epilogue.

Every output is a chain of K fused multiply-adds and three roundings of the scalars, each off by at most 2^-53 of its partial sum.
"""
import numpy as np
import pytest

from cases import to_equation
from oracle_lib import F64, Contraction
from test_scaled_epilogues_gpu import SCALARS, scaled_run

pytestmark = pytest.mark.gpu

# name -> (descriptor, tiles across slabs)
FORMS = {
    "mn_k": ("ab", "ak", "kb", dict(a=272, b=97), False),
    "mn_mn_odd_columns": ("abc", "ak", "bck", dict(a=146, b=34, c=3), False),
    "mn_8_wide_slabs": ("abc", "akb", "ck", dict(a=24, b=11, c=60), False),
    "k_mn_unaligned": ("ab", "ka", "bk", dict(a=131, b=62), False),
    "k_k_unaligned": ("ab", "ka", "kb", dict(a=259, b=61), False),
    "fused_rows": ("acb", "abk", "kc", dict(a=6, b=50, c=61), False),
    "across": ("abcd", "dbka", "kc", dict(a=24, b=3, c=60, d=34), True),
    "across_next_mode_a_row": ("abcd", "dkba", "ck", dict(a=8, b=9, c=62, d=48), True),
}


@pytest.mark.parametrize("name", list(FORMS))
@pytest.mark.parametrize("columns", ["32", "64"])
@pytest.mark.parametrize("k", [8, 24, 72, 136])
def test_forms(engine, oracle, monkeypatch, name, columns, k):
    monkeypatch.setenv("TCONT_KERNEL", "tma")
    monkeypatch.setenv("TCONT_SPLITK", "1")
    monkeypatch.setenv("TCONT_SCALE_PASSES", "1")
    monkeypatch.setenv("TCONT_DMMA_BN", columns)
    C, A_, B_, ext, across = FORMS[name]
    c = Contraction(C, A_, B_, dict(ext, k=k), F64)
    A, B = oracle.inputs(c, 23, -1.0, 1.0)
    C0 = np.random.default_rng(5).uniform(-4.0, 4.0, c.size(C))
    desc, got = scaled_run(engine, c, A, B, C0, SCALARS)
    assert desc["kernel"] == "dmma_f64_tma" and desc["umma"]["store_across_slabs"] == across
    assert desc["umma"]["BN"] == 64 and ("narrow" in desc) == (columns == "32") == (not desc["umma"]["in_use"])
    product, scale = oracle.contract(c, A, B), oracle.contract(c, np.abs(A), np.abs(B))
    for (alpha, beta), out in zip(SCALARS, got):
        bound = (k + 4) * 2.0**-53 * (abs(alpha) * scale + abs(beta * C0))
        assert (np.abs(out - (alpha * product + beta * C0)) <= bound).all(), (alpha, beta)


@pytest.mark.parametrize("name", list(FORMS) + ["several_tiles", "several_tiles_across"])
@pytest.mark.parametrize("groups", ["2", "3"])
@pytest.mark.parametrize("k", [8, 40, 104])
def test_two_and_three_groups(engine, oracle, monkeypatch, name, groups, k):
    """128 x 32 tiles in either number of consumer groups, whichever the planner would take."""
    monkeypatch.setenv("TCONT_KERNEL", "tma")
    monkeypatch.setenv("TCONT_SPLITK", "1")
    monkeypatch.setenv("TCONT_SCALE_PASSES", "1")
    monkeypatch.setenv("TCONT_DMMA_BN", "32")
    monkeypatch.setenv("TCONT_DMMA_GROUPS", groups)
    several = {"several_tiles": ("ab", "ak", "kb", dict(a=1930, b=2100), False), "several_tiles_across": ("abc", "cka", "kb", dict(a=24, b=1100, c=210), True)}
    C, A_, B_, ext, across = (FORMS | several)[name]
    c = Contraction(C, A_, B_, dict(ext, k=k), F64)
    A, B = oracle.inputs(c, 47, -1.0, 1.0)
    C0 = np.random.default_rng(11).uniform(-4.0, 4.0, c.size(C))
    desc, got = scaled_run(engine, c, A, B, C0, SCALARS)
    assert desc["narrow"]["groups"] == [int(groups)] * 2 and desc["umma"]["store_across_slabs"] == across
    product, scale = oracle.contract(c, A, B), oracle.contract(c, np.abs(A), np.abs(B))
    for (alpha, beta), out in zip(SCALARS, got):
        bound = (k + 4) * 2.0**-53 * (abs(alpha) * scale + abs(beta * C0))
        assert (np.abs(out - (alpha * product + beta * C0)) <= bound).all(), (alpha, beta)


@pytest.mark.parametrize("columns", ["32", "64"])
def test_several_tiles_a_group(engine, oracle, monkeypatch, columns):
    """Rings, tables and staged values come round: 9 to 18 tiles a block, all slabs whole but the last."""
    monkeypatch.setenv("TCONT_KERNEL", "tma")
    monkeypatch.setenv("TCONT_DMMA_BN", columns)
    monkeypatch.setenv("TCONT_SCALE_PASSES", "1")
    for C, A_, B_, ext in (("ab", "ak", "kb", dict(a=5130, b=2100, k=24)), ("abc", "cka", "kb", dict(a=24, b=2100, c=210, k=40))):
        c = Contraction(C, A_, B_, ext, F64)
        A, B = oracle.inputs(c, 29, -1.0, 1.0)
        C0 = np.random.default_rng(6).uniform(-4.0, 4.0, c.size(C))
        desc, got = scaled_run(engine, c, A, B, C0, [(1.0, 1.0), (1.0, 0.0)])
        assert ("narrow" in desc) == (columns == "32")
        product, scale = oracle.contract(c, A, B), oracle.contract(c, np.abs(A), np.abs(B))
        for beta, out in zip((1.0, 0.0), got):
            assert (np.abs(out - (product + beta * C0)) <= (ext["k"] + 4) * 2.0**-53 * (scale + abs(beta * C0))).all()


# what has few tiles -> (descriptor, kernel without narrow tiles)
RANGES = {
    "from_the_gather_kernel": ("abcd", "aebf", "fdec", dict(a=24, b=24, c=24, d=24, e=16, f=16), "simt"),
    "more_ranges_of_less": ("abcd", "aedf", "fbec", dict(a=8, b=16, c=16, d=16, e=56, f=56), "dmma_f64_tma"),
    "one_range": ("abcd", "deca", "be", dict(a=24, b=40, c=24, d=32, e=312), "dmma_f64_tma"),
}


@pytest.mark.parametrize("name", list(RANGES))
def test_ranges(engine, oracle, monkeypatch, name):
    C, A_, B_, ext, instead_of = RANGES[name]
    c = Contraction(C, A_, B_, ext, F64)
    A, B = oracle.inputs(c, 31, -1.0, 1.0)
    C0 = np.random.default_rng(7).uniform(-4.0, 4.0, c.size(C))
    desc, got = scaled_run(engine, c, A, B, C0, SCALARS, 0)
    ranges = desc["narrow"]["k_splits"]
    assert desc["kernel"] == "dmma_f64_tma" and (ranges == 1) == (name == "one_range") and desc["narrow"]["instead_of"] == instead_of
    assert desc["umma"]["k_splits"] != ranges
    product, scale = oracle.contract(c, A, B), oracle.contract(c, np.abs(A), np.abs(B))
    k = int(np.prod([ext[m] for m in ext if m not in C]))
    for (alpha, beta), out in zip(SCALARS, got):   # (and a rounding for each partial sum)
        bound = (k + ranges + 4) * 2.0**-53 * (abs(alpha) * scale + abs(beta * C0))
        assert (np.abs(out - (alpha * product + beta * C0)) <= bound).all(), (alpha, beta)


def test_no_room_for_ranges(engine, oracle, monkeypatch):
    """The gather kernel runs where the partial sums find no room: one kernel a launch, no sum behind it."""
    import torch
    C, A_, B_, ext, _ = RANGES["from_the_gather_kernel"]
    c = Contraction(C, A_, B_, ext, F64)
    A, B = oracle.inputs(c, 31, -1.0, 1.0)
    from tcont_b200 import api
    plan = engine.plan(to_equation(engine, c, 0))
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    dC = torch.zeros(c.size(C), dtype=dA.dtype, device="cuda")

    def kernels():
        return api.prepare_on_device(plan, dA.data_ptr(), dB.data_ptr(), dC.data_ptr(), keep=(dA, dB, dC)).time_launches(1)[1]
    assert kernels() == 2   # the ranges and their sum
    monkeypatch.setenv("TCONT_TEST_NO_ROOM", "1000")
    assert kernels() == 1
    desc, got = scaled_run(engine, c, A, B, np.ones(c.size(C)), [(1.0, 1.0), (1.0, 0.0)], 0)
    assert desc["narrow"]["k_splits"] > 1 and desc["narrow"]["instead_of"] == RANGES["from_the_gather_kernel"][4]
    product, scale = oracle.contract(c, A, B), oracle.contract(c, np.abs(A), np.abs(B))
    for beta, out in zip((1.0, 0.0), got):
        assert (np.abs(out - (product + beta)) <= (256 + 8) * 2.0**-53 * (scale + beta)).all()


@pytest.mark.parametrize("columns", ["32", "64"])
@pytest.mark.parametrize("beta", [0.0, 1.0])
@pytest.mark.parametrize("skip", [2, 8, 17])
def test_bounded_wait_gives_up_cleanly(engine, oracle, monkeypatch, columns, beta, skip):
    """The first, second or fourth tile of every block and those behind it are never filled, and the waits for them are given up after 2 ms:
    the run's status says so, what is stored of C is right, nothing outside it is written, and the next run is right."""
    import torch
    from tcont_b200 import api
    monkeypatch.setenv("TCONT_KERNEL", "tma")
    monkeypatch.setenv("TCONT_DMMA_BN", columns)
    k = 72
    c = Contraction("ab", "ak", "kb", dict(a=5130, b=700, k=k), F64)
    A, B = oracle.inputs(c, 43, -1.0, 1.0)
    C0 = np.random.default_rng(10).uniform(-4.0, 4.0, c.size("ab"))
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    guarded = torch.full((C0.size + 64,), 7.0, dtype=torch.float64, device="cuda")
    plan = engine.plan(to_equation(engine, c, 1))
    desc = plan.describe()
    assert desc["kernel"] == "dmma_f64_tma" and ("narrow" in desc) == (columns == "32") and desc["umma"]["k_iters"] == 5
    want = oracle.contract(c, A, B) + beta * C0
    bound = (k + 4) * 2.0**-53 * (oracle.contract(c, np.abs(A), np.abs(B)) + abs(beta * C0))

    def launched(**hooks):
        for name, value in hooks.items():
            monkeypatch.setenv(name, value)
        run = api.prepare_on_device(plan, dA.data_ptr(), dB.data_ptr(), guarded[32:].data_ptr(), keep=(dA, dB, guarded))
        for name in hooks:
            monkeypatch.delenv(name)
        run.set_scalars(1.0, beta)
        guarded[32:32 + C0.size].copy_(torch.from_numpy(C0))
        engine.launch(run)
        torch.cuda.synchronize()
        got = guarded.cpu().numpy()
        assert (got[:32] == 7.0).all() and (got[32 + C0.size:] == 7.0).all()
        return run.device_status(), got[32:32 + C0.size]
    status, got = launched(TCONT_TEST_WAIT_LIMIT_NS="2000000", TCONT_TEST_SKIP_STAGE=str(skip))
    right = np.abs(got - want) <= bound
    assert status == 1 and not right.all() and (right | (got == C0)).all()
    status, got = launched()
    assert status == 0 and (np.abs(got - want) <= bound).all()


@pytest.mark.parametrize("A_,B_", [("ak", "kb"), ("ka", "bk")])
def test_wide_tiles_where_old_values_are_read(engine, oracle, A_, B_):
    """A C of 152 MB, rows along C: one run takes narrow tiles for plain launches and 128 x 64 for accumulating ones, in any order."""
    c = Contraction("ab", A_, B_, dict(a=16400, b=1160, k=72), F64)
    A, B = oracle.inputs(c, 53, -1.0, 1.0)
    C0 = np.random.default_rng(12).uniform(-4.0, 4.0, c.size("ab"))
    scalars = [(1.0, 1.0), (1.0, 0.0), (0.3, -0.7), (-0.75, 0.0), (1.0, 1.0)]
    desc, got = scaled_run(engine, c, A, B, C0, scalars)
    assert desc["kernel"] == "dmma_f64_tma" and desc["narrow"]["wide_reads"]
    at = np.sort(np.random.default_rng(13).integers(0, C0.size, 20000))
    product, scale = oracle.contract_sampled(c, A, B, at), oracle.contract_sampled(c, np.abs(A), np.abs(B), at)
    for (alpha, beta), out in zip(scalars, got):
        bound = (72 + 4) * 2.0**-53 * (abs(alpha) * scale + abs(beta * C0[at]))
        assert (np.abs(out[at] - (alpha * product + beta * C0[at])) <= bound).all(), (alpha, beta)
    assert (got[0] == got[4]).all()


@pytest.mark.parametrize("extents,k,forms", [(dict(a=48, b=96, c=24, d=192), 48, (False, True)), (dict(a=40, b=132, c=22, d=288), 32, (False, False))])
def test_slim_where_old_values_are_read(engine, oracle, extents, k, forms):
    """Across slabs, C of 170 and 268 MB: three column fragments a warp in accumulating launches only, and two consumer groups in plain ones only."""
    c = Contraction("abcd", "dbka", "kc", dict(extents, k=k), F64)
    A, B = oracle.inputs(c, 59, -1.0, 1.0)
    C0 = np.random.default_rng(14).uniform(-4.0, 4.0, c.size("abcd"))
    scalars = [(1.0, 1.0), (1.0, 0.0), (0.3, -0.7), (-0.75, 0.0), (1.0, 1.0)]
    desc, got = scaled_run(engine, c, A, B, C0, scalars)
    u = desc["umma"]
    assert desc["kernel"] == "dmma_f64_tma" and u["in_use"] and (u["slim"], u["slim_reads"]) == forms
    assert u["groups"] == ([3, 3] if k == 48 else [2, 3])
    at = np.sort(np.random.default_rng(15).integers(0, C0.size, 20000))
    product, scale = oracle.contract_sampled(c, A, B, at), oracle.contract_sampled(c, np.abs(A), np.abs(B), at)
    for (alpha, beta), out in zip(scalars, got):
        bound = (k + 4) * 2.0**-53 * (abs(alpha) * scale + abs(beta * C0[at]))
        assert (np.abs(out[at] - (alpha * product + beta * C0[at])) <= bound).all(), (alpha, beta)
    assert (got[0] == got[4]).all()
