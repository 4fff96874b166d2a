"""C = alpha A B + beta C where the kernel that writes C applies the scalars, over the forms of the two TMA-fed epilogues.

C starts from values of its own, so that an old value taken from the wrong element shows.  FP64: every output is a chain of
K fused multiply-adds and three roundings of the scalars, each off by at most 2^-53 of its partial sum.  Float32: held to
the TF32-operand oracle like the overwriting kernel, plus the roundings of the scalars.
"""
import numpy as np
import pytest

from cases import to_equation
from oracle_lib import F32, F64, Contraction

pytestmark = pytest.mark.gpu

# name -> (descriptor, what the plan has to say): A and B along the rows (MN) or along k, tiles 64 or 32 columns wide, rows of
# a tile along C or across slabs, C's columns on odd multiples of 8 bytes (extents 131, 67), ragged tiles, several per block
FP64_FORMS = {
    "mn_mn_64": ("ab", "ak", "bk", dict(a=192, b=192, k=40), ("MN", "MN", 64, False)),
    "mn_k_64": ("ab", "ak", "kb", dict(a=130, b=190, k=24), ("MN", "K", 64, False)),
    "k_mn_64": ("ab", "ka", "bk", dict(a=131, b=120, k=40), ("K", "MN", 64, False)),
    "k_k_64": ("ab", "ka", "kb", dict(a=131, b=121, k=56), ("K", "K", 64, False)),
    "mn_mn_32": ("ab", "ak", "bk", dict(a=144, b=24, k=40), ("MN", "MN", 32, False)),
    "mn_k_32": ("ab", "ak", "kb", dict(a=130, b=21, k=24), ("MN", "K", 32, False)),
    "k_mn_32": ("ab", "ka", "bk", dict(a=131, b=24, k=40), ("K", "MN", 32, False)),
    "k_k_32": ("ab", "ka", "kb", dict(a=67, b=19, k=56), ("K", "K", 32, False)),
    "across_slabs_64": ("abcd", "dbea", "ec", dict(a=24, b=5, c=60, d=34, e=40), ("MN", "K", 64, True)),
    "across_slabs_32": ("abcd", "dbea", "ec", dict(a=16, b=3, c=24, d=20, e=24), ("MN", "K", 32, True)),
    "fused_rows": ("acb", "abk", "kc", dict(a=6, b=50, c=21, k=24), ("MN", "K", 32, False)),
    "many_tiles": ("ab", "ak", "bk", dict(a=1930, b=1930, k=24), ("MN", "MN", 64, False)),
}


def scaled_run(engine, c, A, B, C0, scalars, selection=1):
    import torch
    from tcont_b200 import api
    plan = engine.plan(to_equation(engine, c, selection))
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    dC = torch.empty(C0.size, dtype=dA.dtype, device="cuda")
    run = api.prepare_on_device(plan, dA.data_ptr(), dB.data_ptr(), dC.data_ptr(), keep=(dA, dB, dC))
    got = []
    for alpha, beta in scalars:
        dC.copy_(torch.from_numpy(C0))
        run.set_scalars(alpha, beta)
        engine.launch(run)
        torch.cuda.synchronize()
        got.append(dC.cpu().numpy())
    assert run.device_status() == 0
    return plan.describe(), got


SCALARS = [(1.0, 1.0), (-0.75, 0.0), (0.3, -0.7), (1.0, 0.0)]


@pytest.mark.parametrize("name", list(FP64_FORMS))
@pytest.mark.parametrize("passes", ["1", "2"])
def test_fp64(engine, oracle, monkeypatch, name, passes):
    monkeypatch.setenv("TCONT_KERNEL", "tma")
    monkeypatch.setenv("TCONT_SPLITK", "1")
    monkeypatch.setenv("TCONT_SCALE_PASSES", passes)
    C, A_, B_, ext, form = FP64_FORMS[name]
    c = Contraction(C, A_, B_, ext, F64)
    A, B = oracle.inputs(c, 17, -1.0, 1.0)
    C0 = np.random.default_rng(3).uniform(-4.0, 4.0, c.size(C))
    desc, got = scaled_run(engine, c, A, B, C0, SCALARS)
    u = desc["umma"]
    assert desc["kernel"] == "dmma_f64_tma" and (u["a_major"], u["b_major"], u["BN"], u["store_across_slabs"]) == form, u
    assert (u["a_fused"] > 0) == (name == "fused_rows")
    product, scale = oracle.contract(c, A, B), oracle.contract(c, np.abs(A), np.abs(B))
    k = ext.get("k", ext.get("e"))
    for (alpha, beta), out in zip(SCALARS, got):
        bound = (k + 4) * 2.0**-53 * (abs(alpha) * scale + abs(beta * C0))
        assert (np.abs(out - (alpha * product + beta * C0)) <= bound).all(), (alpha, beta)


# pairs and single CTAs, one producer and two, columns by chunk (wide slabs) and one by one (fused or narrow slabs)
FLOAT32_FORMS = {
    "pair": ("ab", "ka", "kb", dict(a=520, b=264, k=96), 1, {"TCONT_UMMA_PAIR": "1"}),
    "pair_two_producers": ("ab", "ka", "kb", dict(a=520, b=264, k=96), 1, {"TCONT_UMMA_PAIR": "1", "TCONT_UMMA_PRODUCERS": "2"}),
    "pair_wide": ("ab", "ka", "bk", dict(a=2568, b=2088, k=64), 1, {"TCONT_UMMA_PAIR": "1"}),
    "single_one_producer": ("ab", "ak", "kb", dict(a=200, b=136, k=64), 1, {"TCONT_UMMA_PAIR": "0", "TCONT_UMMA_PRODUCERS": "1"}),
    "single_two_producers": ("ab", "ak", "bk", dict(a=200, b=136, k=64), 1, {"TCONT_UMMA_PAIR": "0", "TCONT_UMMA_PRODUCERS": "2"}),
    "fused_rows_and_columns": ("acbd", "abk", "cdk", dict(a=40, b=24, c=36, d=28, k=64), 1, {"TCONT_UMMA_PAIR": "0"}),
    "fused_columns_pair": ("acbd", "abk", "cdk", dict(a=40, b=24, c=40, d=64, k=64), 1, {"TCONT_UMMA_PAIR": "1"}),
    "narrow_columns": ("acb", "abk", "kc", dict(a=64, b=9, c=20, k=64), 1, {}),
}


@pytest.mark.parametrize("name", list(FLOAT32_FORMS))
def test_float32(engine, oracle, monkeypatch, name):
    C, A_, B_, ext, selection, env = FLOAT32_FORMS[name]
    monkeypatch.setenv("TCONT_SPLITK", "1")
    for key, value in env.items():
        monkeypatch.setenv(key, value)
    c = Contraction(C, A_, B_, ext, F32)
    A, B = oracle.inputs(c, 19, -1.0, 1.0)
    C0 = np.random.default_rng(4).uniform(-4.0, 4.0, c.size(C)).astype(np.float32)
    desc, got = scaled_run(engine, c, A, B, C0, SCALARS, selection)
    u = desc["umma"]
    assert desc["kernel"] == "umma_tf32"
    assert u["pair"] == (env.get("TCONT_UMMA_PAIR") == "1") and u["producers"] == int(env.get("TCONT_UMMA_PRODUCERS", u["producers"])), u
    if name.startswith("fused"):
        assert u["b_fused"] == ext["c"]
    if name == "narrow_columns":
        assert u["b_slab_w"] < 32
    product, scale = oracle.contract(c, A, B, rounding=1), oracle.contract(c, np.abs(A), np.abs(B), rounding=1)
    for (alpha, beta), out in zip(SCALARS, got):
        want = alpha * product + beta * C0.astype(np.float64)
        bound = 2e-5 * abs(alpha) * scale + 4 * 2.0**-24 * (np.abs(alpha * product) + np.abs(beta * C0.astype(np.float64)))
        assert (np.abs(out - want) <= bound).all(), (alpha, beta)


def test_fp64_beyond_l2(engine, oracle, monkeypatch):
    """A C of more than 64 MB: rows across slabs with a k chunk of 16 take a second pass over C, and can be kept from it."""
    monkeypatch.setenv("TCONT_KERNEL", "tma")
    c = Contraction("abcd", "dbea", "ec", dict(a=40, b=16, c=56, d=250, e=16), F64)
    A, B = oracle.inputs(c, 23, -1.0, 1.0)
    C0 = np.random.default_rng(5).uniform(-4.0, 4.0, c.size("abcd"))
    assert C0.nbytes > 64 << 20
    product, scale = oracle.contract(c, A, B), oracle.contract(c, np.abs(A), np.abs(B))
    for passes in (None, "1"):
        if passes:
            monkeypatch.setenv("TCONT_SCALE_PASSES", passes)
        desc, got = scaled_run(engine, c, A, B, C0, [(0.3, -0.7)])
        assert desc["umma"]["store_across_slabs"] and desc["umma"]["BK"] == 16
        bound = 20 * 2.0**-53 * (0.3 * scale + abs(0.7 * C0))
        assert (np.abs(got[0] - (0.3 * product - 0.7 * C0)) <= bound).all()
