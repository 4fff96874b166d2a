"""Float32 on the CUDA cores in 128 x 128 tiles of four wide warps: gathers along rows and along k on either side, a last k tile that is
whole and one that is not, contracted ranges in one ring of offsets and past it, one range and clusters, rows that C and A hold in
different orders; and the sums of small clusters of 64 x 64 tiles.

Every output is a chain of K single-precision fused multiply-adds (the sums of a cluster's ranges a few more additions) and three roundings
of the scalars, each off by at most 2^-24 of its partial sum.
"""
import numpy as np
import pytest

from oracle_lib import F32, F64, Contraction
from test_scaled_epilogues_gpu import SCALARS, scaled_run

pytestmark = pytest.mark.gpu

# name -> (descriptor, cluster)
FORMS = {
    "rows_rows": ("ab", "ak", "bk", dict(a=1665, b=1537, k=417), 4),
    "rows_k_whole_k_tiles": ("ab", "ak", "kb", dict(a=1665, b=1537, k=448), 4),
    "k_rows_ring_of_offsets": ("ab", "ka", "bk", dict(a=3201, b=3203, k=259), 1),
    "k_k_offsets_kept": ("ab", "ka", "kb", dict(a=3201, b=3203, k=161), 1),
    "k_k_large_cluster": ("ab", "ka", "kb", dict(a=1153, b=1151, k=1605), 8),
    "two_contracted_modes": ("abcd", "aebf", "dfce", dict(a=41, b=41, c=39, d=41, e=21, f=23), 4),
    "stored_and_read_along_different_modes": ("abc", "bak", "kc", dict(a=49, b=33, c=1603, k=431), 4),
}


@pytest.mark.parametrize("name", list(FORMS))
def test_forms(engine, oracle, monkeypatch, name):
    monkeypatch.setenv("TCONT_KERNEL", "simt")
    C, A_, B_, ext, cluster = FORMS[name]
    c = Contraction(C, A_, B_, ext, F32)
    A, B = oracle.inputs(c, 31, -1.0, 1.0)
    C0 = np.random.default_rng(7).uniform(-4.0, 4.0, c.size(C)).astype(np.float32)
    desc, got = scaled_run(engine, c, A, B, C0, SCALARS)
    assert desc["kernel"] == "simt" and desc["gather"]["tile"] == 3 and not desc["gather"]["flat"], desc["gather"]
    assert desc["gather"]["cluster"] == cluster and desc["gather"]["form"] == "wide", desc["gather"]
    c64 = Contraction(C, A_, B_, ext, F64)
    product, scale = oracle.contract(c64, A.astype(np.float64), B.astype(np.float64)), oracle.contract(c64, np.abs(A).astype(np.float64), np.abs(B).astype(np.float64))
    k = int(np.prod([ext[m] for m in A_ if m not in C]))
    for (alpha, beta), out in zip(SCALARS, got):
        bound = (k + 20) * 2.0**-24 * (abs(alpha) * scale + abs(beta * C0))
        assert (np.abs(out - (alpha * product + beta * C0)) <= bound).all(), (name, alpha, beta)


@pytest.mark.parametrize("scalar_type,a,b,k,cluster", [(F32, 3001, 131, 131, 2), (F32, 331, 679, 245, 4), (F64, 1061, 679, 131, 2), (F64, 331, 679, 245, 4)])
def test_small_clusters_of_64_by_64_tiles(engine, oracle, monkeypatch, scalar_type, a, b, k, cluster):
    """Sums over 2 and 4 blocks four columns at a time, the last tile of a row with a few columns of its own."""
    monkeypatch.setenv("TCONT_KERNEL", "simt")
    c = Contraction("ab", "ka", "bk", dict(a=a, b=b, k=k), scalar_type)
    A, B = oracle.inputs(c, 37, -1.0, 1.0)
    C0 = np.random.default_rng(8).uniform(-4.0, 4.0, c.size("ab")).astype(A.dtype)
    desc, got = scaled_run(engine, c, A, B, C0, SCALARS)
    assert desc["gather"]["tile"] == 0 and desc["gather"]["cluster"] == cluster and desc["gather"]["form"] == "plain", desc["gather"]
    c64 = Contraction("ab", "ka", "bk", dict(a=a, b=b, k=k), F64)
    product, scale = oracle.contract(c64, A.astype(np.float64), B.astype(np.float64)), oracle.contract(c64, np.abs(A).astype(np.float64), np.abs(B).astype(np.float64))
    unit = 2.0**-24 if scalar_type == F32 else 2.0**-53
    for (alpha, beta), out in zip(SCALARS, got):
        bound = (k + 20) * unit * (abs(alpha) * scale + abs(beta * C0))
        assert (np.abs(out - (alpha * product + beta * C0)) <= bound).all(), (alpha, beta)


@pytest.mark.parametrize("cluster,A_,B_,k", [(1, "ka", "bk", 47), (1, "ka", "bk", 49), (1, "ak", "kb", 48), (2, "ak", "kb", 131), (2, "ka", "bk", 49)])
def test_64_by_64_tiles(engine, oracle, monkeypatch, cluster, A_, B_, k):
    """Warps of 32 x 32 with lanes 8 x 4, and one block's short range of k in warps of full lines."""
    monkeypatch.setenv("TCONT_KERNEL", "simt")
    monkeypatch.setenv("TCONT_GATHER_TILE", "0")
    monkeypatch.setenv("TCONT_GATHER_CLUSTER", str(cluster))
    monkeypatch.setenv("TCONT_GATHER_FLAT", "0")
    ext = dict(a=323, b=103, k=k)
    c, c64 = Contraction("ab", A_, B_, ext, F32), Contraction("ab", A_, B_, ext, F64)
    A, B = oracle.inputs(c, 41, -1.0, 1.0)
    C0 = np.random.default_rng(9).uniform(-4.0, 4.0, c.size("ab")).astype(np.float32)
    desc, got = scaled_run(engine, c, A, B, C0, SCALARS)
    g = desc["gather"]
    assert g["tile"] == 0 and g["cluster"] == cluster and not g["flat"] and g["form"] == ("short" if cluster == 1 and k < 48 else "plain"), g
    product, scale = oracle.contract(c64, A.astype(np.float64), B.astype(np.float64)), oracle.contract(c64, np.abs(A).astype(np.float64), np.abs(B).astype(np.float64))
    for (alpha, beta), out in zip(SCALARS, got):
        bound = (k + 20) * 2.0**-24 * (abs(alpha) * scale + abs(beta * C0))
        assert (np.abs(out - (alpha * product + beta * C0)) <= bound).all(), (alpha, beta)
