"""Tiles and chunks of the TMA-fed FP64 kernel at the sizes where they can go wrong, against the CPU oracle.

Every output is a chain of K fused multiply-adds (in ranges with split-K), each off by at most 2^-53 of its partial sum:
|err| <= (K + splits) 2^-53 sum|ab|.
"""
import numpy as np
import pytest

from cases import to_equation
from oracle_lib import F64, Contraction
from test_contraction_gpu import run_contraction

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
