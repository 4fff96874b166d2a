"""Which Float32 contractions run in IEEE single precision: a faster gather kernel, operand-level fusion of rows or another
transposed layout must not take one of them to TF32 (planner only, no GPU)."""
import os

import pytest

from cases import to_equation
from float32_line import descriptors
from oracle_lib import F32, Contraction

IEEE = {
    # K-major on two different modes, direct; one transpose and the tensor cores would now look cheaper than the gather kernel
    "two_k_majors": (("ab", "cad", "dcb", dict(a=224, b=224, c=16, d=256)), 0),
    # a stride of 6 floats that fusing rows a and g would hide
    "fused_stride": (("bcdea", "bagf", "fcged", dict(a=6, b=6, c=128, d=7, e=12, f=128, g=7)), 0),
    # forced transposed route whose first layout TMA cannot stage
    "forced_route": (("cafbed", "acbg", "fedg", dict(a=72, b=12, c=24, d=4, e=72, f=3, g=12)), 2),
    # estimates of the tcgen05 kernel that fused rows, or another transposed layout, make look cheaper than the CUDA cores
    "cheaper_when_fused_1": (("abcdef", "geac", "dfgb", dict(a=20, b=27, c=16, d=4, e=4, f=8, g=12)), 0),
    "cheaper_when_fused_2": (("abcdef", "gfac", "degb", dict(a=4, b=30, c=16, d=36, e=18, f=16, g=12)), 0),
    "cheaper_when_fused_3": (("abcdef", "dfgb", "geac", dict(a=4, b=3, c=256, d=4, e=512, f=48, g=96)), 0),
    "cheaper_when_fused_4": (("abcdef", "gfac", "degb", dict(a=9, b=12, c=21, d=15, e=13, f=11, g=52)), 0),
    "cheaper_when_fused_5": (("abcdef", "dfgb", "geac", dict(a=4, b=24, c=6, d=6, e=96, f=36, g=32)), 0),
    "cheaper_when_fused_6": (("abcdef", "gfac", "degb", dict(a=4, b=7, c=8, d=32, e=96, f=80, g=12)), 0),
    "ragged": (("abcd", "aebf", "fdec", dict(a=61, b=53, c=47, d=59, e=37, f=23)), 0),
}
TF32 = {
    "matrices": (("abcd", "aedf", "fbec", dict(a=72, b=72, c=72, d=72, e=72, f=72)), 0),
    "k_majors_large": (("abcd", "eafb", "fdec", dict(a=72, b=72, c=72, d=72, e=72, f=72)), 0),
}


@pytest.mark.parametrize("name", list(IEEE) + list(TF32))
def test_precision_of_the_route(engine, name):
    (modes, selection), kernel = (IEEE[name], "simt") if name in IEEE else (TF32[name], "umma_tf32")
    c = Contraction(*modes[:3], modes[3], F32)
    assert engine.plan(to_equation(engine, c, selection)).describe()["kernel"] == kernel


def test_no_contraction_moves_to_tf32(engine, monkeypatch):
    """golden/float32_line.txt: a character per descriptor, 1 where it ran as TF32 when the kernels of TMA-staged operands were
    planned mode by mode and the CUDA-core kernel had 64 x 64 tiles only."""
    here = os.path.dirname(os.path.abspath(__file__))
    monkeypatch.setenv("TCONT_COST_TABLE", os.path.join(os.path.dirname(here), "tcont_b200", "tcont_cost_table.NVIDIA_B200.txt"))
    with open(os.path.join(here, "golden", "float32_line.txt")) as f:
        was = "".join(f.read().split())
    tf32 = 0
    for before, (C, A, B, ext) in zip(was, descriptors(len(was)), strict=True):
        now = engine.plan(engine.TCEquation(C, A, B, ext, "-", engine.ScalarType(0))).describe()["kernel"] == "umma_tf32"
        assert before == "1" or not now, (C, A, B, ext)
        tf32 += now
    assert tf32 > 0.9 * was.count("1")     # (and the tensor cores are still used)


def test_cost_table_sets_the_line(engine, monkeypatch, tmp_path):
    (modes, selection) = IEEE["two_k_majors"]
    table = tmp_path / "table.txt"
    table.write_text("simt_f32_tflops 1\n")      # slow CUDA cores: one transpose and the tensor cores are worth it
    monkeypatch.setenv("TCONT_COST_TABLE", str(table))
    c = Contraction(*modes[:3], modes[3], F32)
    assert engine.plan(to_equation(engine, c, selection)).describe()["kernel"] == "umma_tf32"
    table.write_text("simt_f32_tflops 1\nline_launch_us 1000\n")   # (and two launches more are not)
    assert engine.plan(to_equation(engine, c, selection)).describe()["kernel"] == "simt"
