"""Which Float32 contractions run in IEEE single precision: a faster gather kernel, operand-level fusion of rows or another
transposed layout must not take one of them to TF32 (planner only, no GPU)."""
import pytest

from cases import to_equation
from oracle_lib import F32, Contraction

IEEE = {
    # K-major on two different modes, direct; one transpose and the tensor cores would now look cheaper than the gather kernel
    "two_k_majors": (("ab", "cad", "dcb", dict(a=224, b=224, c=16, d=256)), 0),
    # a stride of 6 floats that fusing rows a and g would hide
    "fused_stride": (("bcdea", "bagf", "fcged", dict(a=6, b=6, c=128, d=7, e=12, f=128, g=7)), 0),
    # forced transposed route whose first layout TMA cannot stage
    "forced_route": (("cafbed", "acbg", "fedg", dict(a=72, b=12, c=24, d=4, e=72, f=3, g=12)), 2),
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
