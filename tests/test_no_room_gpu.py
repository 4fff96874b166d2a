"""Runs whose scratch copies or workspaces find no room: another form of the same precision, or an error that leaves everything as it was."""
import numpy as np
import pytest

from cases import to_equation
from oracle_lib import F32, F64, Contraction
from test_across_tf32_gpu import big
from test_contraction_gpu import check
from test_fp64_tiles_gpu import PADDED, hold

pytestmark = pytest.mark.gpu


def on_device(engine, oracle, c, selection):
    import torch
    from tcont_b200 import api
    A, B = oracle.inputs(c, 53, -1.0, 1.0)
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    dC = torch.zeros(c.size(c.modeC), dtype=dA.dtype, device="cuda")
    plan = engine.plan(to_equation(engine, c, selection))
    desc = plan.describe()

    def prepare():
        return api.prepare_on_device(plan, dA.data_ptr(), dB.data_ptr(), dC.data_ptr(), keep=(dA, dB, dC))

    def output(run):
        engine.launch(run)
        torch.cuda.synchronize()
        return dC.cpu().numpy()
    return A, B, desc, prepare, output


def test_padded_copies(engine, oracle, monkeypatch):
    """Odd strides: the operands are used where they lie, unless the caller asked for the copies."""
    monkeypatch.setenv("TCONT_PADDED_COPIES", "1")
    monkeypatch.setenv("TCONT_KERNEL", "tma")
    C, A_, B_, ext = PADDED["in_order"]
    c = Contraction(C, A_, B_, ext, F64)
    A, B, desc, prepare, output = on_device(engine, oracle, c, 0)
    assert desc["backend"] == "ttgt" and desc["kernel"] == "dmma_f64_tma"
    monkeypatch.setenv("TCONT_TEST_NO_ROOM", "1000")
    run = prepare()
    hold(oracle, c, A, B, output(run), ext["k"])
    assert run.time_launches(1)[1] == 1
    *_, prepare, _ = on_device(engine, oracle, c, 2)
    with pytest.raises(RuntimeError):
        prepare()
    monkeypatch.delenv("TCONT_TEST_NO_ROOM")
    assert prepare().time_launches(1)[1] == 3


@pytest.mark.parametrize("modes,extent,staged", [(("abcd", "aedf", "fbec"), 40, True), (("abcd", "eafb", "fdec"), 24, False)])
def test_float32_keeps_its_precision(engine, oracle, monkeypatch, modes, extent, staged):
    """TF32 behind copies runs without them where the tensor cores can be fed from the operands as they lie, and is refused where not."""
    c = Contraction(*modes, dict.fromkeys("abcdef", extent), F32)
    A, B, desc, prepare, output = on_device(engine, oracle, c, 0)
    assert desc["backend"] == "ttgt" and desc["kernel"] == "umma_tf32"
    monkeypatch.setenv("TCONT_SPLITK", "1")
    monkeypatch.setenv("TCONT_TEST_NO_ROOM", "1000")
    if staged:
        check(oracle, c, A, B, output(prepare()), desc)
    else:
        with pytest.raises(RuntimeError, match="no room"):
            prepare()
    monkeypatch.delenv("TCONT_TEST_NO_ROOM")
    check(oracle, c, A, B, output(prepare()), desc)


def test_scalars(engine, oracle, monkeypatch):
    """set_scalars: no room for the copies of the form that would be faster, for the workspace, for either."""
    import torch

    def scaled(run, dC, held):
        dC.fill_(3.0)
        engine.launch(run)
        torch.cuda.synchronize()
        return held(0.3, -0.7, 3.0)

    # C (157 MB) 50 times A: the form with copies of both operands; without room for them and for a workspace, on A and B as they lie;
    # without room for anything, an error
    run, dC, held = big(engine, oracle, dict(a=32, b=24, c=40, d=32, e=40, f=16))
    monkeypatch.setenv("TCONT_TEST_NO_ROOM", "1")
    with pytest.raises(RuntimeError):
        run.set_scalars(0.3, -0.7)
    engine.launch(run)
    torch.cuda.synchronize()
    assert held(1.0, 0.0, 0.0) and run.time_launches(1)[1] == 1 and run.device_status() == 0
    monkeypatch.setenv("TCONT_TEST_NO_ROOM", "100000000")
    run.set_scalars(0.3, -0.7)
    assert scaled(run, dC, held) and run.time_launches(1)[1] == 3
    run, dC, held = big(engine, oracle, dict(a=32, b=24, c=40, d=32, e=40, f=16))
    monkeypatch.setenv("TCONT_TEST_NO_ROOM", "1000")
    run.set_scalars(0.3, -0.7)
    assert scaled(run, dC, held) and run.time_launches(1)[1] == 1 and run.device_status() == 0
    monkeypatch.delenv("TCONT_TEST_NO_ROOM")
    # C (8 MB) of twice A's size: the workspace; without room for it the form with a copy of A
    run, dC, held = big(engine, oracle, dict(a=64, b=8, c=16, d=4, e=64, f=32))
    monkeypatch.setenv("TCONT_TEST_NO_ROOM", str(dC.numel() * 4))
    run.set_scalars(0.3, -0.7)
    assert scaled(run, dC, held) and run.time_launches(1)[1] >= 1
    monkeypatch.delenv("TCONT_TEST_NO_ROOM")
    run.set_scalars(0.3, -0.7)
    assert scaled(run, dC, held) and run.time_launches(1)[1] == 2 and run.device_status() == 0
