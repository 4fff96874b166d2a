"""Float32 tiles across A's and C's stride-1 modes, at the edges of what a tile holds: 16 of C's mode, 32 of A's, pieces of eight
columns, tiles of 32 or 64, k chunks of 8 to 32; against the TF32-operand oracle like every tensor-core result."""
import numpy as np
import pytest

from cases import to_equation
from oracle_lib import F32, Contraction
from test_contraction_gpu import check

pytestmark = pytest.mark.gpu

# y = C's stride-1 mode, x = A's; name -> (descriptor, BN, BK, B's layout)
FORMS = {
    "whole": ("abcde", "efbad", "cf", dict(a=48, b=3, c=24, d=2, e=64, f=32), 32, 32, "MN"),
    "ragged_all": ("abcd", "dbea", "ec", dict(a=20, b=5, c=11, d=36, e=40), 32, 32, "K"),
    "y_of_8": ("abcd", "dbea", "ec", dict(a=8, b=7, c=33, d=48, e=20), 64, 32, "K"),
    "x_of_4": ("acb", "bka", "kc", dict(a=36, b=4, c=70, k=64), 64, 32, "K"),
    "k_of_8": ("abcd", "dbea", "ce", dict(a=16, b=5, c=24, d=32, e=8), 32, 8, "MN"),
    "k_of_13": ("abcd", "dbea", "ce", dict(a=24, b=5, c=96, d=20, e=13), 64, 16, "MN"),
    "k_chunks_of_24": ("abcd", "dbea", "ce", dict(a=24, b=5, c=36, d=44, e=72), 64, 24, "MN"),
    "two_k": ("abcd", "dfbea", "cfe", dict(a=32, b=3, c=40, d=36, e=12, f=7), 64, 8, "MN"),
    "two_n": ("abcd", "dka", "cbk", dict(a=40, b=6, c=16, d=52, k=33), 32, 32, "MN"),
    "swapped": ("abc", "kb", "cka", dict(a=40, b=21, c=36, k=28), 32, 32, "K"),
    "many_tiles": ("abcd", "dbea", "ec", dict(a=64, b=24, c=20, d=160, e=36), 32, 32, "K"),
}


@pytest.mark.parametrize("name", list(FORMS))
@pytest.mark.parametrize("rows_first", ["0", "1"])
def test_forms(engine, oracle, monkeypatch, name, rows_first):
    """Plain, then alpha and beta through the workspace; nothing outside C is written."""
    import torch
    from tcont_b200 import api
    monkeypatch.setenv("TCONT_ACROSS", "1")
    monkeypatch.setenv("TCONT_ACROSS_ROWS_FIRST", rows_first)
    C, A_, B_, ext, bn, bk, layout = FORMS[name]
    c = Contraction(C, A_, B_, ext, F32)
    A, B = oracle.inputs(c, 37, -1.0, 1.0)
    n = c.size(C)
    C0 = np.random.default_rng(9).uniform(-4.0, 4.0, n).astype(np.float32)
    guarded = torch.full((n + 64,), 7.0, device="cuda")
    dC = guarded[32:32 + n]
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    plan = engine.plan(to_equation(engine, c, 1))
    desc = plan.describe()
    assert desc["kernel"] == "umma_tf32" and (desc["across"]["BN"], desc["across"]["BK"], desc["across"]["b_major"]) == (bn, bk, layout), desc
    run = api.prepare_on_device(plan, dA.data_ptr(), dB.data_ptr(), dC.data_ptr(), keep=(dA, dB, guarded))
    for _ in range(2):
        engine.launch(run)
    torch.cuda.synchronize()
    plain = dC.cpu().numpy()
    check(oracle, c, A, B, plain, desc)
    product, scale = oracle.contract(c, A, B, rounding=1), oracle.contract(c, np.abs(A), np.abs(B), rounding=1)
    for alpha, beta in ((0.3, -0.7), (-2.0, 0.0)):
        dC.copy_(torch.from_numpy(C0))
        run.set_scalars(alpha, beta)
        engine.launch(run)
        torch.cuda.synchronize()
        want = alpha * product + beta * C0.astype(np.float64)
        bound = 2e-5 * abs(alpha) * scale + 4 * 2.0**-24 * (np.abs(alpha * product) + np.abs(beta * C0.astype(np.float64)))
        assert (np.abs(dC.cpu().numpy() - want) <= bound).all(), (alpha, beta)
    run.set_scalars(1.0, 0.0)
    engine.launch(run)
    torch.cuda.synchronize()
    assert np.array_equal(dC.cpu().numpy(), plain) and run.device_status() == 0
    assert bool((torch.cat([guarded[:32], guarded[32 + n:]]) == 7.0).all())


def test_view(engine, oracle, monkeypatch):
    """Sub-tensor views: what lies between the view's elements in C's parent stays as it is."""
    import torch
    from tcont_b200 import api
    monkeypatch.setenv("TCONT_ACROSS", "1")
    ext = dict(a=24, b=5, c=12, d=40, e=36)
    c = Contraction("abcd", "dbea", "ec", ext, F32)
    A, B = oracle.inputs(c, 41, -1.0, 1.0)
    parent_c, parent_a = [28, 6, 12, 44], [44, 5, 40, 26]
    big_c = torch.full(tuple(reversed(parent_c)), 7.0, device="cuda")
    big_a = torch.zeros(tuple(reversed(parent_a)), device="cuda")
    big_a[:24, :36, :5, :40] = torch.from_numpy(A).cuda().reshape(24, 36, 5, 40)
    dB = torch.from_numpy(B).cuda()
    plan = api.plan_views(to_equation(engine, c, 1), parent_c=parent_c, parent_a=parent_a)
    desc = plan.describe()
    assert "across" in desc
    run = api.prepare_on_device(plan, big_a.data_ptr(), dB.data_ptr(), big_c.data_ptr(), keep=(big_a, dB, big_c))
    engine.launch(run)
    torch.cuda.synchronize()
    inside = big_c[:40, :12, :5, :24].contiguous().cpu().numpy().reshape(-1)
    check(oracle, c, A, B, inside, desc)
    big_c[:40, :12, :5, :24] = 7.0
    assert bool((big_c == 7.0).all())


def test_error_compensated_keeps_its_form(engine, oracle, monkeypatch):
    """TCONT_TF32X3 asked for after planning: the run is planned again, and meets the IEEE criterion."""
    monkeypatch.setenv("TCONT_ACROSS", "1")
    c = Contraction("abcd", "dbea", "ec", dict(a=24, b=5, c=12, d=40, e=36), F32)
    A, B = oracle.inputs(c, 43, -1.0, 1.0)
    plan = engine.plan(to_equation(engine, c, 1))
    assert "across" in plan.describe()
    monkeypatch.setenv("TCONT_TF32X3", "1")
    run = engine.prepare(plan, A, B)
    engine.launch(run)
    diff, nonfinite = oracle.compare(oracle.contract(c, A, B, rounding=0), engine.copy_output_to_host(run), F32)
    assert diff == 0 and nonfinite == 0


def test_bounded_wait_gives_up_cleanly(engine, oracle, monkeypatch):
    """One stage of every CTA is neither announced nor filled: the waits behind it run out, the run's status says so, nothing outside
    C is written, and the next run is right."""
    import torch
    from tcont_b200 import api
    monkeypatch.setenv("TCONT_ACROSS", "1")
    c = Contraction("abcd", "dbea", "ec", dict(a=64, b=24, c=20, d=160, e=36), F32)
    A, B = oracle.inputs(c, 9, -1.0, 1.0)
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    n = c.size("abcd")
    guarded = torch.full((n + 64,), 7.0, device="cuda")
    plan = engine.plan(to_equation(engine, c, 1))
    assert plan.describe()["across"]["k_iters"] == 2

    def run():
        return api.prepare_on_device(plan, dA.data_ptr(), dB.data_ptr(), guarded[32:].data_ptr(), keep=(dA, dB, guarded))
    monkeypatch.setenv("TCONT_TEST_WAIT_LIMIT_NS", "2000000")
    monkeypatch.setenv("TCONT_TEST_SKIP_STAGE", "3")   # the second tile's second k iteration
    broken = run()
    monkeypatch.delenv("TCONT_TEST_WAIT_LIMIT_NS")
    monkeypatch.delenv("TCONT_TEST_SKIP_STAGE")
    engine.launch(broken)
    torch.cuda.synchronize()
    assert broken.device_status() == 1
    assert bool((torch.cat([guarded[:32], guarded[32 + n:]]) == 7.0).all())
    del broken
    good = run()
    engine.launch(good)
    torch.cuda.synchronize()
    assert good.device_status() == 0
    check(oracle, c, A, B, guarded[32:32 + n].cpu().numpy(), plan.describe())


def big(engine, oracle, ext):
    """A contraction the planner takes this form for by itself, a run of it on device tensors and 20 000 elements of its product."""
    import torch
    from tcont_b200 import api
    c = Contraction("abcde", "efba", "cfd", ext, F32)
    A, B = oracle.inputs(c, 47, -1.0, 1.0)
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    dC = torch.zeros(c.size("abcde"), device="cuda")
    plan = engine.plan(to_equation(engine, c, 0))
    assert "across" in plan.describe()
    run = api.prepare_on_device(plan, dA.data_ptr(), dB.data_ptr(), dC.data_ptr(), keep=(dA, dB, dC))
    at = np.sort(np.random.default_rng(5).integers(0, dC.numel(), 20000))
    product, scale = (oracle.contract_sampled(c, a, b, at, rounding=1) for a, b in ((A, B), (np.abs(A), np.abs(B))))

    def held(alpha, beta, old):
        got = dC.cpu().numpy()[at]
        want = alpha * product + beta * old
        return bool((np.abs(got - want) <= 2e-5 * abs(alpha) * scale + 4 * 2.0**-24 * (np.abs(alpha * product) + np.abs(beta * old))).all())
    return run, dC, held


# a C 40 times the size of A is accumulated into by the form that applies scalars in its epilogue (copies of both operands in front of
# it), one of A's size by a second pass over a workspace; kernels of a plain launch, of an accumulating one
@pytest.mark.parametrize("ext,kernels", [(dict(a=32, b=24, c=40, d=32, e=40, f=16), 3), (dict(a=64, b=8, c=8, d=4, e=64, f=32), 2)])
def test_form_of_accumulating_launches(engine, oracle, ext, kernels):
    """Chosen when the scalars are set, beside the plain form: a graph that holds a plain launch stays what it is."""
    import torch
    run, dC, held = big(engine, oracle, ext)
    stream = torch.cuda.Stream()
    run.set_stream(stream.cuda_stream)
    with torch.cuda.stream(stream):
        engine.launch(run)
        stream.synchronize()
        assert held(1.0, 0.0, 0.0) and run.time_launches(1)[1] == 1
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            engine.launch(run)
        for alpha, beta in ((0.3, -0.7), (-2.0, 0.0), (1.0, 1.0)):
            dC.fill_(3.0)
            run.set_scalars(alpha, beta)
            engine.launch(run)
            stream.synchronize()
            assert held(alpha, beta, 3.0), (alpha, beta)
        assert run.time_launches(1)[1] == kernels
        dC.fill_(3.0)
        graph.replay()
        stream.synchronize()
        assert held(1.0, 0.0, 0.0)
        run.set_scalars(1.0, 0.0)
        dC.fill_(3.0)
        engine.launch(run)
        stream.synchronize()
        assert held(1.0, 0.0, 0.0) and run.time_launches(1)[1] == 1 and run.device_status() == 0
    other = torch.cuda.Stream()
    run.set_scalars(2.0, 1.0)
    run.set_stream(other.cuda_stream)   # (the other form follows the run's stream)
    with torch.cuda.stream(other):
        dC.fill_(3.0)
        engine.launch(run)
        other.synchronize()
    assert held(2.0, 1.0, 3.0) and run.device_status() == 0


def test_accumulating_parts_of_a_host_pass(engine, oracle, monkeypatch):
    """Each part applies the scalars to its range of C, whose old values are what the pass before left there."""
    monkeypatch.setenv("TCONT_HOST_CHUNKS", "2")
    c = Contraction("abcde", "efba", "cfd", dict(a=32, b=24, c=40, d=16, e=40, f=16), F32)
    A, B = oracle.inputs(c, 59, -1.0, 1.0)
    plan = engine.plan(to_equation(engine, c, 0))
    assert "across" in plan.describe()
    run = engine.prepare(plan, A, B)
    first, second = np.empty(c.size("abcde"), np.float32), np.empty(c.size("abcde"), np.float32)
    run.contract_host(A, B, first)
    run.set_scalars(0.3, -0.7)
    run.contract_host(A, B, second)
    at = np.sort(np.random.default_rng(6).integers(0, first.size, 20000))
    product, scale = (oracle.contract_sampled(c, a, b, at, rounding=1) for a, b in ((A, B), (np.abs(A), np.abs(B))))
    assert (np.abs(first[at] - product) <= 2e-5 * scale).all()
    want = 0.3 * product - 0.7 * first[at].astype(np.float64)
    assert (np.abs(second[at] - want) <= 2e-5 * 0.3 * scale + 4 * 2.0**-24 * (np.abs(0.3 * product) + np.abs(0.7 * first[at]))).all()
