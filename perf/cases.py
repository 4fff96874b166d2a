"""What a program that uses this engine has it do: binary tensor contractions on column-major tensors that lie in GPU
memory, planned and prepared once, launched many times (`plan` -> `prepare_on_device` -> `launch`).

The listed cases and `draw` cover the engine's mode patterns (tensor times matrix, matrix-like, 4-D by 4-D, 6-D output,
short contracted extent), both element types (Float32 = TF32 multiply with fp32 accumulation, Float64), extents that are
multiples of 8 and ragged ones (numbers of orbitals are arbitrary integers), plain and accumulating launches
(C = alpha A B + beta C), and sizes from a few million operations, where latency counts, to several TFLOP.
"""
import math

import torch

import tcont_b200 as tc
import tcont_b200.api  # noqa: F401

F32, F64 = 0, 1


def _case(name, C, A, B, st, extents, alpha=1.0, beta=0.0):
    modes = sorted(set(C + A + B))
    c = {"C": C, "A": A, "B": B, "f64": st == F64, "alpha": alpha, "beta": beta}
    c.update({"ext_" + m: int(e) for m, e in zip(modes, extents)})
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one small term of a coupled-cluster residual: a loop over many of these is bound by latency and launches
        _case("f64_4d_small", "abcd", "aebf", "fdec", F64, (24, 24, 24, 24, 16, 16)),
        # the same for Float32 with ragged extents (no stride is a multiple of 16 bytes)
        _case("f32_3d_small_ragged", "abc", "adc", "db", F32, (63, 47, 11, 41)),
        # one index of a 4-D tensor transformed by a matrix; the tensor's fastest mode is not the output's
        _case("f64_tensor_matrix", "abcd", "dbea", "ec", F64, (72, 72, 24, 72, 72)),
        # the same for a 5-D tensor in Float32
        _case("f32_tensor_matrix_5d", "abcde", "efbad", "cf", F32, (48, 32, 24, 32, 48, 32)),
        # two 4-D tensors over two modes, the particle-particle / ring terms of coupled cluster: bound by arithmetic
        _case("f64_4d", "abcd", "aebf", "fdec", F64, (72,) * 6),
        _case("f32_4d", "abcd", "aedf", "fbec", F32, (72,) * 6),
        # perturbative triples: a 6-D output from a short contracted mode; terms are added up in the same output
        _case("f64_6d_accumulate", "abcdef", "dega", "gfbc", F64, (24, 16, 16, 24, 16, 16, 24), 1.0, 1.0),
        _case("f32_6d", "abcdef", "gdab", "efgc", F32, (24, 16, 16, 24, 16, 16, 24)),
        # ragged extents at a size where the arithmetic counts
        _case("f64_4d_ragged", "abcd", "aebf", "fdec", F64, (61, 53, 47, 59, 37, 23)),
        # matrix-like with a permuted output, compute bound
        _case("f32_3d", "abc", "adc", "db", F32, (256, 1024, 256, 1024)),
        # short contracted mode, permuted inputs: bound by memory bandwidth
        _case("f32_5d_low_k", "abcde", "efba", "cfd", F32, (48, 48, 48, 48, 48, 8)),
        # the largest: 8.8 TFLOP in one launch
        _case("f32_4d_large", "abcd", "aebf", "cfde", F32, (128,) * 6),
    ]


# family -> (mode patterns, range of operations, range of the contracted extent of one mode)
_FAMILIES = {
    "tensor_matrix": (["abc bda dc", "abc dca bd", "abcd dbea ec", "abcd deca be", "abcd ebad ce", "abcde efbad cf",
                       "abcde ecbfa fd", "abcde efcad bf", "abcd ea ebcd", "abcd eb aecd", "abcd ec abed"],
                      (2e6, 2e10), (16, 320)),
    "matrix_like": (["ab ac cb", "ab acd dbc", "ab cad dcb", "abc acd db", "abc ad bdc", "abc adc bd", "abc adc db",
                     "abc adec ebd"], (2e6, 1e12), (16, 1024)),
    "four_d": (["abcd aebf dfce", "abcd aebf fdec", "abcd aecf bfde", "abcd aecf fbed", "abcd aedf bfce", "abcd aedf fbec",
                "abcd aefb fdce", "abcd aefc fbed", "abcd eafb fdec", "abcd eafc bfde", "abcd eafd fbec", "abcd aebf cfde"],
               (2e6, 1e12), (8, 128)),
    "six_d": (["abcdef dega gfbc", "abcdef degb gfac", "abcdef degc gfab", "abcdef dfga gebc", "abcdef dfgb geac",
               "abcdef dfgc geab", "abcdef efga gdbc", "abcdef efgb gdac", "abcdef efgc gdab", "abcdef gdab efgc",
               "abcdef gdac efgb", "abcdef gdbc efga", "abcdef geab dfgc", "abcdef geac dfgb", "abcdef gebc dfga",
               "abcdef gfab degc", "abcdef gfac degb", "abcdef gfbc dega", "abcijk aeij bcek"],
              (2e6, 2e10), (12, 64)),
    "low_k": (["abcde efba cfd"], (2e6, 4e9), (4, 16)),
}


def draw(rng):
    while True:
        patterns, (lo, hi), (klo, khi) = _FAMILIES[rng.choice(sorted(_FAMILIES))]
        C, A, B = rng.choice(patterns).split()
        st = rng.choice((F32, F64))
        ragged = rng.random() < 0.4
        beta = 1.0 if rng.random() < 0.2 else 0.0
        # FP64 and ragged Float32 run at a fraction of the TF32 rate: keep them below the largest listed case
        top = min(hi, 1e11 if st == F64 or ragged else hi)
        flops = math.exp(rng.uniform(math.log(lo), math.log(top)))
        modes = sorted(set(C + A + B))
        contracted = [m for m in modes if m not in C]
        ext = {m: math.exp(rng.uniform(math.log(klo), math.log(khi))) for m in contracted}
        k = math.prod(ext.values())
        outer = [m for m in modes if m in C]
        each = (flops / (2.0 * k)) ** (1.0 / len(outer)) if flops > 2.0 * k else 0.0
        for m in outer:
            ext[m] = each * math.exp(rng.uniform(-0.5, 0.5))
        if ragged:
            sizes = {m: 2 * int(e / 2) + 1 if rng.random() < 0.7 else int(e) for m, e in ext.items()}
        else:
            step = 8 if min(ext.values()) >= 8 else 4
            sizes = {m: step * round(e / step) for m, e in ext.items()}
        if min(sizes.values()) < 2:
            continue
        case = _case(None, C, A, B, st, [sizes[m] for m in modes], 1.0, beta)
        w = work(case)
        if 1e6 <= w["flops"] <= 2.0 * top and w["bytes"] <= 2e9:
            return case


def _extent(case):
    return {k[4:]: v for k, v in case.items() if k.startswith("ext_")}


def _count(case, tensor):
    e = _extent(case)
    return math.prod(e[m] for m in case[tensor])


def prepare(case, seed):
    """Tensors in GPU memory, the plan and the run that a program keeps for a contraction it repeats."""
    dtype = torch.float64 if case["f64"] else torch.float32
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    a, b, c = (torch.empty(_count(case, t), dtype=dtype, device="cuda").uniform_(-1.0, 1.0, generator=g) for t in "ABC")
    eq = tc.TCEquation(case["C"], case["A"], case["B"], _extent(case), "+", tc.ScalarType(F64 if case["f64"] else F32))
    run_ = tc.api.prepare_on_device(tc.plan(eq), a.data_ptr(), b.data_ptr(), c.data_ptr(), keep=(a, b, c))
    if (case["alpha"], case["beta"]) != (1.0, 0.0):
        run_.set_scalars(case["alpha"], case["beta"])
    return run_, c


def run(state):
    run_, c = state
    tc.launch(run_)
    return c


def work(case):
    """Both inputs read once, the output written once (and read once where it is accumulated into)."""
    n = {t: _count(case, t) for t in "ABC"}
    k = math.prod(e for m, e in _extent(case).items() if m not in case["C"])
    elt = 8 if case["f64"] else 4
    return {"bytes": elt * (n["A"] + n["B"] + n["C"] * (2 if case["beta"] else 1)), "flops": 2.0 * n["C"] * k}


def tolerance(case):
    # Measured against the product in 64 bits (its sums in another order).  Float64: 2e-16 to 2.5e-15 relative to the
    # result's norm with the contracted extent from 24 to 5 184, the worst single value 2e-14.  Float32: operands
    # narrowed to TF32 (10 stored mantissa bits, truncated) give 6.9e-4 whatever the contracted extent, the worst
    # single value 2.2e-3.
    return {"rel": 1e-14, "max": 1e-13} if case["f64"] else {"rel": 2.8e-3, "max": 1e-2}


def exact(case, seed):
    """The same contraction by torch.einsum in 64 bits; column-major tensors are row-major ones with their modes reversed."""
    dtype = torch.float64 if case["f64"] else torch.float32
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    e = _extent(case)
    a, b, c = (torch.empty(_count(case, t), dtype=dtype, device="cuda").uniform_(-1.0, 1.0, generator=g).double()
               .reshape([e[m] for m in reversed(case[t])]) for t in "ABC")
    out = torch.einsum("%s,%s->%s" % (case["A"][::-1], case["B"][::-1], case["C"][::-1]), a, b)
    return (case["alpha"] * out + case["beta"] * c).reshape(-1)
