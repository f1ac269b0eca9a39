"""General fused passes (register stages) against the oracle: tiles with every
split of targets, low-order qubits as first and last targets, swaps that relabel
the line bits, phases and flips on tile and outer bits, zero pairs, programs too
long for one plan.  Exact form: every bit, signs of zeros included.  Fast forms:
rounding of at most a few ulp per operation, each at most sqrt(2) times the
state's norm times eps, so ops * eps covers relL2 with a margin (errors add in
quadrature)."""
import numpy as np
import pytest

import oracle as O
import tmfqsfullstate_b200 as tq

pytestmark = pytest.mark.gpu


def circuit(n, count, seed, kinds="hxcpsf", only=None):
    rng = np.random.default_rng(seed)
    pool = list(range(n)) if only is None else only
    ops = []
    for _ in range(count):
        a, b = (int(v) for v in rng.permutation(pool)[:2])
        c = int(rng.integers(0, n))
        k = kinds[int(rng.integers(0, len(kinds)))]
        ops.append({"h": lambda M: M.h(a), "x": lambda M: M.x(a), "c": lambda M: M.cnot(c if c != a else b, a),
                    "p": lambda M, t=float(rng.uniform(-4, 4)): M.cphase(c if c != a else b, a, t),
                    "s": lambda M: M.swap(a, b), "f": lambda M, s=int(rng.integers(0, 1 << n)): M.phase_flip(s)}[k])
        ops[-1] = (ops[-1], a, b, c)
    return ops


def build(ops, M):
    return [f(M) for f, *_ in ops]


def inputs(kind, n, seed):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((1 << n, 2))
    if kind == "sparse":
        a[rng.random(1 << n) < 0.9] = 0.0
        a[rng.random(1 << n) < 0.2, 0] = -0.0
    elif kind == "basis":
        a[:] = 0.0
        a[(1 << n) * 5 // 7, 0] = 1.0
    a /= np.linalg.norm(a)
    return a.reshape(-1)


def want(n, a, ops):
    r = O.OracleRegister(n, amps=a)
    r.run(build(ops, O))
    return r.amplitudes()


CASES = [("hxcpsf", None), ("hxcpf", None), ("hp", None), ("xcs", None), ("pf", None), ("hcps", "low"), ("hcps", "high"), ("hs", "ends")]


@pytest.mark.parametrize("kind", ["random", "sparse", "basis"])
@pytest.mark.parametrize("n", [12, 13, 14, 17])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_exact_bits(n, case, kind):
    kinds, where = CASES[case]
    only = {None: None, "low": list(range(n - 5, n)), "high": list(range(5)), "ends": [0, 1, 2, n - 3, n - 2, n - 1]}[where]
    ops = circuit(n, 60, 10 * n + case, kinds, only)
    a = inputs(kind, n, n + case)
    with tq.GpuState(tq.FP64) as g:
        g.load(n, a)
        g.apply_ops(build(ops, tq))
        got = g.export()
    ref = want(n, a, ops)
    assert np.array_equal(got, ref)
    if "s" not in kinds:  # the reference's swap is three CNOTs, which leave a (+0, -0) pair alone; ours exchanges it
        assert np.array_equal(np.signbit(got[got == 0]), np.signbit(ref[got == 0]))


@pytest.mark.parametrize("n", [12, 13, 14, 16, 18])
@pytest.mark.parametrize("form", ["c64", "f64fast"])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_fast_forms(n, case, form):
    kinds, where = CASES[case]
    only = {None: None, "low": list(range(n - 5, n)), "high": list(range(5)), "ends": [0, 1, 2, n - 3, n - 2, n - 1]}[where]
    ops = circuit(n, 80, 100 * n + case, kinds, only)
    a = inputs("random", n, n)
    with tq.GpuState(tq.FP32 if form == "c64" else tq.FP64) as g:
        if form == "f64fast":
            g.set_option(tq.OPT_EXACT, 0)
        g.load(n, a)
        g.apply_ops(build(ops, tq))
        got = g.export()
    eps = 2.0 ** -24 if form == "c64" else 2.0 ** -53
    assert O.rel_l2(want(n, a, ops), got) <= 80 * eps


@pytest.mark.parametrize("prec", [tq.FP64, tq.FP32])
def test_more_operations_than_one_plan_holds(prec):
    n = 14
    ops = circuit(n, 400, 3, "hp", list(range(9)))
    a = inputs("random", n, 5)
    with tq.GpuState(prec) as g:
        g.load(n, a)
        g.apply_ops(build(ops, tq))
        got = g.export()
    ref = want(n, a, ops)
    if prec == tq.FP64:
        assert np.array_equal(got, ref)
    else:
        assert O.rel_l2(ref, got) <= 400 * 2.0 ** -24


@pytest.mark.parametrize("n", [13, 14, 16])
@pytest.mark.parametrize("form,size", [("c64", 1e30), ("c64", 1e-30), ("f64fast", 1e290)])
def test_many_hadamards_far_from_norm_one(n, form, size):
    """220 operations, mostly Hadamards, on values next to the ends of the range: the outstanding powers of sqrt(2) stay small."""
    ops = circuit(n, 220, n, "hhhhhhhhc", list(range(8)))
    a = inputs("random", n, 7) * size
    with tq.GpuState(tq.FP32 if form == "c64" else tq.FP64) as g:
        if form == "f64fast":
            g.set_option(tq.OPT_EXACT, 0)
        g.load(n, a)
        g.apply_ops(build(ops, tq))
        got = g.export()
    ref = want(n, a / size, ops)
    assert O.rel_l2(ref, got / size) <= 220 * (2.0 ** -24 if form == "c64" else 2.0 ** -53)


def rings(n, layers, seed, extra):
    """Hadamard layers with rings of phases, and `extra` random phases after each (pairs in every position)."""
    rng = np.random.default_rng(seed)
    ops = []
    for _ in range(layers):
        ops += [lambda M, q=q: M.h(q) for q in range(n)]
        pairs = [(q, (q + 1) % n) for q in range(n)] + [tuple(int(v) for v in rng.permutation(n)[:2]) for _ in range(extra)]
        ops += [lambda M, c=c, q=q, x=float(rng.uniform(-4, 4)): M.cphase(c, q, x) for c, q in pairs]
    return ops


@pytest.mark.parametrize("n", [12, 13, 14, 15, 17, 19])
@pytest.mark.parametrize("form", ["c64", "f64fast"])
@pytest.mark.parametrize("extra", [0, 40])
def test_merged_phase_runs(n, form, extra):
    ops = rings(n, 3, n, extra)
    a = inputs("random", n, n)
    r = O.OracleRegister(n, amps=a)
    r.run([f(O) for f in ops])
    with tq.GpuState(tq.FP32 if form == "c64" else tq.FP64) as g:
        if form == "f64fast":
            g.set_option(tq.OPT_EXACT, 0)
        g.load(n, a)
        g.apply_ops([f(tq) for f in ops])
        got = g.export()
    assert O.rel_l2(r.amplitudes(), got) <= len(ops) * (2.0 ** -24 if form == "c64" else 2.0 ** -53)


@pytest.mark.parametrize("n", [20, 22])
def test_relabelled_tiles_of_one_stage(n):
    """A swap and few targets: one register stage, several tiles per block, every amplitude stored elsewhere in its tile."""
    ops = [lambda M: M.h(4), lambda M: M.swap(3, n - 1), lambda M: M.x(5), lambda M: M.cnot(1, 4)]
    a = inputs("random", n, 9)
    with tq.GpuState(tq.FP64) as g, tq.GpuState(tq.FP64) as one:
        one.set_option(tq.OPT_FUSION, 0)
        for s in (g, one):
            s.load(n, a)
            s.apply_ops([f(tq) for f in ops])
        assert g.compare(one)["bitwise_equal"]


def test_load_apply_runs_general_first_passes_in_slabs():
    n = 18
    ops = circuit(n, 40, 8, "hxcp", list(range(8, 18)))
    a = inputs("random", n, 6)
    with tq.GpuState(tq.FP64) as g:
        g.load_apply_ops(n, a, build(ops, tq))
        assert np.array_equal(g.export(), want(n, a, ops))
