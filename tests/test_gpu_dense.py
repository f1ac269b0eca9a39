"""Dense gates against the oracle's applyGate: the tiled kernel at every k it
takes (targets on the lowest, highest and scattered qubits, states of one tile
and more), one- and two-qubit gates inside fused passes, and the sizes around
them.  Exact form: every bit.  Fast forms: a dot product of 2^k complex terms is
off by at most (2^(k+1) + 2) eps times its operands' norms, and the unitary keeps
the state's norm, so relL2 <= sum of (2^(k+1) + 2) eps 2^(k/2) over the gates
bounds it for rows of norm 1."""
import numpy as np
import pytest

import oracle as O
import tmfqsfullstate_b200 as tq

pytestmark = pytest.mark.gpu


def unitary(d, seed):
    rng = np.random.default_rng(seed)
    q, r = np.linalg.qr(rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


def state(n, seed, sparse=False):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((1 << n, 2))
    if sparse:
        a[rng.random(1 << n) < 0.97] = 0.0
    return (a / np.linalg.norm(a)).reshape(-1)


def apply(form, n, a, ops):
    with tq.GpuState(tq.FP32 if form == "c64" else tq.FP64) as g:
        if form == "f64fast":
            g.set_option(tq.OPT_EXACT, 0)
        g.load(n, a)
        g.apply_ops(ops)
        return g.export()


def want(n, a, ops):
    r = O.OracleRegister(n, amps=a)
    r.run(ops)
    return r.amplitudes()


def bound(form, ks):
    eps = 2.0 ** -24 if form == "c64" else 2.0 ** -53
    return sum((2.0 ** (k + 1) + 2) * 2.0 ** (k / 2) for k in ks) * eps


def targets(n, k, where):
    rng = np.random.default_rng(n * 100 + k)
    return {"low": list(range(n - 1, n - 1 - k, -1)), "high": list(range(k)), "any": [int(v) for v in rng.permutation(n)[:k]]}[where]


@pytest.mark.parametrize("n,k", [(11, 3), (11, 6), (12, 3), (12, 4), (13, 5), (13, 6), (14, 7), (13, 8), (12, 10), (13, 9)])
@pytest.mark.parametrize("where", ["low", "high", "any"])
def test_wide_gates(n, k, where):
    u, q, a = unitary(1 << k, k), targets(n, k, where), state(n, n + k)
    ref = want(n, a, [O.gate(u, q)])
    assert np.array_equal(apply("f64", n, a, [tq.gate(u, q)]), ref)
    sparse = state(n, k, sparse=True)
    assert np.array_equal(apply("f64", n, sparse, [tq.gate(u, q)]), want(n, sparse, [O.gate(u, q)]))
    assert O.rel_l2(ref, apply("f64fast", n, a, [tq.gate(u, q)])) <= bound("f64fast", [k])
    if k not in (4, 5):  # those run on the tensor cores
        assert O.rel_l2(ref, apply("c64", n, a, [tq.gate(u, q)])) <= bound("c64", [k])


@pytest.mark.parametrize("n,k", [(14, 3), (15, 3), (16, 3), (15, 6), (16, 7), (15, 8), (16, 8), (16, 9), (17, 9), (17, 10), (18, 10)])
def test_wide_gates_where_the_kernel_changes(n, k):
    """Registers on both sides of the line between one CTA per block and the tiled kernel."""
    for where in ("low", "any"):
        u, q = unitary(1 << k, k), targets(n, k, where)
        for a in (state(n, n + k), state(n, k, sparse=True)):
            ref = want(n, a, [O.gate(u, q)])
            assert np.array_equal(apply("f64", n, a, [tq.gate(u, q)]), ref)
            for form in ("f64fast", "c64"):
                assert O.rel_l2(ref, apply(form, n, a, [tq.gate(u, q)])) <= bound(form, [k])


def mixed(n, count, seed, dense_only=False):
    rng = np.random.default_rng(seed)
    ours, theirs, ks = [], [], []
    for i in range(count):
        q = [int(v) for v in rng.permutation(n)[:2]]
        kind = int(rng.integers(0, 2 if dense_only else 6))
        if kind < 2:
            u = unitary(2 << kind, seed * 1000 + i)
            q = q[:kind + 1]
            ours.append(tq.gate(u, q))
            theirs.append(O.gate(u, q))
        else:
            t = float(rng.uniform(-3, 3))
            for M, out in ((tq, ours), (O, theirs)):
                out.append([M.h(q[0]), M.cnot(*q), M.cphase(q[0], q[1], t), M.swap(*q)][kind - 2])
        ks.append(2)
    return ours, theirs, ks


@pytest.mark.parametrize("n", [5, 11, 12, 13, 14, 16])
@pytest.mark.parametrize("dense_only", [False, True])
@pytest.mark.parametrize("form", ["f64", "f64fast", "c64"])
def test_small_gates_in_passes(n, dense_only, form):
    ours, theirs, ks = mixed(n, 50, n, dense_only)
    for sparse in (False, True):
        a = state(n, n, sparse)
        got, ref = apply(form, n, a, ours), want(n, a, theirs)
        if form == "f64":
            assert np.array_equal(got, ref)
        else:
            assert O.rel_l2(ref, got) <= bound(form, ks)


@pytest.mark.parametrize("form", ["f64", "c64"])
def test_dense_gate_alone_and_at_pass_limits(form):
    """One gate (no pass), 70 one-qubit gates on few qubits (over one plan's operations), and an invalid gate after good ones."""
    n = 14
    a = state(n, 1)
    u = unitary(4, 3)
    got, ref = apply(form, n, a, [tq.gate(u, [3, 9])]), want(n, a, [O.gate(u, [3, 9])])
    assert np.array_equal(got, ref) if form == "f64" else O.rel_l2(ref, got) <= bound(form, [2])
    us = [unitary(2, i) for i in range(70)]
    got = apply(form, n, a, [tq.gate(x, [i % 9]) for i, x in enumerate(us)])
    ref = want(n, a, [O.gate(x, [i % 9]) for i, x in enumerate(us)])
    assert np.array_equal(got, ref) if form == "f64" else O.rel_l2(ref, got) <= bound(form, [1] * 70)
    with tq.GpuState(tq.FP32 if form == "c64" else tq.FP64) as g:
        g.load(n, a)
        with pytest.raises(tq.InvalidArgument):
            g.apply_ops([tq.h(0), tq.gate(u, [3, 9]), tq.gate(u, [4, 4])])
        ref = want(n, a, [O.h(0), O.gate(u, [3, 9])])
        assert np.array_equal(g.export(), ref) if form == "f64" else O.rel_l2(ref, g.export()) <= bound(form, [1, 2])


@pytest.mark.parametrize("n", [12, 14, 17])
@pytest.mark.parametrize("k", [1, 2])
@pytest.mark.parametrize("where", ["before", "between", "after"])
@pytest.mark.parametrize("form", ["f64", "f64fast", "c64"])
def test_gates_beside_rings_of_phases(n, k, where, form):
    """Layers of small gates around a layer of Hadamards and a ring of controlled phases (the run of phases merges in
    the fast complex128 form), fused and gate by gate."""
    rng = np.random.default_rng(n + k)

    def gates(M, seed):
        return [M.gate(unitary(1 << k, seed + q), list(range(q, q + k))) for q in range(0, n - k + 1, k)]

    def ops(M):
        t = np.random.default_rng(n).uniform(-3, 3, n)
        ring = [M.cphase(q, (q + 1) % n, float(t[q])) for q in range(n)]
        hs = [M.h(q) for q in range(n)]
        first = {"before": gates(M, 1) + hs + ring, "between": hs + gates(M, 1) + ring, "after": hs + ring + gates(M, 1)}[where]
        return first + ring + gates(M, 50)

    a = rng.standard_normal(2 << n)
    a /= np.linalg.norm(a)
    ref = want(n, a, ops(O))
    others = len(ops(tq)) - 2 * len(gates(tq, 1))
    limit = bound(form, [k] * (2 * len(gates(tq, 1)))) + others * (2.0 ** -24 if form == "c64" else 2.0 ** -53)
    for fusion in (1, 0):
        with tq.GpuState(tq.FP32 if form == "c64" else tq.FP64) as g:
            if form == "f64fast":
                g.set_option(tq.OPT_EXACT, 0)
            g.set_option(tq.OPT_FUSION, fusion)
            g.load(n, a)
            g.apply_ops(ops(tq))
            got = g.export()
        assert np.array_equal(got, ref) if form == "f64" else O.rel_l2(ref, got) <= limit
