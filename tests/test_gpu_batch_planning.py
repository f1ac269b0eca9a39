"""Planning of long batches: the search for runs of operations within five
qubits that hold a dense gate takes time in proportion to the batch, and finds
the same blocks wherever such runs begin, overlap and end."""
import time

import numpy as np
import pytest

import oracle as O
import tmfqsfullstate_b200 as tq

pytestmark = pytest.mark.gpu


def unitary(d, seed):
    rng = np.random.default_rng(seed)
    q, _ = np.linalg.qr(rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d)))
    return q


def state(form):
    g = tq.GpuState(tq.FP32 if form == "c64" else tq.FP64)
    if form == "f64fast":
        g.set_option(tq.OPT_EXACT, 0)
    return g


@pytest.mark.parametrize("form", ["c64", "f64fast"])
def test_long_runs_on_few_qubits(form):
    """8000 operations on four qubits with two gates among them, between operations elsewhere (so that they are no block of
    their own): planned in about the time of the same batch without the gates."""
    n = 14
    u = unitary(4, 1)
    run = [tq.cphase(i % 4, (i + 1) % 4, 0.1 + i % 7) if i % 3 else tq.x(i % 4) for i in range(8000)]

    def batch(gates):
        ops = list(run)
        for i in gates:
            ops[i] = tq.gate(u, (1, 2))
        return [tq.h(9), tq.h(10)] + ops + [tq.h(11), tq.h(12)]

    def seconds(ops):
        with state(form) as g:
            g.init_basis(n, 5)
            g.apply_ops(ops)
            t = time.perf_counter()
            g.apply_ops(ops)
            g.sync()
            return time.perf_counter() - t

    plain, gates = seconds(batch(())), seconds(batch((3990, 7999)))
    assert gates <= 5 * plain + 0.2, (plain, gates)


@pytest.mark.parametrize("form", ["c64", "f64fast"])
@pytest.mark.parametrize("n,seed", [(14, 1), (14, 2), (15, 3), (16, 4), (9, 5)])
def test_runs_of_every_kind(form, n, seed):
    """Batches of clusters of operations on few qubits: gates of one to four qubits, swaps between, runs that a wide gate,
    a flip or the end of the batch cuts."""
    rng = np.random.default_rng(seed)
    make, ks = [], []
    for _ in range(25):
        pool = [int(v) for v in rng.permutation(n)[:int(rng.integers(2, 6))]]
        for _ in range(int(rng.integers(1, 9))):
            q = [int(v) for v in rng.permutation(pool)]
            k = int(rng.integers(1, min(4, len(pool)) + 1))
            t, kind = float(rng.uniform(-3, 3)), int(rng.integers(0, 8))
            u = unitary(1 << k, len(make))
            make.append([lambda M, q=q: M.h(q[0]), lambda M, q=q: M.x(q[0]), lambda M, q=q: M.cnot(q[0], q[1]),
                         lambda M, q=q, t=t: M.cphase(q[0], q[1], t), lambda M, q=q: M.swap(q[0], q[1]),
                         lambda M, q=q, k=k, u=u: M.gate(u, q[:k]), lambda M, q=q, k=k, u=u: M.gate(u, q[:k]),
                         lambda M, q=q: M.phase_flip(3)][kind])
            ks.append(k if kind in (5, 6) else 1)
    a = rng.standard_normal(2 << n)
    a /= np.linalg.norm(a)
    r = O.OracleRegister(n, amps=a)
    r.run([f(O) for f in make])
    with state(form) as g:
        g.load(n, a)
        g.apply_ops([f(tq) for f in make])
        got = g.export()
    eps = 2.0 ** -24 if form == "c64" else 2.0 ** -53
    # A dense gate's row sums: (2^(k+1) + 2) 2^(k/2) eps of the norm; a block is at most a gate of five qubits.
    assert O.rel_l2(r.amplitudes(), got) <= sum((2.0 ** (max(k, 2) + 1) + 2) * 2.0 ** (max(k, 2) / 2) for k in ks) * eps
