"""Several host threads, each with its own handle, whose launches of the same
kernels need different amounts of shared memory: every call succeeds and every
pass gives the same bits as the thread's first."""
import random
import threading

import numpy as np
import pytest

import tmfqsfullstate_b200 as tq

pytestmark = pytest.mark.gpu


def circuit(n, count, seed):
    r, ops = random.Random(seed), []
    for _ in range(count):
        a, b = r.sample(range(n), 2)
        ops.append([tq.h(a), tq.h(b), tq.cphase(a, b, r.uniform(-3, 3)), tq.cnot(a, b), tq.x(a), tq.swap(a, b)][r.randrange(6)])
    return ops


def wide(k, seed):
    q, _ = np.linalg.qr(np.random.default_rng(seed).standard_normal((1 << k, 1 << k)))
    return tq.gate(q.astype(complex), list(range(k)))


BATCHES = {
    "circuits": lambda k: (13, circuit(13, 20 + 50 * k, k)),
    "circuit sizes": lambda k: (9 + 2 * k, circuit(9 + 2 * k, 60, k)),
    "qft sizes": lambda k: (12 + k, tq.qft_ops(12 + k)),
    "wide gates": lambda k: (13, [wide(3 + 2 * k, k)]),
}


@pytest.mark.parametrize("batch", list(BATCHES))
@pytest.mark.parametrize("form", ["f64", "f64fast", "c64"])
def test_threads_with_their_own_handles(batch, form):
    errors = []

    def work(k):
        try:
            n, ops = BATCHES[batch](k)
            with tq.GpuState(tq.FP32 if form == "c64" else tq.FP64) as g:
                g.set_option(tq.OPT_EXACT, int(form == "f64"))
                amps, first = tq.random_phase(n, k), None
                for _ in range(500):
                    g.load(n, amps)
                    g.apply_ops(ops)
                    got = np.asarray(g.export()).view(np.float64).copy()
                    first = got if first is None else first
                    assert np.array_equal(first, got)
        except Exception as e:  # noqa: BLE001 (reported by the test's thread)
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
