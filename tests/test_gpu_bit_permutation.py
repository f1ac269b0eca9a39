"""Swap runs long enough for a bit permutation: every amplitude ends where the
swapped qubits put it, byte for byte, for pairs inside the low bits, between low
and high bits, among the high bits only, and states from one tile to several
waves of tiles."""
import numpy as np
import pytest

import oracle as O
import tmfqsfullstate_b200 as tq

pytestmark = pytest.mark.gpu


def pairs_of(kind, n, seed):
    if kind == "reversal":
        return [(i, n - 1 - i) for i in range(n // 2)]
    if kind == "neighbours":
        return [(i, i + 1) for i in range(0, n - 1, 2)]
    if kind == "halves":
        return [(i, i + n // 2) for i in range(n // 2)]
    if kind == "high":  # qubit 0 is the highest index bit
        return [(i, 7 - i) for i in range(4)]
    p = np.random.default_rng(seed).permutation(n)
    return [(int(p[2 * i]), int(p[2 * i + 1])) for i in range(max(4, n // 2 - seed % 3))]


@pytest.mark.parametrize("prec", [tq.FP64, tq.FP32])
@pytest.mark.parametrize("n", [9, 12, 17, 20, 23])
@pytest.mark.parametrize("kind", ["reversal", "neighbours", "halves", "high", "random"])
def test_swap_run_moves_amplitudes(kind, n, prec):
    for seed in range(3 if kind == "random" else 1):
        pairs = pairs_of(kind, n, seed)
        amps = np.random.default_rng(n).standard_normal((1 << n, 2)).astype(np.float32).astype(np.float64)
        want = amps.reshape((2,) * n + (2,))
        for a, b in pairs:
            want = np.swapaxes(want, a, b)
        with tq.GpuState(prec) as g:
            g.load(n, amps)
            g.apply_ops([tq.swap(a, b) for a, b in pairs])
            out = np.asarray(g.export())
        out = np.ascontiguousarray(out).view(np.float64).reshape(1 << n, 2)
        assert np.ascontiguousarray(want).reshape(1 << n, 2).tobytes() == out.tobytes()


@pytest.mark.parametrize("form", ["f64", "f64fast", "c64"])
@pytest.mark.parametrize("n,fq", [(5, 0), (9, 0), (11, 0), (12, 0), (13, 0), (13, 5), (14, 3), (16, 7)])
@pytest.mark.parametrize("swaps", [1, 2, 3, 5])
def test_swap_runs_between_passes(swaps, n, fq, form):
    """Swap runs alone, after, before and between Hadamards and phases, or after a CNOT, on tiles narrower than a full one:
    in the pass or a permutation of their own."""
    rng = np.random.default_rng(100 * n + swaps)
    perm = [int(v) for v in rng.permutation(n)]
    run = [("swap", perm[2 * i], perm[2 * i + 1]) for i in range(min(swaps, n // 2))]
    hs = [("h", int(q)) for q in rng.permutation(n)[:3]] + [("cphase", perm[0], perm[1], 0.7)]
    amps = rng.standard_normal(2 << n)
    amps /= np.linalg.norm(amps)
    for ops in (run, hs + run, run + hs, hs + run + hs, hs + [("cnot", perm[1], perm[2])] + run, run + run[::-1] + hs):
        want = O.OracleRegister(n, amps=amps)
        want.run([getattr(O, k)(*a) for k, *a in ops])
        with tq.GpuState(tq.FP32 if form == "c64" else tq.FP64) as g:
            g.set_option(tq.OPT_EXACT, int(form == "f64"))
            if fq:
                g.set_option(tq.OPT_FUSED_QUBITS, fq)
            g.load(n, amps)
            g.apply_ops([getattr(tq, k)(*a) for k, *a in ops])
            got = g.export()
        if form == "f64":
            assert np.array_equal(got, want.amplitudes())
        else:  # a Hadamard or phase rounds by a few eps of the norm
            assert O.rel_l2(want.amplitudes(), got) <= 4 * len(ops) * 2.0 ** -(24 if form == "c64" else 53)
