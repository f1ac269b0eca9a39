"""Swap runs long enough for a bit permutation: every amplitude ends where the
swapped qubits put it, byte for byte, for pairs inside the low bits, between low
and high bits, among the high bits only, and states from one tile to several
waves of tiles."""
import numpy as np
import pytest

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
