"""QFT passes of three and more register stages run as two blocks per SM with one
tile buffer each where the tiles keep both busy (from 592 tiles: 23 qubits of
complex64, 22 of complex128), else as one block with a ring of buffers.  Both
sides of that line, with two, three and four stages, a last stage in the
copy-out or not, and Hadamards only, against the exact complex128 form.

Tolerances: fast FP64 relative L2 <= 1e-12, complex64 <= 1e-5 (an operation adds
at most a few eps of the norm, and there are at most 91 of them)."""
import numpy as np
import pytest

import tmfqsfullstate_b200 as tq

pytestmark = pytest.mark.gpu

TOL = {tq.FP64: 1e-12, tq.FP32: 1e-5}


def ops_of(kind, n, bits):
    ops = []
    for t in range(n - bits, n):
        ops.append(tq.h(t))
        if kind == "qft":
            ops += [tq.cphase(c, t, np.pi / float(1 << (c - t))) for c in range(t + 1, n)]
    return ops


@pytest.mark.parametrize("prec", [tq.FP64, tq.FP32])
@pytest.mark.parametrize("n", [21, 22, 23, 24])
@pytest.mark.parametrize("kind,bits", [("qft", 8), ("qft", 10), ("qft", 11), ("qft", 12), ("qft", 13), ("walsh", 12)])
def test_pass_block_shapes(kind, bits, n, prec):
    amps = np.random.default_rng(n).standard_normal((1 << n, 2))
    amps = (amps / np.linalg.norm(amps)).astype(np.float32).astype(np.float64)
    ops = ops_of(kind, n, bits)
    res = []
    for p, exact in ((tq.FP64, 1), (prec, 0)):
        with tq.GpuState(p) as g:
            g.set_option(tq.OPT_EXACT, exact)
            g.load(n, amps)
            g.apply_ops(ops)
            res.append(np.asarray(g.export()).view(np.float64).ravel())
            if not exact:
                assert g.stats()["qft_passes"] >= 1
    assert np.linalg.norm(res[1] - res[0]) <= TOL[prec] * np.linalg.norm(res[0])


@pytest.mark.parametrize("n", [22, 29])
def test_factor_rows_of_two_block_passes(n):
    """Fast complex128 QFTs one of whose two-block passes multiplies by factors of the tile's outer bits (the first at 22
    qubits, the second at 29): against the exact form, and the same bits in every repetition."""
    import torch

    gen = torch.Generator(device="cuda:0")
    gen.manual_seed(n)
    amps = torch.randn(2 << n, generator=gen, device="cuda:0", dtype=torch.float64)
    amps /= torch.linalg.vector_norm(amps)
    ops = tq.qft_ops(n)

    def run(g, exact):
        g.set_option(tq.OPT_EXACT, exact)
        g.init_zero(n)
        g.tensor().copy_(amps)
        torch.cuda.synchronize()
        g.apply_ops(ops)

    with tq.GpuState(tq.FP64) as exact, tq.GpuState(tq.FP64) as first, tq.GpuState(tq.FP64) as again:
        run(exact, 1)
        run(first, 0)
        assert first.stats()["qft_passes"] >= 2
        assert exact.compare(first)["rel_l2"] <= TOL[tq.FP64]
        for _ in range(20 if n < 25 else 4):
            run(again, 0)
            assert first.compare(again)["bitwise_equal"]
