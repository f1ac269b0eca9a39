"""The exact sequential sums at the sizes and inputs where the tiled replay can
go wrong: tile, group and direct-walk edges, sums that hover at a power of two
(both candidate binades of every tile in play), terms half-way between grid
points, sign changes, zeros, and values that leave the normal range.  The
reference is numpy's cumsum, a left-to-right double sum: every value and index
must be identical."""
import numpy as np
import pytest

import tmfqsfullstate_b200 as tq

pytestmark = pytest.mark.gpu

SIZES = [1, 6, 11, 12, 13, 14, 15, 17, 18, 20]


def state(kind, n, seed=0):
    rng = np.random.default_rng(1000 * n + seed)
    N = 1 << n
    a = np.zeros((N, 2))
    if kind == "random":
        a = rng.standard_normal((N, 2)) / np.sqrt(2 * N)
    elif kind == "uniform":
        a[:, 0] = 2.0 ** (-n / 2)
    elif kind == "halves":  # the running sum sits just below 1/2, then just above
        a[:, 0] = 1e-9
        a[N // 7, 1] = np.sqrt(0.5) * (1 - 1e-12)
        a[N // 2, 1] = 1e-4
    elif kind == "ties":  # |a|^2 = odd multiples of 2^-54 after a first 1: half-way on the grid of [1, 2)
        a[:, 0] = 2.0 ** -27 * np.sqrt(rng.integers(0, 2, N) * 8 + 1)
        a[0, 0] = 1.0
    elif kind == "sparse":
        i = rng.integers(0, N, max(1, N // 997))
        a[i] = rng.standard_normal((len(i), 2))
    elif kind == "growing":  # a binade crossing every few terms
        a[:, 0] = 2.0 ** (np.arange(N) / max(1, N // 200) / 2 - 60)
    elif kind == "tiny":  # squares that are subnormal or zero
        a = rng.standard_normal((N, 2)) * 1e-160
    elif kind == "huge":
        a = rng.standard_normal((N, 2)) * 1e120
        a[N // 2] = 1e153
    return a


def terms(a):
    return a[:, 0] * a[:, 0] + a[:, 1] * a[:, 1]


@pytest.mark.parametrize("kind", ["random", "uniform", "halves", "ties", "sparse", "growing", "huge"])
@pytest.mark.parametrize("n", SIZES)
def test_total_and_draws(kind, n):
    a = state(kind, n)
    cdf = np.cumsum(terms(a))
    with tq.GpuState(tq.FP64) as g:
        g.load(n, a.reshape(-1))
        assert g.total_probability() == cdf[-1]
        at = [0, (1 << n) // 3, (1 << n) // 2, (1 << n) - 1]
        draws = [0.0, 0.25, 0.5, 0.9999] + [v for i in at for v in (cdf[i], np.nextafter(cdf[i], 0), np.nextafter(cdf[i], 2))]
        for r in draws:
            if not 0.0 <= r < 1.0:
                continue
            want = int(np.argmax(r <= cdf)) if (r <= cdf).any() else None
            if want is None:
                with pytest.raises(tq.RuntimeFailure):
                    g.sample(float(r))
            else:
                assert g.sample(float(r)) == want, (kind, n, r)


@pytest.mark.parametrize("kind", ["random", "uniform", "halves", "sparse", "growing", "huge"])
@pytest.mark.parametrize("n", SIZES)
def test_amplitude_sums(kind, n):
    a = state(kind, n, 1)
    if kind == "growing":  # alternating signs: the sum changes sign and binade all the time
        a[::3, 0] *= -1.0
    a[:, 1] = a[::-1, 0]
    with tq.GpuState(tq.FP64) as g:
        g.load(n, a.reshape(-1))
        assert g.amplitude_sum() == (np.cumsum(a[:, 0])[-1], np.cumsum(a[:, 1])[-1])


@pytest.mark.parametrize("n", [5, 14, 16])
def test_subnormal_and_nonfinite(n):
    a = state("tiny", n)
    with tq.GpuState(tq.FP64) as g:
        g.load(n, a.reshape(-1))
        assert g.total_probability() == np.cumsum(terms(a))[-1]
        for bad in (np.inf, np.nan):
            b = state("random", n)
            b[(1 << n) * 2 // 3, 0] = bad
            g.load(n, b.reshape(-1))
            with np.errstate(invalid="ignore"):
                want = np.cumsum(terms(b))[-1]
                re = np.cumsum(b[:, 0])[-1]
            assert np.array_equal(g.total_probability(), want, equal_nan=True)
            assert np.array_equal(g.amplitude_sum()[0], re, equal_nan=True)
            assert g.sample(0.25) == int(np.argmax(0.25 <= np.cumsum(terms(b))))


@pytest.mark.parametrize("n", [9, 13, 16, 18])
def test_complex64_and_overlay(n):
    """complex64 terms (short mantissas: many half-way terms) and the overlay branches."""
    a = state("random", n, 2).astype(np.float32)
    d = a.astype(np.float64)
    scale, bias = (-1.0, 0.0), (2.0 ** (-n / 2) * 1.25, 0.0)
    with tq.GpuState(tq.FP32) as g:
        g.load(n, d.reshape(-1))
        cdf = np.cumsum(terms(d))
        assert g.total_probability() == cdf[-1]
        assert g.sample(0.7) == int(np.argmax(0.7 <= cdf))
        re = (scale[0] * d[:, 0] - scale[1] * d[:, 1]) + bias[0]
        im = (scale[0] * d[:, 1] + scale[1] * d[:, 0]) + bias[1]
        cdf = np.cumsum(terms(np.stack([re, im], 1)))
        assert g.overlay_total_probability(scale, bias) == cdf[-1]
        assert g.overlay_sample(scale, bias, 0.3) == int(np.argmax(0.3 <= cdf))
        assert g.overlay_sum(scale, bias) == (np.cumsum(re)[-1], np.cumsum(im)[-1])


@pytest.mark.parametrize("n,marked", [(22, 1), (23, 2)])
def test_search_result_at_a_power_of_two(n, marked):
    """After these searches 1 - P is 2e-11: the running sum stays next to 1/2 and 1 for most of the register."""
    N = 1 << n
    states = [N // 5, N // 2][:marked]
    a = np.full((N, 2), 0.0)
    a[:, 0] = np.sqrt(2.04e-11 / N)
    a[states, 0] = np.sqrt((1 - 2.04e-11) / marked)
    cdf = np.cumsum(terms(a))
    with tq.GpuState(tq.FP64) as g:
        g.load(n, a.reshape(-1))
        assert g.total_probability() == cdf[-1]
        for r in (0.1, 0.49, 0.7, 1 - 3e-12):
            if r <= cdf[-1]:
                assert g.sample(r) == int(np.argmax(r <= cdf))


@pytest.mark.parametrize("n", [11, 14, 15, 17, 22])
@pytest.mark.parametrize("kind", ["all", "zeros", "mixed"])
def test_nan_is_never_lost(n, kind):
    """All NaN, one NaN in an otherwise zero tile of a basis state, one NaN among terms of both signs: the total and the
    sums are NaN, and a draw finds its index only among the terms before the NaN."""
    N = 1 << n
    rng = np.random.default_rng(n)
    for at in ((0,) if kind == "all" else (N // 3, N - 7)):
        for part in (0, 1):
            a = np.zeros((N, 2))
            if kind == "all":
                a[:, part] = np.nan
            elif kind == "zeros":
                a[N // 2, 0] = 1.0
                a[at, part] = np.nan
            else:
                a = (1.0 + 2.0 * rng.standard_normal((N, 2))) / np.sqrt(10.0 * N)
                a[at, part] = np.nan
            with np.errstate(invalid="ignore"):
                cdf, sums = np.cumsum(terms(a)), np.cumsum(a, axis=0)[-1]
                hit = 0.25 <= cdf
            assert np.isnan(cdf[-1])
            with tq.GpuState(tq.FP64) as g:
                g.load(n, a.reshape(-1))
                assert np.isnan(g.total_probability())
                assert np.array_equal(g.amplitude_sum(), sums, equal_nan=True)
                if hit.any():
                    assert g.sample(0.25) == int(np.argmax(hit))
                else:
                    with pytest.raises(tq.RuntimeFailure):
                        g.sample(0.25)


@pytest.mark.parametrize("n", [9, 12, 13, 15, 18])
@pytest.mark.parametrize("share", [0.002, 0.02, 0.2, 0.5])
def test_terms_added_one_by_one(n, share):
    """Sums that the steps over whole tiles do not carry: signed ones that hover around zero with a few or many terms that
    are not zero (windows of 32 with none, some and all of them), totals whose binade doubles every 4 to 40 terms or that
    stay below the normal range, and draws that end inside such a run."""
    N = 1 << n
    rng = np.random.default_rng(n)
    a = rng.standard_normal((N, 2)) * (rng.random((N, 2)) < share)
    a[rng.random((N, 2)) < 0.01] = -0.0
    grow = np.zeros((N, 2))
    grow[:, 0] = 2.0 ** (((np.arange(N) % 4000) / (8.0 / share) - 480.0) / 2) * (rng.random(N) < 0.9)
    tiny = rng.standard_normal((N, 2)) * 1e-153 * (rng.random((N, 2)) < share)
    for b in (a, grow, tiny):
        cdf = np.cumsum(terms(b))
        with tq.GpuState(tq.FP64) as g:
            g.load(n, b.reshape(-1))
            assert g.total_probability() == cdf[-1]
            assert g.amplitude_sum() == (np.cumsum(b[:, 0])[-1], np.cumsum(b[:, 1])[-1])
            for i in (0, 5, N // 3, N // 2 + 17, N - 1):
                for r in (cdf[i], np.nextafter(cdf[i], 0), np.nextafter(cdf[i], 2)):
                    if 0.0 <= r < 1.0 and r <= cdf[-1]:
                        assert g.sample(float(r)) == int(np.argmax(r <= cdf))
