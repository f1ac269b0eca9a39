"""The workloads whose speed is tracked: what programs do with a GpuState.

Each case is a dict of plain values; `listed()` names the standing ones and
`draw()` gives others of the same ranges.  `prepare` makes the state, inputs
and op list that a program holds before the call, `run` makes one pass through
the public entry points, `work` counts the bytes and operations that the pass
cannot do without, and `exact` gives the same outputs in 64 bits from plain
torch and numpy.

Kinds:
  qft      one QFT of a register that is resident on the GPU
  circuit  a circuit of H, X, CNOT, controlled phases and swaps
  dense    a brickwork of two-qubit unitaries with a few wider ones between
  grover   a whole search: basis state, Hadamard layer, iterations, total
           probability and one measurement
  adjoint  expectation and gradient of the layered controlled-phase circuit
  measure  total probability and one measurement of a resident register
  call     the small end-to-end call: host input, QFT, total probability,
           measurement, host output

Forms: f64 (complex128, bit-identical to the sequential reference), f64fast
(complex128 with OPT_EXACT off), c64 (complex64).
"""
import math
import random

import numpy as np
import torch

import tmfqsfullstate_b200 as tq

DEV = "cuda:0"


def listed():
    return [
        # A small register through the whole call, as the qftG command does it: latency and launch count.
        {"name": "call_f64_n12", "kind": "call", "form": "f64", "n": 12},
        # The headline benchmark: QFT-28 on a random-phase input, the form that matches the reference bit for bit.
        {"name": "qft_f64_n28", "kind": "qft", "form": "f64", "n": 28},
        # The same circuit in complex128 without the bit-for-bit order of operations.
        {"name": "qft_f64fast_n27", "kind": "qft", "form": "f64fast", "n": 27},
        # The large complex64 QFT (8 GiB state).
        {"name": "qft_c64_n30", "kind": "qft", "form": "c64", "n": 30},
        # Mixed circuits of an odd and an even register size, no QFT structure in them.
        {"name": "circuit_f64_n23", "kind": "circuit", "form": "f64", "n": 23, "ops": 120},
        {"name": "circuit_c64_n26", "kind": "circuit", "form": "c64", "n": 26, "ops": 160},
        # Variational circuits of dense gates.
        {"name": "dense_f64_n24", "kind": "dense", "form": "f64", "n": 24, "layers": 1, "wide": 3},
        {"name": "dense_c64_n27", "kind": "dense", "form": "c64", "n": 27, "layers": 2, "wide": 3},
        # Grover-20 with materialised diffusion (the reference's own example) and the lazy form with four marked states.
        {"name": "grover_f64_n20", "kind": "grover", "form": "f64", "n": 20, "marked": 1, "lazy": False},
        {"name": "grover_lazy_f64_n26", "kind": "grover", "form": "f64", "n": 26, "marked": 4, "lazy": True},
        # The gradient benchmark: 24 qubits, 20 layers, 480 angles, checkpoints every 48 operations.
        {"name": "adjoint_c64_n24", "kind": "adjoint", "form": "c64", "n": 24, "layers": 20, "every": 48},
        # What follows a simulation: the norm check and a draw.
        {"name": "measure_f64_n28", "kind": "measure", "form": "f64", "n": 28},
    ]


def draw(rng):
    kind = rng.choice(["call", "qft", "qft", "circuit", "circuit", "dense", "dense", "grover", "grover", "adjoint", "measure"])
    if kind == "call":
        return {"kind": kind, "form": rng.choice(["f64", "f64", "c64"]), "n": rng.randint(8, 18)}
    if kind == "qft":
        form = rng.choice(["f64", "f64fast", "c64"])
        return {"kind": kind, "form": form, "n": rng.randint(16, {"f64": 28, "f64fast": 29, "c64": 30}[form])}
    if kind == "circuit":
        form = rng.choice(["f64", "f64fast", "c64"])
        return {"kind": kind, "form": form, "n": rng.randint(14, 24 if form == "f64" else 26), "ops": rng.randint(40, 160)}
    if kind == "dense":
        form = rng.choice(["f64", "c64"])
        return {"kind": kind, "form": form, "n": rng.randint(14, 24 if form == "f64" else 27), "layers": rng.randint(1, 2),
                "wide": rng.randint(0, 3)}
    if kind == "grover":
        lazy = rng.random() < 0.5
        form = rng.choice(["f64", "f64", "f64fast", "c64"])
        top = 21 if form == "f64" and not lazy else 25
        return {"kind": kind, "form": form, "n": rng.randint(14, top), "marked": rng.randint(1, 6), "lazy": lazy}
    if kind == "adjoint":
        form = rng.choice(["c64", "c64", "f64fast"])
        return {"kind": kind, "form": form, "n": rng.randint(14, 24 if form == "c64" else 22), "layers": rng.randint(3, 20),
                "every": rng.choice([24, 48, 96])}
    form = rng.choice(["f64", "f64", "c64"])
    return {"kind": "measure", "form": form, "n": rng.randint(16, 28 if form == "f64" else 29)}


# ---- inputs ----------------------------------------------------------------

def _real(case):
    return torch.float32 if case["form"] == "c64" else torch.float64


def _amplitudes(case, seed):
    """The register's input on the GPU, interleaved: random phases of equal
    weight (qft, call) or a random state (the others)."""
    n = case["n"]
    if case["kind"] == "call":
        ph = torch.from_numpy(np.random.default_rng(seed).random(1 << n)) * (2.0 * math.pi)
    else:
        gen = torch.Generator(device=DEV)
        gen.manual_seed(seed)
        if case["kind"] != "qft":
            a = torch.randn(2 << n, generator=gen, device=DEV, dtype=_real(case))
            return a.div_(torch.linalg.vector_norm(a, dtype=torch.float64).to(a.dtype))
        ph = torch.rand(1 << n, generator=gen, device=DEV, dtype=_real(case)).mul_(2.0 * math.pi)
    out = torch.empty(2 << n, dtype=ph.dtype, device=ph.device)
    torch.cos(ph, out=out[0::2])
    torch.sin(ph, out=out[1::2])
    return out.mul_(2.0 ** (-n / 2))


def _unitary(rng, dim):
    z = rng.standard_normal((dim, dim)) + 1j * rng.standard_normal((dim, dim))
    q, r = np.linalg.qr(z)
    d = np.diag(r)
    return q * (d / np.abs(d))


def _gates(case, seed):
    """The circuit as plain tuples: ("h", q), ("cp", c, t, theta), ("u", matrix, qubits), ..."""
    n, rng = case["n"], random.Random(seed)
    if case["kind"] == "circuit":
        out = []
        for _ in range(case["ops"]):
            a, b = rng.sample(range(n), 2)
            k = rng.choices(["h", "cp", "cnot", "x", "swap"], [30, 30, 20, 10, 10])[0]
            out.append(("h", a) if k == "h" else ("x", a) if k == "x" else ("cp", a, b, rng.uniform(0.0, 2.0 * math.pi))
                       if k == "cp" else (k, a, b))
        return out
    npr = np.random.default_rng(seed)
    out = []
    for layer in range(case["layers"]):
        for first in (0, 1):
            out += [("u", _unitary(npr, 4), (q, q + 1)) for q in range(first, n - 1, 2)]
    for _ in range(case["wide"]):
        k = rng.randint(3, 6)
        out.insert(rng.randint(0, len(out)), ("u", _unitary(npr, 1 << k), tuple(rng.sample(range(n), k))))
    return out


def _ops(gates):
    make = {"h": tq.h, "x": tq.x, "cp": tq.cphase, "cnot": tq.cnot, "swap": tq.swap, "u": tq.gate}
    return [make[g[0]](*g[1:]) for g in gates]


def _draw_of(seed):
    return random.Random(seed + 77).random()


def _marked(case, seed):
    return sorted(random.Random(seed).sample(range(1 << case["n"]), case["marked"]))


def _iterations(case):
    return int(math.pi / 4.0 * math.sqrt((1 << case["n"]) / case["marked"]))


def _angles(case, seed):
    return np.random.default_rng(seed).random((case["layers"], case["n"])) * (2.0 * math.pi)


def prepare(case, seed):
    n, kind = case["n"], case["kind"]
    g = tq.GpuState(tq.FP32 if case["form"] == "c64" else tq.FP64, 0)
    if case["form"] == "f64fast":
        g.set_option(tq.OPT_EXACT, 0)
    s = {"case": case, "g": g, "rnd": _draw_of(seed)}
    if kind == "call":
        s["input"] = torch.empty(2 << n, dtype=torch.float64, pin_memory=True).copy_(_amplitudes(case, seed)).numpy()
        s["output"] = torch.empty(2 << n, dtype=torch.float64, pin_memory=True).numpy()
        s["ops"] = tq.qft_ops(n)
        return s
    g.init_zero(n)
    s["state"] = g.tensor()  # the register's own buffer: it lives as long as the handle does
    s["state"].owner = g
    if kind == "grover":
        s["ops"] = [tq.h(q) for q in range(n)]
        s["marked"] = _marked(case, seed)
        return s
    if kind == "adjoint":
        s["ops"] = tq.layered_cphase_ops(n, _angles(case, seed))
        s["masks"], s["weights"] = tq.zz_ring_observable(n)
        return s
    s["state"].copy_(_amplitudes(case, seed))
    torch.cuda.synchronize()
    if kind != "measure":
        s["ops"] = tq.qft_ops(n) if kind == "qft" else _ops(_gates(case, seed))
    return s


def run(s):
    case, g = s["case"], s["g"]
    n, kind = case["n"], case["kind"]
    if kind == "call":
        g.load(n, s["input"])
        g.apply_ops(s["ops"])
        total = g.total_probability()
        index = g.sample(s["rnd"])
        return {"state": g.export(s["output"]), "total": total, "index": index}
    if kind == "grover":
        g.init_basis(n, 0)
        g.apply_ops(s["ops"])
        v = g.grover_run(tq.RegisterView.fresh(), s["marked"], _iterations(case), not case["lazy"])
        scale, bias = (v.scale_re, v.scale_im), (v.bias_re, v.bias_im)
        if v.overlay:
            total, index = g.overlay_total_probability(scale, bias), g.overlay_sample(scale, bias, s["rnd"])
        else:
            total, index = g.total_probability(), g.sample(s["rnd"])
        return {"state": s["state"], "total": total, "index": index, "overlay": [*scale, *bias], "sum": v.sum_re}
    if kind == "adjoint":
        g.init_basis(n, 0)
        e, grads = g.adjoint_gradient(s["ops"], s["masks"], s["weights"], case["every"])
        return {"state": s["state"], "expectation": e, "gradient": grads}
    if kind == "measure":
        return {"total": g.total_probability(), "index": g.sample(s["rnd"])}
    g.apply_ops(s["ops"])
    return {"state": s["state"]}


# ---- what a pass cannot do without ------------------------------------------

def work(case):
    n, kind = case["n"], case["kind"]
    N = float(1 << n)
    amp = 8.0 if case["form"] == "c64" else 16.0
    if kind == "call":  # host input and output, both complex128
        return {"bytes": 2.0 * N * 16.0, "flops": 5.0 * N * n + 4.0 * N}
    if kind == "qft":
        return {"bytes": 2.0 * N * amp, "flops": 5.0 * N * n}
    if kind == "circuit":  # 4 a Hadamard, 6 for a quarter of the amplitudes a controlled phase
        return {"bytes": 2.0 * N * amp, "flops": case["ops"] * N * (0.3 * 4.0 + 0.3 * 1.5)}
    if kind == "dense":
        gates = case["layers"] * (n - 1)
        return {"bytes": 2.0 * N * amp, "flops": N * 8.0 * (gates * 4.0 + case["wide"] * 20.0)}
    if kind == "grover":  # the state written once and read once by the measurement
        each = 0.0 if case["lazy"] or case["form"] != "f64" else 2.0
        return {"bytes": 2.0 * N * amp, "flops": N * (4.0 + each * _iterations(case))}
    if kind == "adjoint":  # forward and backward; a quarter of the state in each derivative
        per_layer = n * 4.0 + n * 1.5
        return {"bytes": 2.0 * N * amp, "flops": N * case["layers"] * (3.0 * per_layer + n * 1.0)}
    return {"bytes": N * amp, "flops": 4.0 * N}


# ---- the same in 64 bits -----------------------------------------------------

def _bits(a, n, *qubits):
    """`a` (2^n) viewed with one axis of 2 for each of the qubits (ascending) and the rest between them."""
    shape, last = [], -1
    for q in qubits:
        shape += [1 << (q - last - 1), 2]
        last = q
    return a.view(*shape, 1 << (n - 1 - last))


def _apply(a, n, g):
    """One gate of _gates() on a complex128 vector, which is overwritten."""
    k = g[0]
    if k in ("h", "x"):
        v = _bits(a, n, g[1])
        x, y = v[:, 0].clone(), v[:, 1].clone()
        v[:, 0], v[:, 1] = (y, x) if k == "x" else ((x + y) / math.sqrt(2.0), (x - y) / math.sqrt(2.0))
        return a
    if k == "u":
        m, qs = torch.from_numpy(g[1]).to(a.device), g[2]
        order = sorted(qs)
        v = _bits(a, n, *order)
        at = [2 * order.index(q) + 1 for q in qs]
        rest = [d for d in range(v.dim()) if d not in at]
        w = v.permute(*at, *rest)
        return (m @ w.reshape(1 << len(qs), -1)).view(w.shape).permute(*np.argsort(at + rest).tolist()).reshape(-1)
    lo, hi = sorted(g[1:3])
    v = _bits(a, n, lo, hi)
    if k == "cp":
        v[:, 1, :, 1].mul_(complex(math.cos(g[3]), math.sin(g[3])))
        return a
    if k == "swap":
        x, y = (0, 1), (1, 0)
    else:
        x, y = ((1, 0), (1, 1)) if g[1] < g[2] else ((0, 1), (1, 1))
    p, q = v[:, x[0], :, x[1]], v[:, y[0], :, y[1]]
    t = p.clone()
    p.copy_(q)
    q.copy_(t)
    return a


def _flat(a):
    return torch.view_as_real(a).reshape(-1)


def _adjoint_exact(case, seed):
    n, th = case["n"], _angles(case, seed)
    a = torch.zeros(1 << n, dtype=torch.complex128, device=DEV)
    a[0] = 1.0
    ring = [(q, (q + 1) % n) for q in range(n)]

    def hs(v):
        for q in range(n):
            _apply(v, n, ("h", q))

    for layer in th:
        hs(a)
        for (c, t), x in zip(ring, layer):
            _apply(a, n, ("cp", c, t, float(x)))
    hs(a)
    state = _flat(a.clone())
    index = torch.arange(1 << n, device=DEV)
    obs = torch.zeros(1 << n, dtype=torch.float64, device=DEV)
    for c, t in ring:
        obs += 1.0 - 2.0 * ((index >> (n - 1 - c) ^ index >> (n - 1 - t)) & 1).double()
    e = float((torch.view_as_real(a).square().sum(-1) * obs).sum())
    lam = a * obs
    grad = np.zeros_like(th)
    for l in range(len(th) - 1, -1, -1):
        hs(a)
        hs(lam)
        for j in range(n - 1, -1, -1):
            lo, hi = sorted(ring[j])
            x, y = (_bits(v, n, lo, hi)[:, 1, :, 1] for v in (lam, a))
            grad[l, j] = -2.0 * float((x.real * y.imag - x.imag * y.real).sum())
            back = complex(math.cos(th[l, j]), -math.sin(th[l, j]))
            x.mul_(back)
            y.mul_(back)
    return {"state": state, "expectation": e, "gradient": grad.reshape(-1)}


def _grover_exact(case, seed):
    n, marked = case["n"], _marked(case, seed)
    N, k = 1 << n, case["marked"]
    a0 = u = m = 1.0 / math.sqrt(N)  # an unmarked and a marked amplitude
    sign, bias = 1.0, 0.0
    for _ in range(_iterations(case)):
        mean = ((N - k) * u - k * m) / N
        u, m = 2.0 * mean - u, 2.0 * mean + m
        sign, bias = -sign, 2.0 * mean - bias
    out = torch.zeros(N, 2, dtype=torch.float64, device=DEV)
    lazy = case["lazy"]
    out[:, 0] = a0 if lazy else u
    out[torch.tensor(marked, device=DEV), 0] = (m - bias) / sign if lazy else m
    return {"state": out.view(-1), "total": (N - k) * u * u + k * m * m, "index": None,
            "overlay": [sign, 0.0, bias, 0.0] if lazy else [1.0, 0.0, 0.0, 0.0], "sum": (N - k) * u + k * m}


def exact(case, seed):
    n, kind = case["n"], case["kind"]
    if kind == "grover":
        return _grover_exact(case, seed)
    if kind == "adjoint":
        return _adjoint_exact(case, seed)
    a = torch.view_as_complex(_amplitudes(case, seed).to(DEV, torch.float64).view(-1, 2))
    if kind == "measure":
        return {"total": float(torch.view_as_real(a).square().sum()), "index": None}
    if kind in ("qft", "call"):
        a = torch.fft.ifft(a, norm="ortho")
        if kind == "call":
            return {"state": _flat(a).cpu(), "total": float(torch.view_as_real(a).square().sum()), "index": None}
        return {"state": _flat(a)}
    for g in _gates(case, seed):
        a = _apply(a, n, g)
    return {"state": _flat(a)}
