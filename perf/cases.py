"""Workloads of the ring-Ising engine, for timing it and for comparing its results.

``listed()`` names the calls that stand for the framework's use, ``draw(rng)``
takes one more from the same ranges, ``prepare`` builds what a caller holds
before the call (an engine handle and its angles), ``run`` makes one call
through the public entry points, ``exact`` evaluates the same quantities with
plain torch in complex128, and ``work`` counts what a call cannot do without.

Three kinds of case:
  * ``circuit``: energy (and gradient) of one circuit of n qubits and L layers,
    through the device entry point, the drop-in host wrapper, the autograd
    Function (forward and backward), or energy only;
  * ``batch``: a list of circuits of mixed or equal shape in one call;
  * ``mlp``: loss and gradient of the warm-start network on a full batch.
"""

import math

import numpy as np
import torch

from gpu_simulation_b200 import BatchEngine, Engine, RingIsingAdjointBackend, StandaloneBackendConfig
from gpu_simulation_b200.autograd import ring_ising_energy
from gpu_simulation_b200.warmstart import WarmStartMLP

#: 2^n * n * L of the largest single circuit (n = 28, L = 4)
MOST_GATE_AMPLITUDES = (1 << 28) * 28 * 4
#: and of the largest batch (its sum over the circuits)
MOST_BATCH_AMPLITUDES = 4096 * 1_500_000


def circuit(name, entry, n, layers, field=1.0):
    return {"name": name, "kind": "circuit", "entry": entry, "n": n, "layers": layers, "field": field}


def listed():
    return [
        # the smallest call: a host-side optimiser loop over a toy circuit (8 qubits x 8 layers)
        circuit("dropin_n8_l8", "dropin", 8, 8),
        # one optimiser step's forward and backward of the n = 12, L = 3 Adam example
        circuit("autograd_n12_l3", "autograd", 12, 3),
        # a deep circuit that fits one tile: angles and results stay on the device
        circuit("device_n12_l8", "device", 12, 8),
        # a mid-size circuit through the drop-in wrapper, host arrays in and out
        circuit("dropin_n16_l4", "dropin", 16, 4),
        # the differentiation example: forward and backward at n = 20, L = 8
        circuit("autograd_n20_l8", "autograd", 20, 8),
        # an odd size and a depth between the benchmark's: energies only, as a line search asks for
        circuit("energy_n23_l6", "energy", 23, 6, 0.7),
        # the large-circuit sweep: n = 24, L = 4
        circuit("device_n24_l4", "device", 24, 4),
        # a large and deep circuit of odd size, out of L2
        circuit("device_n25_l7", "device", 25, 7, 1.3),
        # the headline: n = 28, L = 4
        circuit("device_n28_l4", "device", 28, 4),
        # 4096 circuits of mixed shape in one launch
        {"name": "batch_4096_mixed", "kind": "batch", "count": 4096, "n_min": 6, "n_max": 16, "l_min": 1, "l_max": 16,
         "shapes": 7},
        # one VQE step of the warm-start evaluation: 128 fields of the n = 16, L = 6 family
        {"name": "batch_128_n16_l6", "kind": "batch", "count": 128, "n_min": 16, "n_max": 16, "l_min": 6, "l_max": 6,
         "shapes": 8},
        # one full-batch training gradient of the warm-start network on 512 rows (float32)
        {"name": "mlp_512", "kind": "mlp", "rows": 512, "outputs": 192},
    ]


def log_uniform(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    kind = rng.random()
    if kind < 0.1:
        return {"kind": "mlp", "rows": log_uniform(rng, 32, 1024), "outputs": 2 * rng.randint(8, 20) * rng.randint(2, 8)}
    if kind < 0.3:
        while True:
            n_min, l_min = rng.randint(4, 16), log_uniform(rng, 1, 16)
            c = {"kind": "batch", "count": log_uniform(rng, 16, 4096), "n_min": n_min, "n_max": rng.randint(n_min, 16),
                 "l_min": l_min, "l_max": rng.randint(l_min, 16), "shapes": rng.randrange(1 << 16)}
            # the mean of 2^n n over the range, times the mean depth and the count
            span = range(c["n_min"], c["n_max"] + 1)
            mean = sum((1 << n) * n for n in span) / len(span)
            if c["count"] * mean * (c["l_min"] + c["l_max"]) / 2 <= MOST_BATCH_AMPLITUDES:
                return c
    while True:
        n, layers = rng.randint(4, 28), log_uniform(rng, 1, 16)
        if (1 << n) * n * layers <= MOST_GATE_AMPLITUDES:
            return {"kind": "circuit", "entry": rng.choice(["device", "dropin", "autograd", "energy"]), "n": n,
                    "layers": layers, "field": round(rng.uniform(0.2, 2.0), 3)}


def angles(count, seed):
    """Seeded angles U[0, 2 pi) on the GPU, the start of every VQE run here."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(count, dtype=torch.float64, device="cuda", generator=g) * (2.0 * math.pi)


def batch_shapes(case):
    """Qubits, layers and field of every circuit; they belong to the case, the angles to the seed."""
    rng = np.random.default_rng(case["shapes"])
    return (rng.integers(case["n_min"], case["n_max"] + 1, case["count"]).astype(np.int32),
            rng.integers(case["l_min"], case["l_max"] + 1, case["count"]).astype(np.int32),
            rng.uniform(0.2, 2.0, case["count"]))


def mlp_inputs(case, seed):
    """Rows (h, n / 16, L / 16), target angles as the warm start trains on, and packed weights
    (He-scaled normals, small biases)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    rows = case["rows"]
    x = torch.empty(rows, 3, device="cuda")
    x[:, 0] = 0.2 + 1.8 * torch.rand(rows, device="cuda", generator=g)
    x[:, 1] = 1.0
    x[:, 2] = 6.0 / 16.0
    target = math.pi * (2.0 * torch.rand(rows, case["outputs"], device="cuda", generator=g) - 1.0)
    parts, widths = [], (3, 256, 256, case["outputs"])
    for k, m in zip(widths, widths[1:]):
        parts += [torch.randn(m * k, device="cuda", generator=g) * math.sqrt(2.0 / k),
                  0.1 * torch.randn(m, device="cuda", generator=g)]
    return x, target, widths, torch.cat(parts)


def prepare(case, seed):
    if case["kind"] == "mlp":
        x, target, widths, weights = mlp_inputs(case, seed)
        net = WarmStartMLP(widths)
        net.weights.copy_(weights)
        return {"case": case, "net": net, "x": x, "target": target}
    if case["kind"] == "batch":
        engine = BatchEngine(max_qubits=case["n_max"])
        engine.set_circuits(*batch_shapes(case))
        p = angles(engine.num_params, seed)
        return {"case": case, "engine": engine, "p": p,
                "energy": torch.empty(case["count"], dtype=torch.float64, device="cuda"), "grad": torch.empty_like(p)}
    n, layers, field = case["n"], case["layers"], case["field"]
    p = angles(2 * n * layers, seed)
    if case["entry"] == "dropin":
        backend = RingIsingAdjointBackend(StandaloneBackendConfig(n, layers, field, "structured_adjoint"))
        return {"case": case, "backend": backend, "p": p.cpu().numpy().reshape(layers, n, 2)}
    engine = Engine(n, layers, field)
    if case["entry"] == "autograd":
        return {"case": case, "engine": engine, "p": p.reshape(layers, n, 2).requires_grad_()}
    return {"case": case, "engine": engine, "p": p, "energy": torch.empty(1, dtype=torch.float64, device="cuda"),
            "grad": torch.empty_like(p)}


def run(state):
    case = state["case"]
    if case["kind"] == "mlp":
        loss, grad = state["net"].gradient(state["x"], state["target"])
        return {"loss": loss, "grad": grad}
    if case["kind"] == "batch":
        state["engine"].run_device(state["p"], state["energy"], state["grad"])
        return {"energy": state["energy"], "grad": state["grad"]}
    if case["entry"] == "dropin":
        energy, grad = state["backend"].energy_and_grad(state["p"])
        return {"energy": energy, "grad": grad.reshape(-1)}
    if case["entry"] == "autograd":
        energy = ring_ising_energy(state["p"], state["engine"])
        (grad,) = torch.autograd.grad(energy, state["p"])
        return {"energy": energy.detach(), "grad": grad.reshape(-1)}
    if case["entry"] == "energy":
        state["engine"].energy_and_grad_device(state["p"], state["energy"])
        return {"energy": state["energy"]}
    state["engine"].energy_and_grad_device(state["p"], state["energy"], state["grad"])
    return {"energy": state["energy"], "grad": state["grad"]}


def circuit_flops(n, layers, grad):
    """An L-layer circuit is summed exactly either over its 2^n amplitudes, layer
    by layer, or along the ring over the 2^(L-1) values that its CNOTs carry
    from wire to wire (twice for bra and ket, twice for the ring's two ends):
    the cheaper of the two."""
    amplitudes = (1 << (n - 1)) * n * layers * (104 if grad else 28) + (1 << n) * (2 * n + 8)
    ring = n * 16 ** (layers - 1) * max(1, 2 * (layers - 1)) * 40 * (3 if grad else 1)
    return float(min(amplitudes, ring))


def work(case):
    if case["kind"] == "mlp":
        sizes = [3 * 256, 256 * 256, 256 * case["outputs"]]
        weights = sum(sizes) + 512 + case["outputs"]
        return {"bytes": 4.0 * (2 * weights + case["rows"] * (3 + case["outputs"])),
                "flops": 2.0 * case["rows"] * (3 * sum(sizes) - sizes[0])}
    if case["kind"] == "batch":
        ns, ls, _ = batch_shapes(case)
        return {"bytes": float(sum(8 * (4 * int(n) * int(l) + 2) for n, l in zip(ns, ls))),
                "flops": sum(circuit_flops(int(n), int(l), True) for n, l in zip(ns, ls))}
    n, layers, grad = case["n"], case["layers"], case["entry"] != "energy"
    return {"bytes": 8.0 * (2 * n * layers * (2 if grad else 1) + 1), "flops": circuit_flops(n, layers, grad)}


# ---------------------------------------------------------------------------
# The same quantities with plain torch in 64 bits: circuits of one shape at
# once, state [count, 2^n], bit w of the index is wire w.
# ---------------------------------------------------------------------------


def wire(state, w):
    return state.view(state.shape[0], -1, 2, 1 << w)


def column(v):
    return v.view(-1, 1, 1)


def apply_ry(state, w, theta):
    c, s = column(torch.cos(theta / 2)), column(torch.sin(theta / 2))
    v = wire(state, w)
    a, b = v[:, :, 0].clone(), v[:, :, 1]
    v[:, :, 0].mul_(c).sub_(s * b)
    v[:, :, 1].mul_(c).add_(s * a)


def apply_rz(state, w, phi):
    v = wire(state, w)
    z = column(torch.polar(torch.ones_like(phi), phi / 2))
    v[:, :, 0].mul_(z.conj())
    v[:, :, 1].mul_(z)


def apply_cnot(state, control, target):
    lo, hi = min(control, target), max(control, target)
    v = state.view(state.shape[0], -1, 2, 1 << (hi - lo - 1), 2, 1 << lo)
    one = v[:, :, 1] if control == hi else v[:, :, :, :, 1]
    axis = 3 if control == hi else 2  # the other wire's axis in what is left
    a, b = one.select(axis, 0), one.select(axis, 1)
    keep = a.clone()
    a.copy_(b)
    b.copy_(keep)


def inner(a, b):
    """Re <a|b> per circuit."""
    return torch.sum(a.real * b.real + a.imag * b.imag, dim=tuple(range(1, a.dim())))


def hamiltonian(psi, n, fields):
    index = torch.arange(1 << n, device=psi.device)
    walls = torch.zeros(1 << n, dtype=torch.float64, device=psi.device)
    for w in range(n):
        walls += ((index >> w) ^ (index >> ((w + 1) % n))) & 1
    lam = psi * (2.0 * walls - n)
    del index, walls
    for w in range(n):
        out, v = wire(lam, w), wire(psi, w)
        out[:, :, 0].sub_(fields.view(-1, 1, 1) * v[:, :, 1])
        out[:, :, 1].sub_(fields.view(-1, 1, 1) * v[:, :, 0])
    return lam


def exact_circuits(n, layers, fields, p, grad):
    """Energies [count] and gradients [count, layers, n, 2] for angles p of that shape."""
    psi = torch.zeros(p.shape[0], 1 << n, dtype=torch.complex128, device=p.device)
    psi[:, 0] = 1.0
    for l in range(layers):
        for w in range(n):
            apply_ry(psi, w, p[:, l, w, 0])
            apply_rz(psi, w, p[:, l, w, 1])
        for w in range(n):
            apply_cnot(psi, w, (w + 1) % n)
    lam = hamiltonian(psi, n, fields)
    energy = inner(lam, psi)
    if not grad:
        return energy, None
    g = torch.empty_like(p)
    for l in reversed(range(layers)):
        for w in reversed(range(n)):
            apply_cnot(psi, w, (w + 1) % n)
            apply_cnot(lam, w, (w + 1) % n)
        for w in reversed(range(n)):
            a, b = wire(lam, w), wire(psi, w)
            # RZ = exp(-i phi Z / 2): dE/dphi = Im <lam|Z|psi>; RY likewise with Y
            g[:, l, w, 1] = inner(a[:, :, 0], -1j * b[:, :, 0]) + inner(a[:, :, 1], 1j * b[:, :, 1])
            apply_rz(psi, w, -p[:, l, w, 1])
            apply_rz(lam, w, -p[:, l, w, 1])
            g[:, l, w, 0] = inner(a[:, :, 1], b[:, :, 0]) - inner(a[:, :, 0], b[:, :, 1])
            apply_ry(psi, w, -p[:, l, w, 0])
            apply_ry(lam, w, -p[:, l, w, 0])
    return energy, g


def exact_mlp(case, seed):
    x, target, widths, packed = mlp_inputs(case, seed)
    target, packed = target.double(), packed.double().requires_grad_()
    at, y = 0, x.double()
    for l in range(1, len(widths)):
        k, m = widths[l - 1], widths[l]
        w, b = packed[at:at + m * k].view(m, k), packed[at + m * k:at + m * k + m]
        at += m * k + m
        y = y @ w.T + b
        if l + 1 < len(widths):
            y = torch.nn.functional.gelu(y)
    loss = torch.mean((y - target) ** 2)
    (grad,) = torch.autograd.grad(loss, packed)
    return {"loss": loss.detach().reshape(1), "grad": grad}


def exact(case, seed):
    if case["kind"] == "mlp":
        return exact_mlp(case, seed)
    if case["kind"] == "batch":
        ns, ls, hs = batch_shapes(case)
        sizes = 2 * ns.astype(np.int64) * ls
        offsets = np.concatenate([[0], np.cumsum(sizes)])
        p = angles(int(offsets[-1]), seed)
        energy, grad = torch.empty(len(ns), dtype=torch.float64, device="cuda"), torch.empty_like(p)
        for n, layers in sorted(set(zip(ns.tolist(), ls.tolist()))):
            at = np.flatnonzero((ns == n) & (ls == layers))
            where = torch.from_numpy(offsets[at][:, None] + np.arange(2 * n * layers)).cuda()
            e, g = exact_circuits(n, layers, torch.from_numpy(hs[at]).cuda(), p[where].view(len(at), layers, n, 2), True)
            energy[torch.from_numpy(at).cuda()] = e
            grad[where] = g.view(len(at), -1)
        return {"energy": energy, "grad": grad}
    n, layers = case["n"], case["layers"]
    p = angles(2 * n * layers, seed).view(1, layers, n, 2)
    fields = torch.full((1,), case["field"], dtype=torch.float64, device="cuda")
    energy, grad = exact_circuits(n, layers, fields, p, case["entry"] != "energy")
    if case["entry"] == "dropin":
        return {"energy": float(energy), "grad": grad.reshape(-1).cpu().numpy()}
    if case["entry"] == "autograd":
        return {"energy": energy.reshape(()), "grad": grad.reshape(-1)}
    return {"energy": energy} if grad is None else {"energy": energy, "grad": grad.reshape(-1)}
