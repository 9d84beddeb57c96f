"""Workloads of this package as a user's program runs them, for timing and comparing builds.

Every case goes through a public entry point: cost and gradient of parameter batches
(CostEvaluator, RaggedBatch), the circuit applied to matrices and state vectors
(Circuit.apply_to_device / apply_state_device) and decompositions on the device
(BatchedDecomposer, bfgs_decompose_graph).  Sizes come from the package's benchmark, tests and
workload definitions, with ragged and odd ones between them.
"""
import importlib
import random

import numpy as np
import torch

sqg = importlib.import_module("sequential-quantum-gate-decomposer_gb300")
ragged = importlib.import_module("sequential-quantum-gate-decomposer_gb300.ragged")
batched = importlib.import_module("sequential-quantum-gate-decomposer_gb300.batched")

DEV = "cuda"
TWO_PI = 2.0 * np.pi


# ---- circuits as plain gate lists: (name, target, control) -------------------------------------
def nn_ansatz(n, blocks):
    """U3 on every qubit, then blocks of [CNOT(c, t), U3(c), U3(t)] over the ordered
    nearest-neighbour pairs: the ansatz of the decomposition benchmarks."""
    pairs = []
    for q in range(n - 1):
        pairs += [(q, q + 1), (q + 1, q)]
    gates = [("U3", q, -1) for q in range(n)]
    for k in range(blocks):
        c, t = pairs[k % len(pairs)]
        gates += [("CNOT", t, c), ("U3", c, -1), ("U3", t, -1)]
    return gates


def any_pair_ansatz(n, blocks, rng):
    """The same blocks over uniformly drawn ordered pairs (imported circuits)."""
    gates = [("U3", q, -1) for q in range(n)]
    for _ in range(blocks):
        c, t = rng.sample(range(n), 2)
        gates += [("CNOT", t, c), ("U3", c, -1), ("U3", t, -1)]
    return gates


def random_gates(n, count, rng, names):
    """`count` gates drawn uniformly from `names` on uniform qubits."""
    gates = []
    for _ in range(count):
        name = rng.choice(names)
        if name in ("CNOT", "CZ", "CRY"):
            c, t = rng.sample(range(n), 2)
            gates.append((name, t, c))
        else:
            gates.append((name, rng.randrange(n), -1))
    return gates


def simulation_circuit(n, levels):
    """SQUANDER's state-vector simulation benchmark: sweeps over all pairs c < t of
    [U3(t), U3(c), CRY(t, c)], then a U3 on qubit 0."""
    gates = []
    for _ in range(levels):
        for c in range(n - 1):
            for t in range(c + 1, n):
                gates += [("U3", t, -1), ("U3", c, -1), ("CRY", t, c)]
    return gates + [("U3", 0, -1)]


FIVE = ("U3", "RY", "CNOT", "CZ", "CRY")
SEVEN = ("U3", "RX", "RY", "RZ", "CNOT", "CZ", "CRY")
PARAMS = {"U3": 3, "RX": 1, "RY": 1, "RZ": 1, "CRY": 1, "CNOT": 0, "CZ": 0}


def gate_list(case):
    rng = random.Random(case.get("structure", 0))
    n, kind = case["n"], case["circuit"]
    if kind == "nn":
        return nn_ansatz(n, case["blocks"])
    if kind == "pairs":
        return any_pair_ansatz(n, case["blocks"], rng)
    if kind == "sim":
        return simulation_circuit(n, case["levels"])
    return random_gates(n, case["gates"], rng, FIVE if kind == "five" else SEVEN)


def param_num(gates):
    return sum(PARAMS[g[0]] for g in gates)


def make_circuit(n, gates):
    c = sqg.Circuit(n)
    for name, t, ctl in gates:
        if ctl >= 0:
            getattr(c, "add_" + name)(t, ctl)
        else:
            getattr(c, "add_" + name)(t)
    return c


# ---- inputs ------------------------------------------------------------------------------------
def generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def haar(n, gen, count=None):
    N = 1 << n
    shape = (N, N) if count is None else (count, N, N)
    a = torch.complex(torch.randn(shape, generator=gen, device=DEV, dtype=torch.float64),
                      torch.randn(shape, generator=gen, device=DEV, dtype=torch.float64))
    q, r = torch.linalg.qr(a)
    d = torch.diagonal(r, dim1=-2, dim2=-1)
    return (q * (d / d.abs()).unsqueeze(-2)).contiguous()


def angles(shape, gen):
    return torch.rand(shape, generator=gen, device=DEV, dtype=torch.float64) * TWO_PI


def eval_inputs(case, seed):
    gen = generator(seed)
    n, B = case["n"], case["batch"]
    gates = gate_list(case)
    cols, off = case.get("cols", 1 << n), case.get("offset", 0)
    u = haar(n, gen, B if case.get("own_targets") else None)
    target = u[..., :, off:off + cols].contiguous()
    return gates, target, angles((B, param_num(gates)), gen)


def state_inputs(case, seed):
    """Parameters and either B states of 2^n amplitudes or B matrices of 2^n x cols."""
    gen = generator(seed)
    n, B, cols = case["n"], case["batch"], case.get("cols", 1)
    gates = gate_list(case)
    theta = angles((B, param_num(gates)), gen)
    shape = (B, 1 << n) if case["what"] == "state" else (B, 1 << n, cols)
    v = torch.randn(shape + (2,), generator=gen, device=DEV, dtype=torch.float64)
    v /= v.square().sum(dim=(1, -1), keepdim=True).sqrt()
    return gates, theta, torch.view_as_complex(v)


def ragged_inputs(case, seed):
    """`count` instances, qubit counts cycling over 3..n, the nearest-neighbour ansatz of
    3 n (n - 1) / 2 blocks each."""
    gen = generator(seed)
    rng = random.Random(case["structure"])
    out = []
    for i in range(case["count"]):
        n = 3 + rng.randrange(case["n"] - 2)
        gates = nn_ansatz(n, 3 * n * (n - 1) // 2)
        out.append((n, gates, haar(n, gen), angles((1, param_num(gates)), gen)))
    return out


def decompose_inputs(case, seed):
    gen = generator(seed)
    n, B = case["n"], case["batch"]
    gates = nn_ansatz(n, case["blocks"])
    u = haar(n, gen, B)
    return gates, u, angles((B, param_num(gates)), gen)


# ---- the cases ---------------------------------------------------------------------------------
def listed():
    return [
        # one evaluation handed to a host optimizer: the smallest call, latency and launches
        dict(name="grad_n3_one", what="grad", circuit="nn", n=3, blocks=14, batch=1),
        # one evaluation per target of a batch of four-qubit targets (P = 252)
        dict(name="grad_n4_batch", what="grad", circuit="nn", n=4, blocks=40, batch=1024, own_targets=True),
        # a six-qubit decomposition on the device within a budget of evaluations
        dict(name="loop_n6_bfgs", what="loop", circuit="nn", n=6, blocks=20, calls=40),
        # state preparation and isometries: a narrow, ragged block of columns, every gate kind,
        # the Hilbert-Schmidt cost
        dict(name="grad_n7_narrow", what="grad", circuit="seven", n=7, gates=300, structure=7, batch=5, cols=50,
             variant=3),
        # the eight-qubit ansatz of 360 blocks (P = 2184) over a batch of parameter vectors
        dict(name="grad_n8_batch", what="grad", circuit="nn", n=8, blocks=360, batch=128),
        # ten qubits, arbitrary pairs (P = 1830)
        dict(name="grad_n10", what="grad", circuit="pairs", n=10, blocks=300, structure=12, batch=6),
        # cost only: line searches and population optimizers
        dict(name="cost_n8_batch", what="cost", circuit="nn", n=8, blocks=120, batch=200),
        # the largest benchmark matrix: 2000 gates of five kinds on 4096 x 4096
        dict(name="apply_n12", what="apply", circuit="five", n=12, gates=2000, structure=5, batch=1, cols=4096),
        # state-vector simulation, the largest benchmark register
        dict(name="state_n24", what="state", circuit="sim", n=24, levels=1, batch=1),
        # an ordinary register, a few states at once
        dict(name="state_n15_batch", what="state", circuit="seven", n=15, gates=400, structure=15, batch=7),
        # many circuits of different registers in one launch
        dict(name="ragged_3to8", what="ragged", n=8, count=60, structure=3),
        # multi-start screening: 3-qubit BFGS decompositions within a budget of evaluations
        dict(name="decompose_n3", what="decompose", n=3, blocks=14, batch=4096, calls=24),
    ]


def spread(rng, lo, hi):
    """An integer of lo..hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    what = rng.choice(("grad", "grad", "grad", "grad_small", "cost", "apply", "state", "ragged", "decompose", "loop"))
    if what == "grad_small":
        n = rng.randint(2, 5)
        return dict(what="grad", circuit="nn", n=n, blocks=spread(rng, 4, 50), batch=spread(rng, 1, 3000),
                    own_targets=rng.random() < 0.5, variant=rng.choice((0, 0, 0, 3, 9)))
    if what in ("grad", "cost"):
        n = rng.randint(6, 10)
        kind = rng.choice(("nn", "pairs", "five", "seven"))
        cols = rng.choice((1 << n, 1 << n, 1 << n, rng.randint(1, (1 << n) - 1)))
        c = dict(what=what, circuit=kind, n=n, structure=rng.randrange(1000), cols=cols,
                 variant=rng.choice((0, 0, 0, 3, 9)))
        if cols < (1 << n) and c["variant"] == 0:
            c["offset"] = rng.randint(0, (1 << n) - cols)
        if kind in ("nn", "pairs"):
            c["blocks"] = spread(rng, 5, 300)
            work = 2 * c["blocks"]
        else:
            c["gates"] = spread(rng, 10, 900)
            work = c["gates"]
        most = int(720 * 128 * 65536 / (work * cols * (1 << n)))  # the eight-qubit case's work
        c["batch"] = spread(rng, 1, max(1, min(400, most)))
        return c
    if what == "apply":
        n = rng.randint(5, 12)
        return dict(what="apply", circuit=rng.choice(("nn", "five", "seven")), n=n, structure=rng.randrange(1000),
                    blocks=spread(rng, 5, 300), gates=spread(rng, 20, 1500), batch=rng.randint(1, 3) if n > 10 else rng.randint(1, 20),
                    cols=rng.randint(1 << (n - 1), 1 << n) if n < 11 else rng.randint(500, 1400))
    if what == "state":
        n = rng.randint(8, 23)
        kind = rng.choice(("five", "seven", "pairs"))
        return dict(what="state", circuit=kind, n=n, structure=rng.randrange(1000), blocks=spread(rng, 10, 150),
                    gates=spread(rng, 20, 500), batch=rng.randint(1, 9) if n < 20 else 1)
    if what == "ragged":
        return dict(what="ragged", n=rng.randint(5, 8), count=spread(rng, 3, 60), structure=rng.randrange(1000))
    if what == "loop":
        n = rng.randint(4, 7)
        return dict(what="loop", circuit="nn", n=n, blocks=rng.randint(5, 25), calls=rng.randint(10, 40))
    n = rng.randint(2, 5)
    return dict(what="decompose", n=n, blocks=rng.randint(3, 14), batch=spread(rng, 10, 4096 >> (2 * max(0, n - 3))),
                calls=rng.randint(8, 24))


class State:
    pass


def prepare(case, seed):
    s, what = State(), case["what"]
    s.case = case
    if what in ("grad", "cost"):
        gates, target, s.theta = eval_inputs(case, seed)
        s.evaluator = sqg.CostEvaluator(make_circuit(case["n"], gates), target, trace_offset=case.get("offset", 0),
                                        cost_variant=case.get("variant", 0))
    elif what in ("apply", "state"):
        gates, s.theta, s.v = state_inputs(case, seed)
        s.circuit = make_circuit(case["n"], gates)
        s.circuit.native()
    elif what == "ragged":
        inst = ragged_inputs(case, seed)
        s.batch = ragged.RaggedBatch([make_circuit(n, g) for n, g, _, _ in inst], [u.cpu().numpy() for _, _, u, _ in inst])
        s.theta = torch.cat([t.reshape(-1) for _, _, _, t in inst])
    else:
        gates, s.targets, s.x0 = decompose_inputs(case if what == "decompose" else dict(case, batch=1), seed)
        s.circuit = make_circuit(case["n"], gates)
        s.circuit.native()
        if what == "decompose":
            s.decomposer = sqg.BatchedDecomposer(s.circuit, tolerance=1e-8, max_calls=case["calls"], max_outer=1)
    return s


def run(s):
    case = s.case
    what = case["what"]
    if what == "grad":
        return s.evaluator.cost_grad(s.theta)
    if what == "cost":
        return s.evaluator.cost_grad(s.theta, with_grad=False)[0]
    if what == "apply":
        return s.circuit.apply_to_device(s.theta, s.v)
    if what == "state":
        return s.circuit.apply_state_device(s.theta, s.v)
    if what == "ragged":
        return s.batch.cost_grad(s.theta)
    if what == "decompose":
        return s.decomposer.run(s.targets, s.x0, seed=1)
    return batched.bfgs_decompose_graph(s.circuit, s.targets[0], s.x0[0], max_calls=case["calls"], max_outer=1)


# ---- what a pass cannot do without -------------------------------------------------------------
# Real operations per complex pair: U3 28 (14 multiply-adds), one-parameter rotations 16 (CRY on
# half of the pairs), CNOT and CZ none.
FLOPS = {"U3": 28, "RX": 16, "RY": 16, "RZ": 16, "CRY": 8, "CNOT": 0, "CZ": 0}


def sweep_flops(gates, n, cols):
    return sum(FLOPS[g[0]] for g in gates) * (1 << n) / 2 * cols


def work(case):
    what, n = case["what"], case["n"]
    if what == "ragged":
        rng = random.Random(case["structure"])
        total = {"bytes": 0.0, "flops": 0.0}
        for _ in range(case["count"]):
            m = 3 + rng.randrange(n - 2)
            one = work(dict(what="grad", circuit="nn", n=m, blocks=3 * m * (m - 1) // 2, batch=1))
            total = {k: total[k] + one[k] for k in total}
        return total
    gates = gate_list(dict(case, circuit=case.get("circuit", "nn")))
    P, B = param_num(gates), case.get("batch", 1)
    cols = case.get("cols", 1 << n)
    if what == "state":
        return {"bytes": 32.0 * B * (1 << n), "flops": B * sweep_flops(gates, n, 1)}
    if what == "apply":
        return {"bytes": 32.0 * B * (1 << n) * cols, "flops": B * sweep_flops(gates, n, cols)}
    targets = B if (case.get("own_targets") or what == "decompose") else 1
    sweeps = 1 if what == "cost" else 3
    evals = case["calls"] if what in ("decompose", "loop") else 1
    return {"bytes": 16.0 * targets * (1 << n) * cols + 8.0 * B * (2 * P + 1),
            "flops": evals * B * sweeps * sweep_flops(gates, n, cols)}


# ---- the same results from plain torch in 64 bits ----------------------------------------------
def matrices(name, p):
    """(B, 2, 2) matrix of a gate and the list of its derivatives for stored parameters p (B, k)."""
    def mat(a, b, c, d):
        e = torch.stack([x.to(torch.complex128) for x in (a, b, c, d)], dim=-1)
        return e.reshape(-1, 2, 2)

    s, c = torch.sin(p[:, 0]), torch.cos(p[:, 0])
    z = torch.zeros_like(s)
    if name == "U3":
        ep, el = torch.exp(1j * p[:, 1]), torch.exp(1j * p[:, 2])
        return (mat(c, -el * s, ep * s, ep * el * c),
                [mat(-s, -el * c, ep * c, -ep * el * s), mat(z, z, 1j * ep * s, 1j * ep * el * c),
                 mat(z, -1j * el * s, z, 1j * ep * el * c)])
    if name == "RX":
        return mat(c, -1j * s, -1j * s, c), [mat(-s, -1j * c, -1j * c, -s)]
    if name == "RZ":
        return mat(c - 1j * s, z, z, c + 1j * s), [mat(-s - 1j * c, z, z, -s + 1j * c)]
    return mat(c, -s, s, c), [mat(-s, -c, c, -s)]


def halves(v, n, t, ctl):
    """Views of v (B, 2^n, m) with the target bit 0 and 1 (control bit 1 where there is one)."""
    B, m = v.shape[0], v.shape[2]
    if ctl < 0:
        w = v.view(B, 1 << (n - 1 - t), 2, (1 << t) * m)
        return w[:, :, 0], w[:, :, 1]
    lo, hi = min(t, ctl), max(t, ctl)
    w = v.view(B, 1 << (n - 1 - hi), 2, 1 << (hi - lo - 1), 2, (1 << lo) * m)
    if ctl == hi:
        return w[:, :, 1, :, 0], w[:, :, 1, :, 1]
    return w[:, :, 0, :, 1], w[:, :, 1, :, 1]


def apply_gate(v, n, name, t, ctl, g):
    x, y = halves(v, n, t, ctl)
    if name == "CNOT":
        x0 = x.clone()
        x.copy_(y)
        y.copy_(x0)
    elif name == "CZ":
        y.neg_()
    else:
        g = g.reshape((-1, 2, 2) + (1,) * (x.dim() - 1))
        nx = g[:, 0, 0] * x + g[:, 0, 1] * y
        ny = g[:, 1, 0] * x + g[:, 1, 1] * y
        x.copy_(nx)
        y.copy_(ny)


def exact_state(case, seed):
    gates, theta, v = state_inputs(case, seed)
    n = case["n"]
    w = v.reshape(v.shape[0], 1 << n, -1).clone()
    k = 0
    for name, t, ctl in gates:
        np_ = PARAMS[name]
        apply_gate(w, n, name, t, ctl, matrices(name, theta[:, k:k + np_])[0] if np_ else None)
        k += np_
    return w.reshape(v.shape)


def exact_eval(n, gates, target, theta, off=0, variant=0, grad=True):
    B, P = theta.shape
    cols = target.shape[-1]
    psi = target.expand(B, 1 << n, cols).clone()
    mats, k = [], 0
    for name, t, ctl in gates:
        np_ = PARAMS[name]
        g, d = matrices(name, theta[:, k:k + np_]) if np_ else (None, [])
        mats.append((g, d, k))
        k += np_
        apply_gate(psi, n, name, t, ctl, g)
    tr = torch.diagonal(psi[:, off:off + cols], dim1=1, dim2=2).sum(1)
    N = float(cols)
    cost = (1 - tr.real / N if variant == 0 else 1 - tr.abs().square() / N ** 2 if variant == 3 else
            1 - (tr.abs().square() / N + 1) / (N + 1))
    if not grad:
        return cost
    lam = torch.zeros_like(psi)
    j = torch.arange(cols, device=psi.device)
    lam[:, j + off, j] = 1
    dt = torch.zeros((B, P), dtype=torch.complex128, device=psi.device)
    for (name, t, ctl), (g, d, k) in zip(reversed(gates), reversed(mats)):
        gd = g.conj().transpose(1, 2) if g is not None else None
        apply_gate(psi, n, name, t, ctl, gd)
        if d:
            px, lx = halves(psi, n, t, ctl), halves(lam, n, t, ctl)
            for q, m in enumerate(d):
                for a in range(2):
                    for b in range(2):
                        o = (lx[a].conj() * px[b]).flatten(1).sum(1)
                        dt[:, k + q] += m[:, a, b] * o
        apply_gate(lam, n, name, t, ctl, gd)
    if variant == 0:
        return cost, -dt.real / N
    scale = -2.0 / N ** 2 if variant == 3 else -2.0 / N / (N + 1)
    return cost, scale * (tr.conj().reshape(-1, 1) * dt).real


def exact(case, seed):
    what = case["what"]
    if what in ("apply", "state"):
        return exact_state(case, seed)
    if what in ("grad", "cost"):
        gates, target, theta = eval_inputs(case, seed)
        return exact_eval(case["n"], gates, target, theta, case.get("offset", 0), case.get("variant", 0), what == "grad")
    if what == "ragged":
        both = [exact_eval(n, g, u, t) for n, g, u, t in ragged_inputs(case, seed)]
        return torch.cat([c for c, _ in both]), torch.cat([g.reshape(-1) for _, g in both])
    return None  # a trajectory of an optimizer
