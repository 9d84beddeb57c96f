"""CZs that no operation meets for long: they wait in the plan, cancel in pairs, and go their own way when too
many wait.  Values against the oracle (1e-12 relative to max(1, |reference|), at most 600 gates); the host's
time for the plan grows with the circuit and not with its square."""
import importlib
import time

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def close(a, b):
    a, b = np.asarray(a), np.asarray(b)
    assert np.max(np.abs(a - b)) <= 1e-12 * max(1.0, np.max(np.abs(b)))


def circuit(sqg, n, kind, rng):
    c = sqg.Circuit(n)
    pair = lambda lo=0: [int(q) for q in lo + rng.choice(n - lo, 2, replace=False)]
    for q in range(n):
        c.add_RY(q)
    if kind == "pairs":  # every CZ an even or odd number of times
        for _ in range(300):
            c.add_CZ(*pair())
        c.add_U3(0)
    elif kind == "far":  # rotations on a qubit that no CZ touches
        for _ in range(150):
            c.add_CZ(*pair(2))
            c.add_RX(0)
            c.add_CRY(0, 1)
    else:  # CNOTs make all rows differ: more than wait at once
        for _ in range(250):
            c.add_CZ(*pair(1))
            c.add_CNOT(*pair(1))
        c.add_U3(0)
    for q in range(n):
        c.add_RX(q)
    return c


@pytest.mark.parametrize("kind", ["pairs", "far", "rows"])
@pytest.mark.parametrize("n", [4, 6, 10])
def test_waiting_czs(sqg, n, kind):
    rng = np.random.default_rng(n)
    c = circuit(sqg, n, kind, rng)
    recs, P, N = c.gate_records(), c.get_Parameter_Num(), 1 << n
    p = rng.uniform(0, 2 * np.pi, P)
    cols = min(N, 40)
    T = np.linalg.qr(rng.standard_normal((N, cols)) + 1j * rng.standard_normal((N, cols)))[0].copy()
    want = O.apply_to(n, recs, p, T.copy())
    A = T.copy()
    c.apply_to(p, A)
    close(A, want)
    v = torch.from_numpy(T[:, 0].copy()).cuda()
    c.apply_state_device(torch.from_numpy(p).cuda(), v)
    close(v.cpu().numpy(), want[:, 0])
    th = torch.from_numpy(p).cuda()
    ev = sqg.CostEvaluator(c, T)
    rc, rg = O.cost_grad_sweep(n, recs, p, T)
    for step in (0, 7):
        cost, grad = ev.cost_grad(th, checkpoint_interval=step)
        close(cost.item(), rc)
        close(grad[0].cpu().numpy(), rg)


def test_plan_time_grows_with_the_circuit(sqg):
    circ = importlib.import_module("sequential-quantum-gate-decomposer_gb300.circuit")

    def seconds(pairs):
        c = sqg.Circuit(12)
        for k in range(pairs):
            c.add_CZ(2 + k % 7, 9 + k % 3)
            c.add_RX(0)
            c.add_CRY(0, 1)
        recs = c.gate_records()
        best = np.inf
        for _ in range(3):
            t = time.perf_counter()
            circ.NativeCircuit(12, recs)
            best = min(best, time.perf_counter() - t)
        return best

    seconds(100)
    assert seconds(24000) <= 9.0 * seconds(6000)  # four times as long, sixteen times its square
