"""Rounding of circuits whose rotations are pushed through two-qubit gates from run to run, against long
double.  Each run of U3s adds an independent error; a thousand runs on two qubits, averaged over 64
vectors, show its size to a few per cent.

Bound per run: what the kernel that applied the gates as given in FP64 left on these circuits, 1.22e-16 of
the amplitudes' norm for one U3 per run and 2.01e-16 for two, and 5 %.  Chains with their numbers in FP64
left 1.53e-16 and 2.24e-16.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

RUNS, BATCH = 1000, 64


def u3(t):
    """(batch, 2, 2) in long double from (batch, 3) stored angles."""
    t = t.astype(np.longdouble)
    c, s = np.cos(t[:, 0]), np.sin(t[:, 0])
    f, l = [np.cos(t[:, k]) + 1j * np.sin(t[:, k]) for k in (1, 2)]
    return np.stack([c + 0j, -l * s, f * s, f * l * c], -1).reshape(-1, 2, 2)


def errors(sqg, two_qubit, members):
    """Norm of the error of each vector's 4 x 4 matrix, relative and per square root of a run."""
    c = sqg.Circuit(2)
    for _ in range(RUNS):
        for _ in range(members):
            c.add_U3(0)
        {"CNOT": c.add_CNOT, "CZ": c.add_CZ}[two_qubit](0, 1)
    p = np.random.default_rng(members).uniform(0, 2 * np.pi, (BATCH, RUNS * members, 3))
    m = torch.eye(4, dtype=torch.complex128, device="cuda").repeat(BATCH, 1, 1)
    c.apply_to_device(torch.from_numpy(p.reshape(BATCH, -1)).cuda(), m)
    A = np.broadcast_to(np.eye(4), (BATCH, 4, 4)).astype(np.clongdouble)
    for k in range(RUNS):
        for j in range(members):
            A = (u3(p[:, k * members + j])[:, None] @ A.reshape(BATCH, 2, 2, 4)).reshape(BATCH, 4, 4)
        A = A[:, [0, 1, 3, 2]] if two_qubit == "CNOT" else A * np.array([1, 1, 1, -1]).reshape(4, 1)
    d = m.cpu().numpy() - A
    return np.sqrt(np.sum(np.abs(d.reshape(BATCH, -1)) ** 2, axis=1).astype(np.float64) / 4.0 / RUNS)


@pytest.mark.parametrize("members", [1, 2])
@pytest.mark.parametrize("two_qubit", ["CNOT", "CZ"])
def test_error_per_run(sqg, two_qubit, members):
    e = np.sqrt(np.mean(errors(sqg, two_qubit, members) ** 2))
    print("%s, %d per run: %.3g" % (two_qubit, members, e))
    assert e <= 1.05 * {1: 1.22e-16, 2: 2.01e-16}[members]
