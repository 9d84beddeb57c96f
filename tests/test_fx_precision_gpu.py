"""Precision of the fixed-point sweeps against the oracle's FP64 gates as given, where the cosines that
the rotations leave out are smallest: angles at and near odd multiples of pi/4, as imported circuits
have them, through runs that are long enough for many of them to gather.

Tolerance 2e-15: some hundred operations of a rounding each leave 2^-53 sqrt(800) = 3e-15 of an
amplitude's size on the oracle's side, and gradients of these circuits are below 0.15; a sweep that
let sixteen such cosines gather was off by 2e-14 to 1e-12.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def circuit(sqg, n, blocks, rng, kind):
    c = sqg.Circuit(n)
    one, two = ("add_RY", "add_CZ") if kind == "ry" else ("add_U3", "add_CNOT")
    for q in range(n):
        getattr(c, one)(q)
    for _ in range(blocks):
        a, b = (int(q) for q in rng.choice(n, 2, replace=False))
        getattr(c, two)(a, b)
        getattr(c, one)(a)
        getattr(c, one)(b)
    return c


@pytest.mark.parametrize("kind", ["ry", "u3"])
@pytest.mark.parametrize("angle", ["pi/4", "near"])
@pytest.mark.parametrize("n,cols,blocks", [(6, 64, 120), (7, 3, 100), (8, 16, 240), (10, 64, 100), (12, 1, 70)])
def test_small_cosines(sqg, n, cols, blocks, angle, kind):
    rng = np.random.default_rng(n + blocks)
    c = circuit(sqg, n, blocks, rng, kind)
    P = c.get_Parameter_Num()
    p = rng.choice([1, 3, 5, 7], P) * (np.pi / 4)
    if angle == "near":
        p = p + 1e-3 * rng.standard_normal(P)
    N = 1 << n
    T = np.linalg.qr(rng.standard_normal((N, cols)) + 1j * rng.standard_normal((N, cols)))[0].copy()
    cost, grad = sqg.CostEvaluator(c, T).cost_grad(torch.from_numpy(p).cuda())
    rc, rg = O.cost_grad(n, c.gate_records(), p, T)
    assert np.max(np.abs(rg)) < 0.15
    assert abs(cost.item() - rc) <= 2e-15
    assert np.max(np.abs(grad[0].cpu().numpy() - rg)) <= 2e-15


@pytest.mark.parametrize("kind", ["ry", "u3"])
def test_deep_circuit_on_the_identity(sqg, kind):
    """A thousand runs on amplitudes that start as zeros and ones: what a product adds to a zero must not
    gather."""
    n = 8
    rng = np.random.default_rng(8)
    c = circuit(sqg, n, 500, rng, kind)
    P = c.get_Parameter_Num()
    p = rng.choice([1, 3, 5, 7], P) * (np.pi / 4) + 1e-3 * rng.standard_normal(P)
    T = np.eye(1 << n).astype(np.complex128)
    ev = sqg.CostEvaluator(c, T)
    cost, grad = ev.cost_grad(torch.from_numpy(p).cuda())
    cost64, grad64 = ev.cost_grad(torch.from_numpy(p).cuda(), checkpoint_interval=50)  # swept in FP64
    assert abs(cost.item() - cost64.item()) <= 2e-15
    assert torch.max(torch.abs(grad - grad64)).item() <= 2e-15
