"""Fixed-point sweeps of targets far from the size of a unitary, against the oracle: compared relative to
the largest reference value, which is asserted not to vanish, so that a wrong power of two shows.

Tolerance 1e-12 of that value, as for the engine's other parity tests.  Small targets are
compared through the Hilbert-Schmidt gradient, which keeps values of any size (the Frobenius one is 1 - x
- 1); below 2^-500 its square leaves the range of a double, and nothing that is returned depends on the
target any more.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def scaled(wl, n, cols, exponent):
    rng = np.random.default_rng(n * cols)
    c = wl.all_gates_circuit(n, 60, rng)
    T = rng.standard_normal((1 << n, cols)) + 1j * rng.standard_normal((1 << n, cols))
    T /= np.linalg.norm(T, axis=0)
    return c, rng.uniform(0, 2 * np.pi, c.get_Parameter_Num()), np.ldexp(T.real, exponent) + 1j * np.ldexp(T.imag, exponent)


@pytest.fixture(scope="module")
def wl():
    from importlib import import_module
    return import_module("sequential-quantum-gate-decomposer_gb300.workloads")


@pytest.mark.parametrize("cols", [1, 21, 64])
@pytest.mark.parametrize("exponent", [-480, -300, -62, -30])
def test_small_targets(sqg, wl, exponent, cols):
    c, p, T = scaled(wl, 6, cols, exponent)
    _, grad = sqg.CostEvaluator(c, T, cost_variant=3).cost_grad(torch.from_numpy(p).cuda())
    rg = O.cost_grad(6, c.gate_records(), p, T, variant=3)[1]
    assert np.max(np.abs(rg)) > 0.0
    assert np.max(np.abs(grad[0].cpu().numpy() - rg)) <= 1e-12 * np.max(np.abs(rg))


@pytest.mark.parametrize("cols", [1, 21, 64])
@pytest.mark.parametrize("exponent", [40, 500, 1000, 1018, 1021])
def test_large_targets(sqg, wl, exponent, cols):
    c, p, T = scaled(wl, 6, cols, exponent)
    ev = sqg.CostEvaluator(c, T)
    cost, grad = ev.cost_grad(torch.from_numpy(p).cuda())
    only = ev.cost_grad(torch.from_numpy(p).cuda(), with_grad=False)[0]
    rc, rg = O.cost_grad(6, c.gate_records(), p, T)
    assert np.all(np.isfinite(rg)) and np.max(np.abs(rg)) > 0.0
    assert abs(cost.item() - rc) <= 1e-12 * max(abs(rc), np.max(np.abs(rg)))
    assert abs(only.item() - rc) <= 1e-12 * max(abs(rc), np.max(np.abs(rg)))
    assert np.max(np.abs(grad[0].cpu().numpy() - rg)) <= 1e-12 * np.max(np.abs(rg))
