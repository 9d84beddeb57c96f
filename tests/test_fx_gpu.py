"""Fixed-point sweeps of cost and gradient: magnitudes over the whole exponent range, vectors of
very different norms in one tile, structured inputs, every tile shape, and the inputs that are
swept in FP64 instead (infinities, NaN, checkpoints).

Tolerance 1e-12 relative to max(1, |reference|): the resolution is 2^-62 of the largest vector's
norm and the errors of some hundred operations add up to less than 2^-50 of it.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def close(a, b):
    a, b = np.asarray(a), np.asarray(b)
    assert np.max(np.abs(a - b)) <= 1e-12 * max(1.0, np.max(np.abs(b)))


def setup(n, cols, gates=60, seed=0):
    from importlib import import_module
    wl = import_module("sequential-quantum-gate-decomposer_gb300.workloads")
    rng = np.random.default_rng(100 * n + cols + seed)
    c = wl.all_gates_circuit(n, gates, rng)
    T = rng.standard_normal((1 << n, cols)) + 1j * rng.standard_normal((1 << n, cols))
    return c, rng.uniform(0, 2 * np.pi, c.get_Parameter_Num()), T / np.linalg.norm(T, axis=0)


def check(sqg, c, p, T, variants=(0, 3)):
    th = torch.from_numpy(p).cuda()
    for v in variants:
        ev = sqg.CostEvaluator(c, np.ascontiguousarray(T), cost_variant=v)
        cost, grad = ev.cost_grad(th)
        rc, rg = O.cost_grad(c.qbit_num, c.gate_records(), p, T, variant=v)
        close(cost.item(), rc)
        close(grad[0].cpu().numpy(), rg)
        close(ev.cost_grad(th, with_grad=False)[0].item(), rc)


@pytest.mark.parametrize("n,cols", [(1, 1), (2, 1), (3, 5), (4, 11), (5, 23), (6, 33), (6, 64), (7, 17), (8, 9), (9, 5),
                                    (11, 2), (12, 1)])
def test_tile_shapes(sqg, n, cols):
    check(sqg, *setup(n, cols))


@pytest.mark.parametrize("exponent", [-1060, -1000, -300, -62, 62, 300, 900])
def test_magnitudes(sqg, exponent):
    c, p, T = setup(6, 21)
    check(sqg, c, p, np.ldexp(T.real, exponent) + 1j * np.ldexp(T.imag, exponent), (0, 3) if abs(exponent) <= 300 else (0,))


@pytest.mark.parametrize("n,cols", [(6, 64), (7, 40)])
def test_unlike_columns_and_structured_inputs(sqg, n, cols):
    c, p, T = setup(n, cols)
    U = T.copy()
    U[:, ::3] *= 1e-9
    U[:, 1::3] = 0.0
    check(sqg, c, p, U)
    check(sqg, c, p, np.zeros_like(T))
    check(sqg, c, p, np.eye(1 << n, cols).astype(np.complex128))
    check(sqg, c, np.zeros_like(p), np.eye(1 << n, cols).astype(np.complex128))
    check(sqg, c, np.full_like(p, np.pi / 4), T)


@pytest.mark.parametrize("where", ["target inf", "target nan", "angle inf", "angle nan"])
def test_not_finite_as_in_fp64(sqg, where):
    """Checkpointed gradients are swept in FP64: the same values, and not finite in the same places."""
    c, p, T = setup(6, 64)
    bad = np.inf if where.endswith("inf") else np.nan
    if where.startswith("target"):
        T[5, 40] = bad
    else:
        p[7] = bad
    th = torch.from_numpy(p).cuda()
    ev = sqg.CostEvaluator(c, T)
    cost, grad = ev.cost_grad(th)
    cost64, grad64 = ev.cost_grad(th, checkpoint_interval=5)
    assert np.array_equal(cost.cpu().numpy(), cost64.cpu().numpy(), equal_nan=True)
    assert np.array_equal(torch.isnan(grad).cpu().numpy(), torch.isnan(grad64).cpu().numpy())
    assert not torch.isfinite(cost).any() and not torch.isfinite(grad).all()
