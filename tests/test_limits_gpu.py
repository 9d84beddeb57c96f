"""Counts beyond the height of a CUDA grid (65535), which the entry points take."""
import importlib

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_more_chains_than_a_grid_is_high(sqg):
    """Every CRY is a chain of its own; from 32 vectors on the plan's numbers are made in three
    launches.  A result of the batch equals that of the vector by itself (70000 operations, 2^-53 sqrt(70000)
    = 3e-14 each way)."""
    rng = np.random.default_rng(1)
    c = sqg.Circuit(2)
    for k in range(70000):
        c.add_CRY(k % 2, 1 - k % 2)
    P = c.get_Parameter_Num()
    th = torch.from_numpy(rng.uniform(0, 2 * np.pi, (32, P))).cuda()
    T = np.linalg.qr(rng.standard_normal((4, 3)) + 1j * rng.standard_normal((4, 3)))[0].copy()
    ev = sqg.CostEvaluator(c, T)
    cost, grad = ev.cost_grad(th)
    cost1, grad1 = ev.cost_grad(th[5:6].contiguous())
    rc, rg = O.cost_grad(2, c.gate_records(), th[5].cpu().numpy(), T)
    assert abs(cost1.item() - rc) <= 1e-12 and abs(cost[5].item() - rc) <= 1e-12
    assert np.max(np.abs(grad1[0].cpu().numpy() - rg)) <= 1e-12
    assert np.max(np.abs(grad[5].cpu().numpy() - rg)) <= 1e-12
    m = torch.from_numpy(np.repeat(T[None], 32, axis=0)).cuda()
    c.apply_to_device(th, m)
    assert np.max(np.abs(m[5].cpu().numpy() - O.apply_to(2, c.gate_records(), th[5].cpu().numpy(), T.copy()))) <= 1e-12
