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
    want = O.apply_to(2, c.gate_records(), th[5].cpu().numpy(), T.copy())
    assert abs(cost[5].item() - (1.0 - np.trace(want[:3]).real / 3)) <= 1e-12
    assert abs(cost[5].item() - cost1.item()) <= 1e-12
    assert torch.max(torch.abs(grad[5] - grad1[0])).item() <= 1e-12
    m = torch.from_numpy(np.repeat(T[None], 32, axis=0)).cuda()
    c.apply_to_device(th, m)
    assert np.max(np.abs(m[5].cpu().numpy() - want)) <= 1e-12


def test_ragged_more_overlaps_than_a_grid_is_high(sqg):
    """An instance whose overlaps are summed by more than 65535 CTAs of 32, against the evaluator of one circuit
    (whose sums are counted in another dimension) and the oracle's matrix.  Tolerance: 700000 operations of a
    rounding each both ways, 2^-53 sqrt(1.4e6) = 1.3e-13, here 1e-11."""
    ragged = importlib.import_module("sequential-quantum-gate-decomposer_gb300.ragged")
    rng = np.random.default_rng(2)
    big, small = sqg.Circuit(2), sqg.Circuit(3)
    for _ in range(65536 * 32 // 3 + 10):  # three overlaps each
        big.add_U3(0)
        big.add_CNOT(0, 1)
        big.add_CNOT(1, 0)
    for q in (0, 1, 2, 0):
        small.add_U3(q)
    cs = [small, big]
    ts = [np.linalg.qr(rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N)))[0] for N in (8, 4)]
    th = [rng.uniform(0, 2 * np.pi, c.get_Parameter_Num()) for c in cs]
    rb = ragged.RaggedBatch(cs, ts)
    cost, grad = rb.cost_grad(rb.pack(th))
    for i, g in enumerate(rb.split(grad)):
        want = O.apply_to(cs[i].qbit_num, cs[i].gate_records(), th[i], ts[i].copy())
        assert abs(cost[i].item() - (1.0 - np.trace(want).real / len(want))) <= 1e-11
        one, one_grad = sqg.CostEvaluator(cs[i], ts[i]).cost_grad(torch.from_numpy(th[i]).cuda())
        assert abs(cost[i].item() - one.item()) <= 1e-11
        assert torch.max(torch.abs(g - one_grad[0])).item() <= 1e-11
