"""The rotation plan against the oracle: chains of rotations pushed through every kind of
two-qubit gate, chains and operation counts at and around the plan's limits, angles at which its
factorisations degenerate, and every direction and cost variant.

Tolerance 1e-12 relative to max(1, |reference|), as for the engine's other parity tests: at most
400 operations with a few roundings of 1.1e-16 each.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def close(a, b):
    a, b = np.asarray(a), np.asarray(b)
    assert np.max(np.abs(a - b)) <= 1e-12 * max(1.0, np.max(np.abs(b)))


def circuit(sqg, n, kind, length):
    """push_*: U3 runs on qubit 0 separated by gates that commute with one axis there."""
    rng = np.random.default_rng(length)
    c = sqg.Circuit(n)
    for k in range(length):
        if kind == "random":
            t = ("U3", "RX", "RY", "RZ", "CNOT", "CZ", "CRY")[rng.integers(7)]
            a, b = rng.choice(n, 2, replace=False)
            getattr(c, "add_" + t)(int(a), int(b)) if t[0] == "C" else getattr(c, "add_" + t)(int(a))
            continue
        c.add_U3(0)
        if k % 5 == 2:  # a run of several gates
            c.add_RX(0)
            c.add_RY(0)
            c.add_RX(0)
        if k % 3 == 1:
            c.add_U3(1)
        if kind == "push_z":
            c.add_CNOT(1, 0) if k % 2 else c.add_CZ(0, 1)
        elif kind == "push_x":
            c.add_CNOT(0, 1)
            if k % 4 == 0:
                c.add_CNOT(0, n - 1)
        elif kind == "push_y":
            c.add_CRY(0, 1)
        else:  # the axis changes from run to run
            (c.add_CNOT, c.add_CRY, c.add_CZ)[k % 3](k % 2, 1 - k % 2)
    return c


def angles(P, which):
    rng = np.random.default_rng(P)
    if which == "any":
        return rng.uniform(0, 2 * np.pi, P)
    if which == "zero":
        return np.zeros(P)
    if which == "tiny":
        return 1e-9 * rng.standard_normal(P)
    return rng.integers(0, 8, P) * (np.pi / 4)  # exchanges, ties of the pivots, the gimbal case


CASES = [(n, kind, length, which) for n, length in ((3, 15), (3, 16), (3, 17), (6, 33), (7, 70))
         for kind in ("push_z", "push_x", "push_y", "mixed") for which in ("any", "eighths")]
CASES += [(4, "random", 31, "any"), (4, "random", 32, "any"), (6, "random", 33, "zero"), (6, "random", 200, "tiny"),
          (8, "random", 300, "eighths"), (2, "push_x", 140, "any"), (5, "mixed", 1, "any")]


@pytest.mark.parametrize("n,kind,length,which", CASES)
def test_plan_against_oracle(sqg, n, kind, length, which):
    c = circuit(sqg, n, kind, length)
    recs, P = c.gate_records(), c.get_Parameter_Num()
    p = angles(P, which)
    rng = np.random.default_rng(n)
    N, cols = 1 << n, (1 << n) // 2 + 1  # too narrow for the environment-matrix evaluation
    T = np.linalg.qr(rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N)))[0][:, :cols].copy()
    M = O.get_matrix(n, recs, p)
    A = T.copy()
    c.apply_to(p, A)
    close(A, M @ T)
    R = np.ascontiguousarray(T.T)
    c.apply_from_right(p, R)
    close(R, T.T @ M)
    psi = np.ascontiguousarray(T[:, 0])
    c.apply_to(p, psi)
    close(psi, M @ T[:, 0])
    th = torch.from_numpy(p).cuda()
    for variant, offset, step in ((0, 0, 0), (0, N - cols, 7), (3, 0, 0), (9, 0, 32)):
        ev = sqg.CostEvaluator(c, T, trace_offset=offset, cost_variant=variant)
        cost, grad = ev.cost_grad(th, checkpoint_interval=step)
        rc, rg = O.cost_grad(n, recs, p, T, trace_offset=offset, variant=variant)
        close(cost.item(), rc)
        close(grad[0].cpu().numpy(), rg)
        close(ev.cost_grad(th, with_grad=False)[0].item(), rc)


def test_ragged_plans_share_a_launch(sqg):
    from importlib import import_module
    ragged = import_module("sequential-quantum-gate-decomposer_gb300.ragged")
    cs = [circuit(sqg, n, kind, length) for n, kind, length in
          ((3, "push_x", 40), (7, "random", 150), (5, "push_y", 3), (2, "push_z", 17), (6, "mixed", 50))]
    rng = np.random.default_rng(3)
    ts = [np.linalg.qr(rng.standard_normal((1 << c.qbit_num,) * 2) + 1j * rng.standard_normal((1 << c.qbit_num,) * 2))[0]
          for c in cs]
    th = [angles(c.get_Parameter_Num(), "any") for c in cs]
    rb = ragged.RaggedBatch(cs, ts)
    for variant in (0, 3, 9):
        cost, grad = rb.cost_grad(rb.pack(th), variant=variant)
        for i, (c, g) in enumerate(zip(cost.cpu().numpy(), rb.split(grad))):
            rc, rg = O.cost_grad(cs[i].qbit_num, cs[i].gate_records(), th[i], ts[i], variant=variant)
            close(c, rc)
            close(g.cpu().numpy(), rg)


@pytest.mark.parametrize("batch", [1, 31, 32, 33, 70])
def test_batches_make_the_same_numbers(sqg, batch):
    """Plans of many vectors are made in three launches, those of a few in one."""
    c = circuit(sqg, 5, "mixed", 60)
    recs, P = c.gate_records(), c.get_Parameter_Num()
    rng = np.random.default_rng(batch)
    p = np.concatenate([angles(P, "eighths")[None], rng.uniform(0, 2 * np.pi, (batch - 1, P))])
    T = np.linalg.qr(rng.standard_normal((32, 32)) + 1j * rng.standard_normal((32, 32)))[0][:, :17].copy()
    cost, grad = sqg.CostEvaluator(c, T).cost_grad(torch.from_numpy(p).cuda())
    for b in {0, batch // 2, batch - 1}:
        rc, rg = O.cost_grad(5, recs, p[b], T)
        close(cost[b].item(), rc)
        close(grad[b].cpu().numpy(), rg)


@pytest.mark.parametrize("n,batch", [(9, 1), (10, 3), (13, 1), (14, 2), (16, 1), (17, 1)])
def test_states_in_small_chunks(sqg, n, batch):
    """Registers whose chunks would leave the device idle are applied in smaller ones, with blocks of
    CNOTs alone among them."""
    rng = np.random.default_rng(n)
    c = circuit(sqg, n, "random", 120)
    for k in range(40):
        c.add_CNOT(*(int(q) for q in rng.choice(n, 2, replace=False)))
    for q in range(0, n, 3):
        c.add_U3(q)
    recs, P = c.gate_records(), c.get_Parameter_Num()
    p = rng.uniform(0, 2 * np.pi, (batch, P))
    v = rng.standard_normal((batch, 1 << n)) + 1j * rng.standard_normal((batch, 1 << n))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    d = torch.from_numpy(v.copy()).cuda()
    c.apply_state_device(torch.from_numpy(p).cuda(), d)
    for b in range(batch):
        close(d[b].cpu().numpy(), O.apply_to(n, recs, p[b], v[b].reshape(-1, 1).copy()).reshape(-1))


@pytest.mark.parametrize("n,gates,batch", [(3, 40, 2), (4, 31, 1), (4, 32, 1), (4, 27, 400), (4, 28, 400), (5, 1, 1),
                                           (5, 60, 3), (3, 111, 400), (3, 112, 400), (4, 39, 64), (4, 40, 64),
                                           (4, 23, 4), (4, 24, 4), (5, 10, 100), (5, 11, 100)])
def test_small_registers_with_and_without_a_workspace(sqg, n, gates, batch):
    """Up to five qubits the environment-matrix evaluation takes the calls that bring no workspace,
    and those where it is the faster one; both agree with the oracle."""
    from importlib import import_module
    native = import_module("sequential-quantum-gate-decomposer_gb300._native")
    c = circuit(sqg, n, "random", gates)
    recs, P = c.gate_records(), c.get_Parameter_Num()
    rng = np.random.default_rng(gates)
    p = rng.uniform(0, 2 * np.pi, (batch, P))
    N = 1 << n
    T = np.linalg.qr(rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N)))[0]
    th, tgt = torch.from_numpy(p).cuda(), torch.from_numpy(T.copy()).cuda()
    ev = sqg.CostEvaluator(c, T)
    room = torch.empty(ev.workspace_bytes(batch, True), dtype=torch.uint8, device="cuda")
    for ws, size in ((None, 0), (room.data_ptr(), room.numel() // 2), (room.data_ptr(), room.numel())):
        cost = torch.full((batch,), np.nan, dtype=torch.float64, device="cuda")
        grad = torch.full((batch, P), np.nan, dtype=torch.float64, device="cuda")
        native.check(native.lib().sqg_cost_grad(
            ev.native.handle, th.data_ptr(), batch, tgt.data_ptr(), N, 0, 0, 0, cost.data_ptr(), grad.data_ptr(), 0, ws,
            size, torch.cuda.current_stream().cuda_stream), "sqg_cost_grad")
        for b in {0, batch - 1}:
            rc, rg = O.cost_grad(n, recs, p[b], T)
            close(cost[b].item(), rc)
            close(grad[b].cpu().numpy(), rg)


@pytest.mark.parametrize("kind", ["push_x", "push_y", "push_z"])
def test_long_chains_keep_the_norm(sqg, kind):
    """The roundings of the plan's numbers have no preferred sign: over L runs the norm walks at random
    by about 1.5e-16 sqrt(L); five times that is allowed."""
    L = 10000
    c = circuit(sqg, 3, kind, L)
    A = np.eye(8, dtype=np.complex128)
    c.apply_to(angles(c.get_Parameter_Num(), "any"), A)
    assert abs(np.mean(np.linalg.norm(A, axis=0)) - 1.0) < 5 * 1.5e-16 * np.sqrt(2 * L)


@pytest.mark.parametrize("n,batch,cols", [(4, 700, 16), (5, 200, 32), (5, 700, 31), (6, 90, 50), (7, 40, 128)])
def test_batches_with_several_pairs_per_thread(sqg, n, batch, cols):
    """Launches with warps to spare take two or four pairs per thread."""
    c = circuit(sqg, n, "random", 60)
    recs, P = c.gate_records(), c.get_Parameter_Num()
    rng = np.random.default_rng(batch)
    p = rng.uniform(0, 2 * np.pi, (batch, P))
    N = 1 << n
    T = np.linalg.qr(rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N)))[0][:, :cols].copy()
    th = torch.from_numpy(p).cuda()
    for variant in (0, 3):
        ev = sqg.CostEvaluator(c, T, cost_variant=variant)
        cost, grad = ev.cost_grad(th)
        only = ev.cost_grad(th, with_grad=False)[0]
        for b in (0, batch - 1):
            rc, rg = O.cost_grad(n, recs, p[b], T, variant=variant)
            close(cost[b].item(), rc)
            close(only[b].item(), rc)
            close(grad[b].cpu().numpy(), rg)


@pytest.mark.parametrize("count", [1, 7, 400])
def test_ragged_tile_widths(sqg, count):
    """Batches of few items get narrower tiles; every width gives the same numbers."""
    from importlib import import_module
    ragged = import_module("sequential-quantum-gate-decomposer_gb300.ragged")
    rng = np.random.default_rng(count)
    cs = [circuit(sqg, 3 + (2 * i + 3) % 5, "random", 30) for i in range(count)]
    ts = [np.linalg.qr(rng.standard_normal((1 << c.qbit_num,) * 2) + 1j * rng.standard_normal((1 << c.qbit_num,) * 2))[0]
          for c in cs]
    th = [rng.uniform(0, 2 * np.pi, c.get_Parameter_Num()) for c in cs]
    for width in (None, 3, 8):
        rb = ragged.RaggedBatch(cs, ts, tile_cols=None if width is None else [width] * count)
        cost, grad = rb.cost_grad(rb.pack(th))
        grads = rb.split(grad)
        for i in {0, count // 2, count - 1}:
            rc, rg = O.cost_grad(cs[i].qbit_num, cs[i].gate_records(), th[i], ts[i])
            close(cost[i].item(), rc)
            close(grads[i].cpu().numpy(), rg)


@pytest.mark.parametrize("n,batch", [(5, 160), (6, 160), (7, 40), (8, 11), (8, 3)])
def test_narrow_tiles_and_a_workspace_for_wide_ones(sqg, n, batch):
    """Launches of two to three CTAs per SM take narrower tiles where the workspace has room for
    them; one that was large enough for the wide tiles still is."""
    from importlib import import_module
    native = import_module("sequential-quantum-gate-decomposer_gb300._native")
    c = circuit(sqg, n, "random", 25)
    recs, P = c.gate_records(), c.get_Parameter_Num()
    rng = np.random.default_rng(n)
    p = rng.uniform(0, 2 * np.pi, (batch, P))
    N = 1 << n
    T = np.linalg.qr(rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N)))[0]
    th, tgt = torch.from_numpy(p).cuda(), torch.from_numpy(T.copy()).cuda()
    ev = sqg.CostEvaluator(c, T)
    size = ev.workspace_bytes(batch, True)
    wide = ev.workspace_bytes(batch, True, 1000)  # checkpointed, none of them stored: wide tiles
    assert wide <= size
    for have in (size, wide):
        guard = torch.full((have + 4096,), 7, dtype=torch.uint8, device="cuda")
        cost = torch.full((batch,), np.nan, dtype=torch.float64, device="cuda")
        grad = torch.full((batch, P), np.nan, dtype=torch.float64, device="cuda")
        native.check(native.lib().sqg_cost_grad(
            ev.native.handle, th.data_ptr(), batch, tgt.data_ptr(), N, 0, 0, 0, cost.data_ptr(), grad.data_ptr(), 0,
            guard.data_ptr(), have, torch.cuda.current_stream().cuda_stream), "sqg_cost_grad")
        assert bool((guard[have:] == 7).all())
        for b in (0, batch - 1):
            rc, rg = O.cost_grad(n, recs, p[b], T)
            close(cost[b].item(), rc)
            close(grad[b].cpu().numpy(), rg)
