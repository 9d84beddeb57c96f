"""Infinities and NaN reach the amplitudes that the gates mix them into and no others: circuits of gates
that act on real and imaginary parts alike (CNOT, CZ, RX, RY, CRY), applied to matrices and states with
an infinite component, and circuits with a NaN angle whose gate leaves half of the amplitudes alone,
against the gates in plain numpy.  Finite values agree to 1e-12 (at most 40 gates)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def apply(n, gates, A):
    """Gate by gate on real and imaginary parts (rows of A)."""
    re, im = A.real.copy(), A.imag.copy()
    rows = np.arange(1 << n)
    for name, t, ctl, a in gates:
        x = rows[((rows >> t) & 1 == 0) & ((ctl < 0) | ((rows >> max(ctl, 0)) & 1 == 1))]
        y = x | 1 << t
        if name == "CNOT":
            re[np.r_[x, y]], im[np.r_[x, y]] = re[np.r_[y, x]], im[np.r_[y, x]]
        elif name == "CZ":
            re[y], im[y] = -re[y], -im[y]
        elif name == "RX":
            c, s = np.cos(a), np.sin(a)
            re[x], im[x], re[y], im[y] = (c * re[x] + s * im[y], c * im[x] - s * re[y], c * re[y] + s * im[x],
                                          c * im[y] - s * re[x])
        else:
            c, s = np.cos(a), np.sin(a)
            for v in (re, im):
                v[x], v[y] = c * v[x] - s * v[y], s * v[x] + c * v[y]
    out = np.empty_like(A)
    out.real, out.imag = re, im
    return out


def draw(sqg, n, names, count, seed, nan_at=-1):
    rng = np.random.default_rng(seed)
    c, gates, p = sqg.Circuit(n), [], []
    for k in range(count):
        name = "CRY" if k == nan_at else names[rng.integers(len(names))]
        t, ctl = (int(q) for q in rng.choice(n, 2, replace=False))
        if name[0] != "C":
            ctl = -1
        getattr(c, "add_" + name)(t, ctl) if ctl >= 0 else getattr(c, "add_" + name)(t)
        a = 0.0
        if name in ("RX", "RY", "CRY"):
            a = np.nan if k == nan_at else rng.uniform(0.1, 6.0)
            p.append(a)
        gates.append((name, t, ctl, a))
    return c, gates, np.array(p)


def same(got, want, nan_too=False):
    """Equal wherever the gates one by one leave a number; nan_too: NaN nowhere else but there.  (Two rotations
    taken as one may avoid an infinity minus itself.)"""
    for g, w in ((got.real, want.real), (got.imag, want.imag)):
        if nan_too:
            assert np.array_equal(np.isnan(g), np.isnan(w))
        n = ~np.isnan(w)
        g, w = g[n], w[n]
        assert np.array_equal(np.isinf(g), np.isinf(w)) and np.array_equal(g[np.isinf(w)], w[np.isinf(w)])
        f = np.isfinite(w)
        assert np.all(np.abs(g[f] - w[f]) <= 1e-12)


CASES = [("CNOT",), ("CNOT", "CZ"), ("CNOT", "CZ", "CRY"), ("RY", "CNOT", "CRY"), ("RX", "CNOT", "CZ")]


@pytest.mark.filterwarnings("ignore::RuntimeWarning")
@pytest.mark.parametrize("names", CASES)
@pytest.mark.parametrize("n", [3, 10])
def test_infinite_amplitude(sqg, n, names):
    count = 6 if n == 3 else 40
    with np.errstate(invalid="ignore"):
        c, gates, p = draw(sqg, n, names, count, n)
        rng = np.random.default_rng(n)
        A = rng.standard_normal((1 << n, 5)) + 1j * rng.standard_normal((1 << n, 5))
        A[2, 1] = complex(np.inf, 0.5)
        A[5, 3] = complex(0.25, -np.inf)
        want = apply(n, gates, A)
        got = A.copy()
        c.apply_to(p, got)
        same(got, want)
        v = torch.from_numpy(np.ascontiguousarray(A[:, 1:4:2].T)).cuda()
        c.apply_state_device(torch.from_numpy(np.stack([p, p])).cuda(), v)
        same(v.cpu().numpy().T, want[:, 1:4:2])


def test_cost_of_an_infinite_amplitude(sqg):
    """The trace's infinite real part; its finite imaginary part is not dragged along."""
    c = sqg.Circuit(6)
    c.add_CZ(0, 1)
    c.add_CNOT(2, 3)
    A = np.eye(64, 40).astype(np.complex128)
    A[0, 0] = complex(np.inf, 0.0)
    cost = sqg.CostEvaluator(c, A).cost_grad(torch.zeros((1, 0), dtype=torch.float64, device="cuda"))[0]
    assert cost.item() == -np.inf


@pytest.mark.parametrize("batch", [1, 40])
@pytest.mark.parametrize("names", [("CNOT", "CZ"), ("RY", "CNOT", "CZ")])
@pytest.mark.parametrize("n", [3, 6, 10])
def test_nan_angle_of_a_controlled_rotation(sqg, n, names, batch):
    """The last gate: amplitudes with control bit 0 stay.  From 32 vectors on the plan's numbers are
    made in three launches."""
    count = 12
    c, gates, p = draw(sqg, n, names, count, 3 * n, nan_at=count - 1)
    rng = np.random.default_rng(n)
    A = rng.standard_normal((1 << n, 5)) + 1j * rng.standard_normal((1 << n, 5))
    want = apply(n, gates, A)
    assert np.isnan(want).any() and not np.isnan(want).all()
    th = torch.from_numpy(np.repeat(p[None], batch, axis=0)).cuda()
    m = torch.from_numpy(np.repeat(A[None], batch, axis=0)).cuda()
    c.apply_to_device(th, m)
    same(m[batch - 1].cpu().numpy(), want, True)
    v = torch.from_numpy(np.repeat(A[None, :, 0], batch, axis=0)).cuda()
    c.apply_state_device(th, v)
    same(v[batch - 1].cpu().numpy(), want[:, 0], True)
    # the cost is NaN where the trace is
    ev = sqg.CostEvaluator(c, A)
    trace = np.trace(want[:5]).real
    for cost in (ev.cost_grad(th)[0], ev.cost_grad(th, checkpoint_interval=4)[0], ev.cost_grad(th, with_grad=False)[0]):
        same(cost[batch - 1:].cpu().numpy(), np.array([1.0 - trace / 5]), True)


@pytest.mark.parametrize("batch", [1, 40])
@pytest.mark.parametrize("which", range(9))
@pytest.mark.parametrize("between", ["CZ", "CNOT", "CRY"])
def test_nan_angle_anywhere_in_a_chain(sqg, between, which, batch):
    """Runs of one and of several U3 whose rotations are pushed through two-qubit gates, one angle NaN:
    matrix, state, cost and gradient are NaN, not a number that looks like a result."""
    n = 6
    c = sqg.Circuit(n)
    for run in (1, 2, 1, 1):
        for _ in range(run):
            c.add_U3(0)
        c.add_U3(1)
        {"CZ": c.add_CZ, "CNOT": c.add_CNOT, "CRY": c.add_CRY}[between](0, 1)
    for q in range(n):
        c.add_RY(q)  # mixes every half that was left alone
    rng = np.random.default_rng(which)
    p = rng.uniform(0.3, 1.2, c.get_Parameter_Num())
    u3 = [r[3] for r in c.gate_records() if r[0] == 7 and r[1] == 0]  # its angles start there
    p[u3[which // 3 + which % 2] + which % 3] = np.nan
    th = torch.from_numpy(np.repeat(p[None], batch, axis=0)).cuda()
    T = np.linalg.qr(rng.standard_normal((1 << n, 1 << n)))[0].astype(np.complex128)
    ev = sqg.CostEvaluator(c, T)
    for kw in ({}, {"checkpoint_interval": 3}):
        cost, grad = ev.cost_grad(th, **kw)
        assert torch.isnan(cost).all() and torch.isnan(grad).any(dim=1).all()
    assert torch.isnan(ev.cost_grad(th, with_grad=False)[0]).all()
    m = torch.from_numpy(np.repeat(T[None], batch, axis=0)).cuda()
    c.apply_to_device(th, m)
    assert torch.isnan(m.real).flatten(1).any(dim=1).all()
    v = torch.from_numpy(np.repeat(T[None, :, 0], batch, axis=0).copy()).cuda()
    c.apply_state_device(th, v)
    assert torch.isnan(v.real).any(dim=1).all()
