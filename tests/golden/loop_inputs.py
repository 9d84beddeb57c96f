"""Inputs of the device optimizer loops whose results are kept in loops.npz.

Made from exactly reproducible numbers (the generator's uniform doubles, scaled by powers of two), so
that every machine starts from the same bits.  The targets are not unitary: their cost stays far
above the tolerance, no run stops early, and the trajectories amplify any change of an evaluation's rounding.
"""
import numpy as np

# name: (engine, qubits, CNOT blocks, columns, trace offset, cost variant, evaluations)
CASES = {
    "bfgs_n6": ("bfgs", 6, 20, 64, 0, 0, 60),
    "bfgs_n7_part": ("bfgs", 7, 12, 50, 30, 0, 40),
    "bfgs_n6_hs": ("bfgs", 6, 10, 64, 0, 3, 40),
    "bfgs_n4_narrow": ("bfgs", 4, 12, 5, 0, 9, 40),  # too narrow for the environment-matrix evaluation
    "bfgs_n9_gates": ("bfgs", 9, 8, 512, 0, 0, 20),
    "adam_n6": ("adam", 6, 8, 64, 0, 0, 200),
}


def make(sqg, name):
    engine, n, blocks, cols, offset, variant, calls = CASES[name]
    rng = np.random.default_rng(sorted(CASES).index(name))
    c = sqg.Circuit(n)
    for q in range(n):
        c.add_U3(q)
    for k in range(blocks):
        a, b = k % n, (k + 1) % n
        c.add_CNOT(a, b) if k % 2 else c.add_CNOT(b, a)
        c.add_U3(a)
        c.add_U3(b)
        if n == 9:  # every other kind of gate
            c.add_RX(a)
            c.add_RY(b)
            c.add_RZ(a)
            c.add_CZ(a, b)
            c.add_CRY(b, a)
    T = (rng.random((1 << n, cols)) - 0.5 + 1j * (rng.random((1 << n, cols)) - 0.5)) / 8.0
    x0 = rng.random(c.get_Parameter_Num()) * 6.0
    kw = dict(engine=engine, trace_offset=offset, cost_variant=variant, max_outer=1, seed=3)
    kw["max_calls" if engine == "bfgs" else "max_iters"] = calls
    return c, T, x0, kw
