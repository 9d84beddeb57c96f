"""The device optimizer loops return the same point, cost and counts bit for bit, whatever the
evaluations outside of them do: trajectories amplify any change of rounding, so which point a
decomposition ends at depends on the last place of every evaluation.  loops.npz holds the results of
the gate-by-gate FP64 evaluation on a GB300 (loop_inputs.py makes the inputs)."""
import importlib
import os

import numpy as np
import pytest

from golden import loop_inputs

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("name", sorted(loop_inputs.CASES))
def test_loop_returns_what_it_returned(sqg, name):
    batched = importlib.import_module("sequential-quantum-gate-decomposer_gb300.batched")
    golden = np.load(os.path.join(os.path.dirname(__file__), "golden", "loops.npz"))
    c, T, x0, kw = loop_inputs.make(sqg, name)
    run = {"bfgs": batched.bfgs_decompose_graph, "adam": batched.adam_decompose_graph}[kw.pop("engine")]
    for got, key in zip(run(c, T, x0, **kw), ("x", "cost", "n1", "n2")):
        assert np.array_equal(got.cpu().numpy(), golden[name + "_" + key]), key
