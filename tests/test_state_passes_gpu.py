"""The fused passes over a state: as many as sqg_state_block_count says, and none that splits a
partition which fits a chunk of 12 qubits.  Passes are counted as the kernels of a captured call: one
makes the plan's numbers (fewer than 32 vectors), the others are the passes."""
import ctypes
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def passes(c, n, batch):
    native = importlib.import_module("sequential-quantum-gate-decomposer_gb300._native")
    lib = native.lib()
    cuda = ctypes.CDLL("libcuda.so.1")
    h = c.native().handle
    P = c.get_Parameter_Num()
    th = torch.zeros((batch, P), dtype=torch.float64, device="cuda")
    v = torch.zeros((batch, 1 << n), dtype=torch.complex128, device="cuda")
    v[:, 0] = 1.0
    ws = torch.empty(lib.sqg_state_workspace_bytes(h, batch), dtype=torch.uint8, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph, count = ctypes.c_void_p(), ctypes.c_size_t()
    assert cuda.cuStreamBeginCapture_v2(ctypes.c_void_p(s.cuda_stream), 2) == 0
    rc = lib.sqg_apply_state(h, th.data_ptr(), batch, v.data_ptr(), 1 << n, 1, ws.data_ptr(), ws.numel(), s.cuda_stream)
    assert cuda.cuStreamEndCapture(ctypes.c_void_p(s.cuda_stream), ctypes.byref(graph)) == 0
    assert rc == 0
    assert cuda.cuGraphGetNodes(graph, None, ctypes.byref(count)) == 0
    assert cuda.cuGraphDestroy(graph) == 0
    return count.value - 1


def block(sqg, n, qubits, rng):
    b = sqg.Circuit(n)
    for _ in range(3):
        for q in qubits:
            b.add_RY(int(q))
        for x, y in zip(qubits, rng.permutation(qubits)):
            if x != y:
                b.add_CRY(int(x), int(y))
    return b


@pytest.mark.parametrize("n", [13, 16, 20])
def test_partitions_of_up_to_a_chunk_are_not_split(sqg, n):
    rng = np.random.default_rng(n)
    c = sqg.Circuit(n)
    parts = 8
    for _ in range(parts):
        c.add_Circuit(block(sqg, n, 5 + rng.permutation(n - 5)[:7], rng))
    assert passes(c, n, 1) == c.state_block_count() <= parts


@pytest.mark.parametrize("n", [9, 13, 16, 20, 22])
def test_block_count_is_the_number_of_passes(sqg, n):
    wl = importlib.import_module("sequential-quantum-gate-decomposer_gb300.workloads")
    c = wl.all_gates_circuit(n, 200, np.random.default_rng(n))
    assert passes(c, n, 1) == c.state_block_count()
