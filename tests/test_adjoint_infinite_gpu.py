"""An infinite dL/dM of a Subdivide's first child, whose piece is absolute: it
reaches the sizes and that child's factor, and leaves the other factors'
gradients, whose terms do not depend on it, what they are without it."""
import numpy as np
import pytest

from operatorgraph_gb300 import grammar as G
from operatorgraph_gb300.grammar import DispatchTable, Entry, block, scalar

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 8])
def test_infinite_gradient_of_an_absolute_piece(n):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from operatorgraph_gb300.autograd import axioms_tensor
    from operatorgraph_gb300.engine import Engine

    values = [0.11, -0.7, 0.07, -0.4, 0.05, 0.13, -0.9, 0.06][:n]
    table = DispatchTable([
        Entry(G.BOX_SUBDIVIDE, [scalar(2)] + [block(k) for k in range(n)], [(1 + k, 0) for k in range(n)]),
    ] + [Entry(G.BOX_GENERATE, [scalar(k)], []) for k in range(n)]).to_array()
    ax = G.make_axioms(1)
    ax["entry"], ax["shape"], ax["size"] = 0, G.SHAPE_BOX, 1.0
    blk = torch.tensor(values, device="cuda")
    eng = Engine(table, node_capacity=1 << 16, max_terminals=1 << 16, block_stride=n, record_tape=True)
    axioms = axioms_tensor(ax)
    out, count, _ = eng.execute(axioms, blocks=blk, capacity=64)
    assert count == n
    z = out[:n].view(torch.float32).view(n, 16)[:, 11]
    grad = torch.zeros((n, 12), device="cuda")
    grad[int(z.argmin()), 11] = float("inf")  # the translation of the first child along the split axis
    g_sizes, g_blk = torch.zeros(3, device="cuda"), torch.zeros(n, device="cuda")
    eng.adjoint_raw(grad.data_ptr(), g_blk.data_ptr(), 1, g_sizes.data_ptr())
    torch.cuda.synchronize()
    assert eng.report()["status"] == 0
    eng.release()
    # z_0 = -S / 2 + f_0 / 2
    assert g_sizes.tolist() == [0.0, 0.0, -float("inf")]
    assert g_blk.tolist() == [float("inf")] + [0.0] * (n - 1)
