"""The adjoint's two launch shapes (k_adjoint and k_adjoint_wide, by the engine's
terminal capacity) on batches with nearly as many terminals as the largest
engine of the first shape holds: the same block and size gradients to FP32
accumulation order."""
import os
import re

import numpy as np
import pytest

import operatorgraph_gb300
from operatorgraph_gb300 import scenes

pytestmark = pytest.mark.gpu


def _wide_from():
    src = os.path.join(os.path.dirname(operatorgraph_gb300.__file__), "csrc", "derive_kernels.cuh")
    return 1 << int(re.search(r"kWideAdjointTerminals = 1ull << (\d+);", open(src).read()).group(1))


@pytest.mark.parametrize("name", ["mixed", "mixed blocks", "city"])
def test_both_shapes_near_the_line(name):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from operatorgraph_gb300.autograd import axioms_tensor
    from operatorgraph_gb300.engine import Engine

    line = _wide_from()
    b = scenes.city(line // 1500) if name == "city" else scenes.mixed(line // 2500, blocks=name.endswith("blocks"))
    n = len(b["axioms"])
    b["axioms"]["position"] = 0.0  # coordinates of one size, so that the gradients' terms are comparable
    axioms = axioms_tensor(b["axioms"])
    blk = None if b["blocks"] is None else torch.from_numpy(b["blocks"]).cuda()
    grads, counts = [], []
    for cap in (line - 1, line):
        eng = Engine(b["entries"], node_capacity=1 << 22, max_terminals=cap, block_stride=b["block_stride"],
                     record_tape=True)
        out, count, _ = eng.execute(axioms, blocks=blk, capacity=cap)
        g = torch.zeros((n, 3), device="cuda")
        gb = None if blk is None else torch.zeros_like(blk)
        eng.adjoint_raw(out.data_ptr(), None if gb is None else gb.data_ptr(), 0 if gb is None else n, g.data_ptr(),
                        grad_stride=16)
        torch.cuda.synchronize()
        assert eng.report()["status"] == 0
        grads.append([x.cpu().numpy().astype(np.float64) for x in (g, gb) if x is not None])
        counts.append(count)
        eng.release()
    assert counts[0] == counts[1] > 0.8 * line
    # At most 8,000 terminals an axiom in a mix and 20,000 in the city: 20000 * 2^-24 = 1.2e-3 of the largest sum.
    for x, y in zip(*grads):
        assert np.isfinite(x).all() and np.abs(x - y).max() <= 1.2e-3 * np.abs(y).max() and np.abs(y).max() > 0
