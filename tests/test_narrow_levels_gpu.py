"""Levels with few work items, whose chunks 2, 4 or 8 warps share: batches whose
levels lie on either side of each step (the grid has some 2,400 warps of 32
items), with the default and with coarse and fine work items, with and without
in-place leaf children; bit for bit against the restatement, and the gradients
of the recorded tape against those of an engine whose items hold one child
each."""
import numpy as np
import pytest

from operatorgraph_gb300 import grammar as G
from operatorgraph_gb300 import scenes

pytestmark = pytest.mark.gpu


def _torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


BATCHES = [("city", n) for n in (1, 2, 17, 300, 900)] + [("menger", n) for n in (1, 5, 130, 700)] + [("forest", 37)]


def _batch(name, n):
    return {"city": scenes.city, "forest": scenes.forest}[name](n) if name != "menger" else scenes.menger(0.15, n)


@pytest.mark.parametrize("sub", [0, 1, 20])
@pytest.mark.parametrize("name,n", BATCHES)
def test_narrow_levels_bit_exact(name, n, sub):
    torch = _torch()
    import oracle
    from operatorgraph_gb300.engine import Engine, terminals_to_numpy

    b = _batch(name, n)
    ref = G.sort_terminals(oracle.derive(G.DEFAULT_PROCS, b["entries"], b["axioms"], capacity=4_000_000), by_path=True)
    for no_inline in (False, True):
        eng = Engine(b["entries"], node_capacity=1 << 22, max_terminals=len(ref) + 64, sub_item=sub,
                     no_inline=no_inline)
        out, count, rep = eng.execute(b["axioms"], capacity=len(ref) + 64)
        got = G.sort_terminals(terminals_to_numpy(out, count), by_path=True)
        assert len(got) == len(ref)
        assert np.array_equal(got["path"], ref["path"]) and np.array_equal(got["rule"], ref["rule"])
        assert np.array_equal(got["m"] + np.float32(0), ref["m"] + np.float32(0))
        starts, _ = eng.levels()
        assert rep["nodes"] >= int(starts[-1]) and rep["levels"] + 1 == len(starts)
        eng.release()


@pytest.mark.parametrize("name,n", [("city", 17), ("menger", 130), ("forest", 37)])
def test_tape_of_shared_chunks_gives_the_gradients_of_single_children(name, n):
    torch = _torch()
    from operatorgraph_gb300.autograd import axioms_tensor
    from operatorgraph_gb300.engine import Engine

    b = _batch(name, n)
    axioms = axioms_tensor(b["axioms"])  # the adjoint reads them again
    grads = []
    for sub in (0, 1):
        eng = Engine(b["entries"], node_capacity=1 << 22, max_terminals=1 << 20, record_tape=True, sub_item=sub)
        out, count, _ = eng.execute(axioms, capacity=1 << 20)
        g = torch.zeros((n, 3), device="cuda")
        eng.adjoint_raw(out.data_ptr(), None, 0, g.data_ptr(), grad_stride=16)  # L = |M|^2 / 2
        torch.cuda.synchronize()
        assert eng.report()["status"] == 0
        grads.append(g.cpu().numpy().astype(np.float64))
        eng.release()
    # two orders of summation in FP32 over the 10^2 .. 10^4 terminals of an axiom: n eps / 2 of the sum of magnitudes
    scale = np.abs(grads[1]).max()
    assert np.abs(grads[0] - grads[1]).max() <= 1e-4 * scale
