"""IfCollides against quads with a z extent, which the axis tests take along the
quad's normal: turned trees among billboards, denser than the scene's own, as
the oracle finds them by testing every stored collider."""
import numpy as np
import pytest

import oracle
from operatorgraph_gb300 import grammar as G
from operatorgraph_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rotate", [False, True], ids=["frame_codes", "general_frames"])
@pytest.mark.parametrize("size,depth", [((150, 40000, 150), 1.0), ((64, 9700, 40), 5.0), ((1, 40, 2), 30.0)])
def test_quads_of_some_depth(size, depth, rotate):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from operatorgraph_gb300.engine import Engine, terminals_to_numpy

    b = scenes.collisions(*size, rotate=rotate)
    ax = b["axioms"]
    ax["position"][:, [0, 2]] *= np.float32(0.45)
    boards = slice(size[0], size[0] + size[2])
    ax["size"][boards, 2] = depth
    ref = G.sort_terminals(oracle.derive(G.DEFAULT_PROCS, b["entries"], ax), by_path=True)
    eng = Engine(b["entries"], node_capacity=1 << 20, max_terminals=1 << 20)
    out, n, rep = eng.execute(ax, capacity=len(ref) + 1000)
    got = G.sort_terminals(terminals_to_numpy(out, n), by_path=True)
    eng.release()
    assert rep["status"] == 0 and n == len(ref)
    assert np.array_equal(got["path"], ref["path"]) and np.array_equal(got["rule"], ref["rule"])
    assert np.array_equal(got["m"] + np.float32(0), ref["m"] + np.float32(0))
