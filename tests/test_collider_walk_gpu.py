"""IfCollides' walk through the colliders' LBVH against the oracle, which tests
every stored collider: dense scenes (many hits and near misses), extents of
either sign, one to a few thousand colliders, and batches on either side of the
sizes at which a warp takes 4, 8, 16 and 32 waiting shapes.  The billboards have
no z extent: the hierarchy's boxes hold a quad as a flat shape, while the axis
tests take its z extent along its own normal, so that a turned tree within that
extent of a billboard, and no nearer, is a hit to the oracle only."""
import numpy as np
import pytest

import oracle
from operatorgraph_gb300 import grammar as G
from operatorgraph_gb300 import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (2, 33, 1), (1, 40, 2), (64, 9700, 40), (64, 9760, 40), (300, 19500, 300), (150, 40000, 150),
         (40, 78000, 40), (2500, 700, 2500)]


@pytest.mark.parametrize("negative", [False, True], ids=["positive", "signed"])
@pytest.mark.parametrize("rotate", [False, True], ids=["frame_codes", "general_frames"])
@pytest.mark.parametrize("size", SIZES)
def test_walk_finds_what_every_pair_finds(size, rotate, negative):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from operatorgraph_gb300.engine import Engine, terminals_to_numpy

    b = scenes.collisions(*size, rotate=rotate)
    ax = b["axioms"]
    stored = size[0] + size[2]
    ax["position"][:, [0, 2]] *= np.float32(0.45)  # about five times as dense
    ax["size"][size[0]:stored, 2] = 0.0
    if negative:
        ax["size"][:stored:3, 0] *= np.float32(-1)
        ax["size"][1:stored:4, 1] *= np.float32(-1)
    ref = G.sort_terminals(oracle.derive(G.DEFAULT_PROCS, b["entries"], ax), by_path=True)
    eng = Engine(b["entries"], node_capacity=1 << 20, max_terminals=1 << 20)
    out, n, rep = eng.execute(ax, capacity=len(ref))
    assert rep["status"] == 0 and n == len(ref)
    got = G.sort_terminals(terminals_to_numpy(out, n), by_path=True)
    assert np.array_equal(got["path"], ref["path"]) and np.array_equal(got["rule"], ref["rule"])
    assert np.array_equal(got["m"] + np.float32(0), ref["m"] + np.float32(0))
    eng.release()
