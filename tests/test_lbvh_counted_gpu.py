"""pga_lbvh_build_counted over one leaf: no tree, but the leaf's key ahead of the
padding, in both forms of the sort (capacities either side of 622,592)."""
import numpy as np
import pytest

from operatorgraph_gb300 import grammar as G
from operatorgraph_gb300 import scenes

pytestmark = pytest.mark.gpu

BOUNDS = (-10.0, -10.0, -10.0, 10.0, 10.0, 10.0)


@pytest.mark.parametrize("capacity", [2, 64, 257, 700001])
def test_key_of_a_single_leaf(capacity):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import oracle
    from operatorgraph_gb300.engine import Engine

    rng = np.random.default_rng(17)
    rec = np.zeros(2, G.TERMINAL_DT)
    rec["m"] = rng.uniform(-9.0, 9.0, (2, 12)).astype(np.float32)
    rec["path"] = rng.integers(1 << 62, 1 << 64, 2, dtype=np.uint64)
    rec["rule"] = 1
    _, _, _, leaf, keys = oracle.lbvh(rec, BOUNDS)  # a key depends on its own record only
    want = np.full(capacity, ~np.uint64(0))
    want[0] = keys[np.nonzero(leaf == 0)[0][0]]
    eng = Engine(scenes.menger_table(0.5), node_capacity=1 << 12, max_terminals=capacity)
    t = torch.zeros((capacity, 64), dtype=torch.uint8, device="cuda")
    t[:2] = torch.from_numpy(rec.view(np.uint8).reshape(2, 64).copy()).cuda()
    bv = eng.lbvh(t, capacity, BOUNDS, count=torch.ones(1, dtype=torch.int64, device="cuda"))
    torch.cuda.synchronize()
    assert np.array_equal(bv["keys"].cpu().numpy().view(np.uint64), want)
    eng.release()
